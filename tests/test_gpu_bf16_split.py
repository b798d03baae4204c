"""BF16 form, the repulsion GEMMs with a tile's negatives split between one to four CTAs
(uneven shares of 1 to 16 chunks of 64 negatives, one to many 128-row tiles, a last tile
of one row), with and without the loss; and device rows set in place or, off a 16-byte
boundary, by a copy.  Against the FP64 oracle at the tolerances of tests/test_gpu_bf16.py
(one minibatch's update within 2e-2 relative L2, loss within 1 %)."""
import numpy as np
import pytest

import distembed_gb300 as de
import oracle
from distembed_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


def bf16_round(x):
    u = np.asarray(x, dtype=np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32).astype(np.float64)


@pytest.mark.parametrize("dim,n,ns", [(64, 100, 64), (64, 129, 130), (128, 257, 190), (128, 1000, 257), (128, 129, 448),
                                      (256, 300, 577), (256, 5000, 1024), (64, 20000, 300)])
@pytest.mark.parametrize("loss", [True, False])
def test_one_minibatch(dim, n, ns, loss):
    _, rp, col = gg.rmat_csr_n(n, 4, seed=dim + ns)
    x0 = bf16_round(gg.init_embedding(n, dim, seed=1))
    want, want_loss = oracle.batch_grad(rp, col, x0, n, ns, 0.02, 0, 0, n, quirks=True)
    with de.Handle(rp, col, dim, precision="bf16", compute_loss=loss) as h:
        h.set_embeddings(x0)
        got_loss = h.run(1, n, ns, 0.02)
        got = h.get_embeddings() - x0
    assert np.linalg.norm(got - want) <= 2e-2 * np.linalg.norm(want)
    if loss:
        assert abs(got_loss[0] - want_loss.sum()) <= 1e-2 * want_loss.sum()


@pytest.mark.parametrize("dim", [64, 128, 256])
def test_device_rows(dim):
    import torch
    n, rp, col = gg.knn_csr(300, 4, 5, 3, seed=dim)
    x0 = torch.from_numpy(gg.init_embedding(n, dim, seed=2).astype(np.float32)).cuda()
    out = []
    for shift in (0, 1):
        store = torch.zeros(n * dim + 4, device="cuda")
        x = store[shift: shift + n * dim].view(n, dim)
        x.copy_(x0)
        torch.cuda.synchronize()
        with de.Handle(rp, col, dim, precision="bf16") as h:
            h.set_embeddings(x)
            assert np.array_equal(h.get_embeddings(dtype=np.float32), x0.cpu().numpy())
            loss = h.run(2, 100, 70, 0.02)
            out.append((h.get_embeddings(), loss))
    with de.Handle(rp, col, dim, precision="bf16") as h:
        h.set_embeddings(x0.cpu().numpy())
        loss = h.run(2, 100, 70, 0.02)
        out.append((h.get_embeddings(), loss))
    for x, loss in out[1:]:
        assert np.array_equal(x, out[0][0]) and np.array_equal(loss, out[0][1])
