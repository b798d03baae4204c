"""SpMM into a device tensor: straight into it where its address is a multiple of 16
bytes, through the handle's own rows elsewhere; the same values either way, nothing
written outside, and they match the FP64 oracle at the tolerance of
tests/test_gpu_spmm.py (1e-5 elementwise).  Rows of 0, 1 and around 8, 16 and 32 CSR
entries (the windows of the kernel), and split rows."""
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


@pytest.mark.parametrize("dim", [32, 64, 128, 256])
@pytest.mark.parametrize("quirks", [True, False])
def test_device_output(dim, quirks):
    import torch
    n = 700
    deg = np.array([0, 1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 64, 65, 600])[np.arange(n) % 14]
    rng = np.random.Generator(np.random.PCG64(dim))
    dst = np.concatenate([rng.choice(n, size=d, replace=False) for d in deg])
    rp, col = gg.coo_to_csr(n, np.repeat(np.arange(n), deg), dst)
    x0 = gg.init_embedding(n, dim, seed=1).astype(np.float32)
    want = oracle.spmm(rp, col, x0.astype(np.float64), 0.02, quirks=quirks)
    with de.Handle(rp, col, dim, quirks=quirks) as h:
        h.set_embeddings(x0)
        got = []
        for shift in (0, 1, 4):
            store = torch.full((n * dim + 8,), 7.0, device="cuda")
            out = store[shift: shift + n * dim].view(n, dim)
            torch.cuda.synchronize()
            h.spmm(100, 0.02, out=out)
            got.append(out.cpu().numpy())
            assert bool((store[:shift] == 7.0).all()) and bool((store[shift + n * dim:] == 7.0).all())
        assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
        assert np.array_equal(got[0], h.spmm(100, 0.02, dtype=np.float32))
    tol = 1e-5 * (np.abs(want) + np.sqrt(np.mean(want ** 2)))
    assert np.all(np.abs(got[0] - want) <= tol)
