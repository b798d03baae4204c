"""Small minibatches of the FP32 plain form run several warps to a work item: against
the FP64 oracle on both sides of the four-, two- and one-warp split, with rows of no
entries, split rows, more draws than a warp's lanes hold at once, and overlapping
launches (minibatch j+1 starts before j ends) bitwise equal to serial ones.

Tolerances: those of tests/test_gpu_plain.py for a run of several epochs (relative L2
1e-4, loss 1e-3), which the rounding of the sums' order does not change."""
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


# minibatches of few to many items around 912 (four warps) and 2,432 / 1,824 (two)
@pytest.mark.parametrize("dim,batch,ns", [(32, 7, 0), (32, 300, 5), (64, 880, 130), (64, 1000, 9), (128, 64, 40),
                                          (128, 2400, 5), (128, 2600, 5), (256, 33, 70), (256, 1500, 3),
                                          (256, 1900, 3)])
def test_small_minibatches_match_oracle(dim, batch, ns):
    n = 5200 if batch > 300 else 900
    _, rp, col = gg.rmat_csr_n(n, 4, seed=dim + batch)  # hubs, and vertices without edges
    assert (np.diff(rp) == 0).any() and (np.diff(rp) > 64).any()
    x0 = gg.init_embedding(n, dim, seed=2).astype(np.float32).astype(np.float64)
    lr = np.array([0.02, 0.01])
    want, want_loss = oracle.run(rp, col, x0, 2, batch, ns, lr, quirks=True)
    got = []
    for pdl in (True, False):
        with de.Handle(rp, col, dim, pdl=pdl) as h:
            h.set_embeddings(x0)
            loss = h.run(2, batch, ns, lr)
            got.append((h.get_embeddings(), loss))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert np.linalg.norm(got[0][0] - want) <= 1e-4 * np.linalg.norm(want)
    assert np.all(np.abs(got[0][1] - want_loss) <= 1e-3 * want_loss)
