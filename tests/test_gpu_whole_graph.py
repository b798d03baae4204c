"""Runs whose minibatch is the whole graph (FP32 plain form) go from one embedding buffer
to another, one launch an epoch: against the FP64 oracle for odd and even numbers of
epochs, with more epochs of losses than are kept at once, the warp teams and the one-warp
kernel, split rows and a resumed run, overlapping launches bitwise equal to serial ones
and a run in pieces bitwise equal to the whole.

Tolerances: those of tests/test_gpu_plain.py for a run of several epochs (relative L2
1e-4, loss 1e-3)."""
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


# n <= batch: one epoch and several, one loss CTA and more (2,048 items each), the minibatch
# exactly full; 3 x 130,000 items do not fit the losses kept (2^18)
@pytest.mark.parametrize("n,dim,batch,ns,epochs", [(1, 32, 1, 2, 2), (37, 64, 100, 5, 1), (900, 32, 16384, 5, 4),
                                                   (1900, 128, 1900, 0, 3), (2600, 256, 2601, 40, 2),
                                                   (5200, 64, 6000, 5, 3), (130_000, 32, 130_000, 3, 3)])
def test_whole_graph_epochs_match_oracle(n, dim, batch, ns, epochs):
    if n < 8:
        rp, col = np.zeros(n + 1, np.int64), np.zeros(0, np.int32)
    else:
        _, rp, col = gg.rmat_csr_n(n, 4, seed=dim + n)
    x0 = gg.init_embedding(n, dim, seed=2).astype(np.float32).astype(np.float64)
    lr = np.linspace(0.02, 0.01, epochs)
    want, want_loss = oracle.run(rp, col, x0, epochs, batch, ns, lr, quirks=True)
    got = []
    for options in ({}, {"pdl": False}):
        with de.Handle(rp, col, dim, **options) as h:
            h.set_embeddings(x0)
            loss = h.run(epochs, batch, ns, lr)
            got.append((h.get_embeddings(), loss))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert np.linalg.norm(got[0][0] - want) <= 1e-4 * np.linalg.norm(want)
    assert np.all(np.abs(got[0][1] - want_loss) <= 1e-3 * np.abs(want_loss))
    with de.Handle(rp, col, dim) as h:
        h.set_embeddings(x0)
        loss = [h.run(1, batch, ns, lr[e:e + 1], first_epoch=e)[0] for e in range(epochs)]
        assert np.array_equal(h.get_embeddings(), got[0][0]) and np.array_equal(loss, got[0][1])
