"""Batched form, teams of several CTAs where few graphs would leave the GPU idle: a graph
alone (a team of eight CTAs) and the same graph among hundreds (fewer CTAs a team) give
the same bits, embeddings and every epoch's loss, with split rows, vertices without
edges, ragged minibatches and no draws at all; and they match the FP64 oracle at the
tolerances of tests/test_gpu_batched.py (relative L2 1e-4, loss 1e-3, FP32 storage)."""
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


def train(graphs, x0s, dim, precision, shape, batch, ns):
    with de.Batch(graphs, dim, precision=precision) as b:
        if shape:
            b.set_shape(**shape)
        for i, x in enumerate(x0s):
            b.set_embeddings(i, x)
        loss = b.run(2, batch, ns, 0.02)
        return [b.get_embeddings(i) for i in range(len(graphs))], loss


REGISTER = dict(kernel="register", vertices_per_warp=2, team_warps=16, edge_cap=16)
STAGED = dict(kernel="staged", team_warps=8, edge_cap=8, pairs=2, stages=3, team_ctas=2)


@pytest.mark.parametrize("dim,precision,shape,batch,ns", [
    (32, "fp32", None, 100, 5), (32, "fp32", REGISTER, 37, 0), (64, "fp32", None, 256, 9), (64, "bf16", None, 100, 5),
    (128, "fp32", None, 64, 33), (128, "bf16", REGISTER, 300, 3), (32, "fp32", STAGED, 100, 5),
    (64, "bf16", STAGED, 256, 9), (128, "fp32", STAGED, 37, 0)])
def test_alone_and_among_many(dim, precision, shape, batch, ns):
    big = gg.rmat_csr_n(700, 6, seed=dim)[1:]
    assert (np.diff(big[0]) == 0).any() and np.diff(big[0]).max() > 33
    many = [big] + [gg.rmat_csr_n(40 + i % 90, 3, seed=i)[1:] for i in range(399)]
    x0s = [gg.init_embedding(len(rp) - 1, dim, seed=i).astype(np.float32) for i, (rp, _) in enumerate(many)]
    alone, la = train(many[:1], x0s[:1], dim, precision, shape, batch, ns)
    mixed, lm = train(many, x0s, dim, precision, shape, batch, ns)
    assert np.array_equal(alone[0], mixed[0]) and np.array_equal(la[0], lm[0])
    if precision == "fp32":
        for i in (0, 1, 200, 399):
            want, want_loss = oracle.run(*many[i], x0s[i].astype(np.float64), 2, batch, ns, 0.02, quirks=True)
            assert np.linalg.norm(mixed[i] - want) <= 1e-4 * np.linalg.norm(want), i
            assert np.all(np.abs(lm[i] - want_loss) <= 1e-3 * np.abs(want_loss)), i
