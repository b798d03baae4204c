"""Handle creation: columns are checked and counted on the GPU in pieces of what the
embedding holds (few vertices with many entries take several pieces), and work lists are
ordered by counting.  The runs match the FP64 oracle (tolerances of
tests/test_gpu_plain.py), and bad graphs are refused as before."""
import numpy as np
import pytest

import distembed_gb300 as de
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


def dense_graph(n, keep, seed):
    """Every pair of n vertices with probability `keep`: far more entries than n."""
    rng = np.random.Generator(np.random.PCG64(seed))
    adj = rng.random((n, n)) < keep
    adj[n // 2] = False  # a vertex without entries
    return np.concatenate([[0], np.cumsum(adj.sum(1))]), np.nonzero(adj)[1].astype(np.int64)


@pytest.mark.parametrize("n,keep,dim,batch,cap", [(300, 0.9, 32, 64, 0), (300, 0.9, 32, 300, 7), (257, 0.3, 64, 100, 1),
                                                  (40, 1.0, 128, 7, 31), (1, 0.0, 32, 5, 0)])
def test_dense_graph_matches_oracle(n, keep, dim, batch, cap):
    rp, col = dense_graph(n, keep, n)
    x0 = np.random.Generator(np.random.PCG64(1)).uniform(-0.5, 0.5, (n, dim)).astype(np.float32).astype(np.float64)
    want, want_loss = oracle.run(rp, col, x0, 2, batch, 5, 0.002, quirks=True)
    with de.Handle(rp, col, dim, edge_cap=cap) as h:
        h.set_embeddings(x0)
        loss = h.run(2, batch, 5, 0.002)
        got = h.get_embeddings()
        assert h.edge_updates(1, n, 0) == len(col) - int((col == n - 1).sum())
    assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want)
    assert np.allclose(loss, want_loss, rtol=1e-3, atol=1e-9)


@pytest.mark.parametrize("at", [0, 4800, 20000, -1])
@pytest.mark.parametrize("value", [-1, 300, 2 ** 32 + 5, -(2 ** 40)])
def test_bad_column_is_refused(at, value):
    rp, col = dense_graph(300, 0.9, 2)
    col = col.copy()
    col[at] = value
    with pytest.raises(de.DEError, match="column index out of range") as err:
        de.Handle(rp, col, 32)
    assert err.value.code == de.DE_ERR_INVALID
