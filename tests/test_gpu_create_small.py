"""Handle creation on both sides of the size up to which the host checks the columns (32,768
entries) and beyond which a kernel does: the same refusals, the same count of edges into
the last vertex, and the same graph (one minibatch against the FP64 oracle, relative L2
1e-5 as in tests/test_gpu_plain.py)."""
import numpy as np
import pytest

import distembed_gb300 as de
import oracle
from distembed_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu

N = 300


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


def graph(nnz):
    """nnz distinct entries of N vertices, some of them into the last one."""
    at = np.sort(np.random.Generator(np.random.PCG64(nnz)).choice(N * N, size=nnz, replace=False))
    return np.concatenate([[0], np.cumsum(np.bincount(at // N, minlength=N))]).astype(np.int64), at % N


@pytest.mark.parametrize("nnz", [0, 1, 1000, 32767, 32768, 32769])
def test_columns(nnz):
    rp, col = graph(nnz)
    x0 = gg.init_embedding(N, 32, seed=1).astype(np.float32).astype(np.float64)
    with de.Handle(rp, col, 32) as h:
        assert h.edge_updates(1, N, 0) == nnz - int((col == N - 1).sum())
        h.set_embeddings(x0)
        h.run(1, N, 5, 0.002)
        got = h.get_embeddings()
    want, _ = oracle.run(rp, col, x0, 1, N, 5, 0.002, quirks=True)
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("nnz", [1, 32768, 32769])
@pytest.mark.parametrize("value", [-1, N, 2 ** 32 + 5, -(2 ** 40)])
@pytest.mark.parametrize("last", [False, True])
def test_bad_column_is_refused(nnz, value, last):
    rp, col = graph(nnz)
    col[-1 if last else 0] = value
    with pytest.raises(de.DEError, match="column index out of range") as err:
        de.Handle(rp, col, 32)
    assert err.value.code == de.DE_ERR_INVALID
