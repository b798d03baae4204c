"""The sparse embedding's pruning at the boundary between kept and dropped entries:
equal values (the lower dim goes first), signed zeros, subnormals, values that differ
only in their low word, absent entries, one entry kept and one dropped; rows in pinned
memory, pageable memory and through the three-step calls.  Compared with a stable sort
in NumPy: exact."""
import numpy as np
import pytest

import distembed_gb300 as de
from distembed_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


def rows_with_ties(n, dim, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = rng.uniform(-0.5, 0.5, (n, dim))
    x[0] = 0.25                                                  # all equal
    x[1] = np.where(np.arange(dim) % 2, 0.0, -0.0)               # equal, with both zeros
    x[2] = rng.integers(-2, 3, dim) * 0.5                        # few values
    x[3] = 0.1 + np.arange(dim)[::-1] * np.spacing(0.1)          # the low word decides
    x[4] = rng.integers(-3, 4, dim) * 5e-324                     # subnormal
    x[5, : dim // 4] = de.Handle.ABSENT                          # absent entries order below all
    x[6] = np.where(np.arange(dim) < dim // 2, 1.0, 1.0 + np.spacing(1.0))
    x[7] = -np.abs(x[7])
    return x


@pytest.mark.parametrize("dim", [32, 64, 128, 256])
@pytest.mark.parametrize("kept", ["one", "half", "all but one"])
def test_boundary(dim, kept):
    import torch
    n, rp, col = gg.knn_csr(300, 4, 5, 3, seed=dim)
    keep = {"one": 1, "half": dim // 2, "all but one": dim - 1}[kept]
    density = (keep + 0.5) / dim
    x0 = rows_with_ties(n, dim, dim)
    want = x0.copy()
    low = np.argsort(np.where(x0 == 0.0, 0.0, x0), axis=1, kind="stable")[:, : dim - keep]
    np.put_along_axis(want, low, 0.0, axis=1)
    want[want == de.Handle.ABSENT] = 0.0
    present = int((x0 != de.Handle.ABSENT).sum()) // n
    assert present > keep or kept == "all but one"
    if present <= keep:  # nothing to prune: absent entries alone become 0
        want = np.where(x0 == de.Handle.ABSENT, 0.0, x0)
    pinned = torch.empty((n, dim), dtype=torch.float64, pin_memory=True).numpy()
    pinned[:] = x0
    with de.Handle(rp, col, dim) as h:
        got, coll = h.sparse_embedding(x0, 3, 64, 5, 0.02, density)
        assert np.array_equal(got, want)
        got, coll_pinned = h.sparse_embedding(pinned, 3, 64, 5, 0.02, density, inplace=True)
        assert got is pinned and np.array_equal(pinned, want) and np.array_equal(coll, coll_pinned)
        h.sparse_set(x0)
        h.sparse_run(3, 64, 5, 0.02, density)
        got, coll_steps = h.sparse_get()
        assert np.array_equal(got, want) and np.array_equal(coll, coll_steps)
