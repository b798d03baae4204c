"""COO -> CSR with the keys made on the GPU, at the edges of its launches (entry counts
around a CTA of 256, one entry, one row, nothing but diagonal entries) and for entries
outside the matrix, the first of which is named as the host check names it.  Integer
work: equal to a NumPy restatement."""
import numpy as np
import pytest

import distembed_gb300 as de

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


@pytest.mark.parametrize("rows,cols,nnz,mirror,diagonal", [
    (1, 1, 1, True, False), (1, 9, 255, False, False), (65537, 65537, 256, True, False), (40, 40, 257, True, True),
    (2 ** 20 + 1, 3, 1000, False, False), (3000, 3000, 200000, True, False), (3000, 70000, 100001, False, False)])
def test_keys_and_merge(rows, cols, nnz, mirror, diagonal):
    rng = np.random.Generator(np.random.PCG64(nnz))
    r = rng.integers(0, rows, nnz)
    c = r.copy() if diagonal else rng.integers(0, cols, nnz)
    key = r * np.int64(cols) + c
    if mirror:
        key = np.concatenate([key, c * np.int64(cols) + r])
    key = np.unique(key)
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(key // cols, minlength=rows))])
    got = de.coo_to_csr(rows, cols, r, c, mirror=mirror)
    assert got[:2] == (rows, cols)
    assert np.array_equal(got[2], rowptr) and np.array_equal(got[3], key % cols)


@pytest.mark.parametrize("bad,mirror,text", [
    ([(5, 3, 7), (9, 10, 0)], False, "COO entry"), ([(700, 0, -1)], False, "COO entry"),
    ([(3, 7, 1), (8, 0, 9)], True, "mirrored"), ([(2, 0, 9), (3, 7, 1)], True, "COO entry"),
    ([(999, 9, 4)], True, "mirrored")])
def test_entries_outside_are_refused(bad, mirror, text):
    # 10 x 5: entry e is (i, j); its mirror image (j, i) must fit as well
    r, c = np.arange(1000) % 4, np.arange(1000) % 4
    for e, i, j in bad:
        r[e], c[e] = i, j
    with pytest.raises(de.DEError, match=text) as err:
        de.coo_to_csr(10, 5, r, c, mirror=mirror)
    assert err.value.code == de.DE_ERR_INVALID
