"""The CSR that de_coo_to_csr keeps on the GPU: copied out again and again, and from several
threads at once, with nothing between building and freeing it but its copies; without
entries it holds nothing."""
import ctypes
import threading

import numpy as np
import pytest

import distembed_gb300 as de

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


@pytest.mark.parametrize("rows,nnz", [(500, 0), (1, 1), (500, 9000), (70000, 400000)])
def test_copies(rows, nnz):
    L = de.lib()
    rng = np.random.Generator(np.random.PCG64(rows))
    src, dst = (rng.integers(0, rows, nnz).astype(np.int64) for _ in range(2))
    key = np.unique(src * rows + dst)
    want = np.concatenate([[0], np.cumsum(np.bincount(key // rows, minlength=rows))]), key % rows
    c = ctypes.c_void_p()
    assert L.de_coo_to_csr(rows, rows, src.ctypes.data, dst.ctypes.data, nnz, 0, 0, ctypes.byref(c)) == de.DE_OK
    got = [(np.full(rows + 1, -1, np.int64), np.full(len(key), -1, np.int64)) for _ in range(7)]

    def copy(i):
        assert L.de_csr_copy(c, got[i][0].ctypes.data, got[i][1].ctypes.data) == de.DE_OK

    for i in range(3):
        copy(i)
    threads = [threading.Thread(target=copy, args=(i,)) for i in range(3, 7)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    L.de_csr_free(c)
    for rowptr, col in got:
        assert np.array_equal(rowptr, want[0]) and np.array_equal(col, want[1])
