"""de_minibatch_noalloc reads row pointers as they are: where one falls, the row has no
entries, and keeps its repulsive pass.  Bitwise against the same rows as an ordinary CSR."""
import ctypes

import numpy as np
import pytest

import distembed_gb300 as de
from distembed_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


@pytest.mark.parametrize("dim,ns", [(32, 5), (128, 9), (256, 70)])
def test_falling_row_pointers(dim, ns):
    import torch
    n = 300
    rp, col = gg.rmat_csr_n(n, 8, seed=4)[1:]
    fall = np.array(rp)
    for r in range(20, n, 40):  # by 5 to 250 entries; the next row starts lower and is longer
        fall[r] = max(0, fall[r] - 5 * (r // 20) ** 2)
    assert fall.min() >= 0 and fall.max() <= len(col) and (np.diff(fall) < -2 * 8).any()
    lists = [col[fall[r]: max(fall[r + 1], fall[r])] for r in range(n)]
    plain = np.concatenate([[0], np.cumsum([len(v) for v in lists])])
    x0 = torch.from_numpy(gg.init_embedding(n, dim, seed=dim).astype(np.float32).reshape(-1)).cuda()
    negs = torch.tensor(de.negatives(n, 0, ns), dtype=torch.int32, device="cuda")
    out = []
    for pointers, columns in ((fall, col), (plain, np.concatenate(lists))):
        rowptr = torch.tensor(pointers, dtype=torch.int32, device="cuda")
        cols = torch.tensor(columns, dtype=torch.int32, device="cuda")
        x, loss = x0.clone(), torch.zeros(1, dtype=torch.float64, device="cuda")
        rc = de.lib().de_minibatch_noalloc(
            n, rowptr.data_ptr(), cols.data_ptr(), dim, x.data_ptr(), 0, n, negs.data_ptr(), ns, n, 1,
            ctypes.c_float(0.02), ctypes.c_float(5.0), loss.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == de.DE_OK, de.lib().de_last_error(None)
        torch.cuda.synchronize()
        out.append((x.cpu().numpy(), loss.item()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
