"""de_minibatch_noalloc against the FP64 oracle at the edges of its row split: rows of
0 to several hundred CSR entries (a group holds 8 pairs, a CTA 8 or 4 groups at once),
0 to 9 negatives, minibatches on both sides of the four- and eight-warp split, and an
embedding that starts 4 bytes past a 16-byte boundary (the 4-byte-load variant).

Tolerance: one FP32 step against FP64, as tests/test_gpu_plain.py's one-minibatch
tests: relative L2 1e-5 of the update, loss 1e-5 relative (FP32 terms, FP64 sums)."""
import ctypes

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


def ladder(n, top):
    """A directed graph whose row r has (r * 7) % top entries, but row 1 has n - 1."""
    deg = (np.arange(n) * 7) % top
    deg[1] = n - 1
    rng = np.random.Generator(np.random.PCG64(5))
    src = np.repeat(np.arange(n), deg)
    dst = np.concatenate([rng.choice(n, size=d, replace=False) for d in deg])
    return gg.coo_to_csr(n, src, dst)


@pytest.mark.parametrize("dim,n,batch,ns,shift", [
    (32, 700, 700, 0, 0), (32, 700, 233, 1, 4), (64, 700, 256, 5, 0), (64, 1300, 1217, 8, 4),
    (128, 1300, 1216, 9, 0), (128, 700, 100, 5, 8), (256, 1300, 1300, 3, 0), (256, 700, 64, 9, 4)])
@pytest.mark.parametrize("first", [True, False])
def test_one_minibatch_matches_oracle(dim, n, batch, ns, shift, first):
    import torch
    rp, col = ladder(n, 70)
    x0 = gg.init_embedding(n, dim, seed=dim + n).astype(np.float32)
    j = 0 if first else (n - 1) // batch  # the last one: ragged where batch does not divide n
    rows = min(batch, n - j * batch)
    want, row_loss = oracle.batch_grad(rp, col, x0.astype(np.float64), batch, ns, 0.02, j, j, rows, quirks=True)
    want, want_loss = want[:rows], row_loss[:rows].sum()
    store = torch.zeros(n * dim + 4, dtype=torch.float32, device="cuda")
    x = store[shift // 4: shift // 4 + n * dim]
    x.copy_(torch.from_numpy(x0).reshape(-1))
    assert x.data_ptr() % 16 == shift
    rowptr = torch.tensor(rp, dtype=torch.int32, device="cuda")
    cols = torch.tensor(col, dtype=torch.int32, device="cuda")
    negs = torch.tensor(np.append(de.negatives(n, j, ns), 0), dtype=torch.int32, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    rc = de.lib().de_minibatch_noalloc(
        n, rowptr.data_ptr(), cols.data_ptr(), dim, x.data_ptr(), j, batch, negs.data_ptr(), ns, rows, 1,
        ctypes.c_float(0.02), ctypes.c_float(5.0), loss.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == de.DE_OK, de.lib().de_last_error(None)
    torch.cuda.synchronize()
    got = x.cpu().numpy().reshape(n, dim).astype(np.float64) - x0
    mine = np.s_[j * batch: j * batch + rows]
    assert not np.delete(got, mine, axis=0).any()  # rows outside the minibatch, and nothing past the embedding
    assert not store[: shift // 4].any() and not store[shift // 4 + n * dim:].any()
    got = got[mine]
    # the update is read back as x1 - x0: its rounding is half an ulp of |x| <= |x0| + |update|
    ulp = np.finfo(np.float32).eps * (np.abs(x0[mine]) + np.abs(want))
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want) + np.linalg.norm(ulp)
    assert abs(float(loss.item()) - want_loss) <= 1e-5 * want_loss + 1e-12


@pytest.mark.parametrize("dim,shift", [(32, 0), (64, 4), (128, 0), (256, 4)])
def test_calls_behind_one_another_match_calls_one_by_one(dim, shift):
    """The same minibatch again and again, then its neighbour: each call reads rows that
    the call queued before it writes; bitwise as with the GPU idle between the calls."""
    import torch
    n, batch, ns = 600, 300, 5
    rp, col = ladder(n, 40)
    x0 = torch.from_numpy(gg.init_embedding(n, dim, seed=dim).astype(np.float32).reshape(-1)).cuda()
    rowptr = torch.tensor(rp, dtype=torch.int32, device="cuda")
    cols = torch.tensor(col, dtype=torch.int32, device="cuda")
    calls = [0] * 10 + [1, 0] * 5
    negs = torch.tensor(np.stack([de.negatives(n, k, ns) for k in range(len(calls))]), dtype=torch.int32, device="cuda")
    out = []
    for idle in (True, False):
        store = torch.zeros(n * dim + 4, dtype=torch.float32, device="cuda")
        x = store[shift // 4: shift // 4 + n * dim]
        x.copy_(x0)
        loss = torch.zeros(len(calls), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for k, j in enumerate(calls):
            rc = de.lib().de_minibatch_noalloc(
                n, rowptr.data_ptr(), cols.data_ptr(), dim, x.data_ptr(), j, batch, negs[k].data_ptr(), ns, batch, 1,
                ctypes.c_float(0.02), ctypes.c_float(5.0), loss[k:].data_ptr(), torch.cuda.current_stream().cuda_stream)
            assert rc == de.DE_OK, de.lib().de_last_error(None)
            if idle:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        out.append((x.cpu().numpy(), loss.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
