"""de_minibatch_noalloc on both sides of its rule for the warps of a row: eight where every
row's CTA is resident at once (six CTAs an SM at dim 32, five at 64, three at 128 and 256),
four beyond; the kernel that runs, and the FP64 oracle.

Tolerance: one FP32 step against FP64, as tests/test_gpu_plain.py's one-minibatch
tests: relative L2 1e-5 of the update, loss 1e-5 relative (FP32 terms, FP64 sums)."""
import ctypes

import numpy as np
import pytest
import torch

import distembed_gb300 as de
import oracle
from distembed_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu

RESIDENT = {32: 152 * 6, 64: 152 * 5, 128: 152 * 3, 256: 152 * 3}


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()
    for _ in range(5):  # the profiler's first session in a process may see nothing
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
            torch.zeros(1, device="cuda").add_(1)
            torch.cuda.synchronize()
        if any(e.device_type == torch.autograd.DeviceType.CUDA for e in p.events()):
            break


@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("dim", sorted(RESIDENT))
def test_warps_of_a_row(dim, more, shift):
    rows, ns = RESIDENT[dim] + more, 5
    n = rows + 40
    rp, col = gg.rmat_csr_n(n, 8, seed=dim)[1:]
    x0 = gg.init_embedding(n, dim, seed=dim).astype(np.float32)
    want, row_loss = oracle.batch_grad(rp, col, x0.astype(np.float64), rows, ns, 0.02, 0, 0, rows, quirks=True)
    want, want_loss = want[:rows], row_loss[:rows].sum()
    store = torch.zeros(n * dim + 4, dtype=torch.float32, device="cuda")
    x = store[shift // 4: shift // 4 + n * dim]
    x.copy_(torch.from_numpy(x0).reshape(-1))
    rowptr = torch.tensor(rp, dtype=torch.int32, device="cuda")
    cols = torch.tensor(col, dtype=torch.int32, device="cuda")
    negs = torch.tensor(de.negatives(n, 0, ns), dtype=torch.int32, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        rc = de.lib().de_minibatch_noalloc(
            n, rowptr.data_ptr(), cols.data_ptr(), dim, x.data_ptr(), 0, rows, negs.data_ptr(), ns, rows, 1,
            ctypes.c_float(0.02), ctypes.c_float(5.0), loss.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    assert rc == de.DE_OK, de.lib().de_last_error(None)
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    kernel = f"noalloc_rows_kernel<{dim}, {4 if dim == 256 else 8}, {4 if more else 8}, "
    assert any(kernel in name for name in names), (kernel, names)
    got = x.cpu().numpy().reshape(n, dim).astype(np.float64) - x0
    assert not got[rows:].any()
    ulp = np.finfo(np.float32).eps * (np.abs(x0[:rows]) + np.abs(want))  # the update is read back as x1 - x0
    assert np.linalg.norm(got[:rows] - want) <= 1e-5 * np.linalg.norm(want) + np.linalg.norm(ulp)
    assert abs(float(loss.item()) - want_loss) <= 1e-5 * want_loss + 1e-12
