"""Warps to a work item of the FP32 plain form, on both sides of every limit of the rule
(608 items: four warps or two, not at dim 32; 1,824 items at dim 64 and 128 and 1,520 at 32
and 256: two or one): the kernel that runs, the FP64 oracle, and overlapping launches
bitwise equal to serial ones.  The minibatches hold exactly that many work items, split
rows and a row without entries among them.

Tolerances: those of tests/test_gpu_plain.py for a run of several epochs (relative L2
1e-4, loss 1e-3), which the rounding of the sums' order does not change."""
import numpy as np
import pytest
import torch

import distembed_gb300 as de
import oracle
from distembed_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu

LIMITS = {32: (0, 1520), 64: (608, 1824), 128: (608, 1824), 256: (608, 1520)}
CASES = [(dim, items + more, 4 if items + more <= four else 2 if items + more <= two else 1)
         for dim, (four, two) in LIMITS.items() for items in (four, two) if items for more in (0, 1)]


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


def graph(n, rows, seed):
    """n rows of 3 entries, but in every `rows` of them one of none and one of 70 (three items)."""
    deg = np.full(n, 3)
    deg[5::rows] = 0
    deg[9::rows] = 70
    rng = np.random.Generator(np.random.PCG64(seed))
    col = np.concatenate([np.sort(rng.choice(n, size=d, replace=False)) for d in deg])
    return np.concatenate([[0], np.cumsum(deg)]).astype(np.int64), col.astype(np.int64)


@pytest.mark.parametrize("dim,items,warps", CASES)
def test_limits(dim, items, warps):
    rows = items - 2
    n = 2 * rows + rows // 3
    rp, col = graph(n, rows, items)
    assert np.maximum(1, -(-np.diff(rp)[:rows] // 32)).sum() == items
    x0 = gg.init_embedding(n, dim, seed=2).astype(np.float32).astype(np.float64)
    lr = np.array([0.02, 0.01])
    want, want_loss = oracle.run(rp, col, x0, 2, rows, 5, lr, quirks=True)
    got = []
    for pdl in (True, False):
        with de.Handle(rp, col, dim, pdl=pdl) as h:
            h.set_embeddings(x0)
            loss = h.run(2, rows, 5, lr)
            got.append((h.get_embeddings(), loss))
            if pdl:
                h.set_embeddings(x0)
                torch.cuda.synchronize()
                with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
                    h.run(1, rows, 5, 0.02, want_loss=False)
                    torch.cuda.synchronize()
                names = {e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA}
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert np.linalg.norm(got[0][0] - want) <= 1e-4 * np.linalg.norm(want)
    assert np.all(np.abs(got[0][1] - want_loss) <= 1e-3 * want_loss)
    kernel = f"plain_team_kernel<{dim}, {warps}>" if warps > 1 else f"plain_batch_kernel<{dim}>"
    assert any(kernel in name for name in names), (kernel, names)
