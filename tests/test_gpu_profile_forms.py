"""A profiled epoch takes the kernels that a run of one epoch takes, for one minibatch, a
few and many, and leaves the same bits; its launches are the kinds and times it reports."""
import numpy as np
import pytest
import torch

import distembed_gb300 as de
from distembed_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


@pytest.fixture(scope="module", autouse=True)
def _profiler(_built):
    for _ in range(5):  # the profiler's first session in a process may see nothing
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
            torch.zeros(1, device="cuda").add_(1)
            torch.cuda.synchronize()
        if any(e.device_type == torch.autograd.DeviceType.CUDA for e in p.events()):
            break


def kernels(f):
    """Names of the library's kernels that f launches, in order."""
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    ev = [e for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA and "_kernel" in e.name]
    return [e.name for e in sorted(ev, key=lambda e: e.time_range.start)]


@pytest.mark.parametrize("compute_loss", [True, False])
@pytest.mark.parametrize("batch,batches", [(1000, 1), (4096, 1), (300, 4), (100, 10)])
def test_profiled_epoch_is_the_run(batch, batches, compute_loss):
    rp, col = gg.rmat_csr_n(1000, 8, seed=3)[1:]
    x0 = gg.init_embedding(1000, 64, seed=1).astype(np.float32).astype(np.float64)
    with de.Handle(rp, col, 64, compute_loss=compute_loss) as h:
        h.set_embeddings(x0)
        ran = kernels(lambda: h.run(1, batch, 5, 0.02, want_loss=False))
        want = h.get_embeddings()
        h.set_embeddings(x0)
        got = []
        profiled = kernels(lambda: got.append(h.profile_epoch(batch, 5, 0.02)))
        ms, kind = got[0]
        assert np.array_equal(h.get_embeddings(), want)
    assert len(ran) >= batches and profiled == ran
    assert list(kind) == [0] * batches + [3] and np.all(ms >= 0)
