"""Batched form: the staging areas a run allocates are those its teams use, of the rows of
its largest minibatch, however many CTAs a team has; and where the graphs are fewer than
the launch's CTAs (an area a graph) a graph trained by a cluster, or alone beside the
others, gives the bits that it gives by itself."""
import numpy as np
import pytest
import torch

import distembed_gb300 as de
from distembed_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu

STAGED = dict(kernel="staged", team_warps=8, edge_cap=8, pairs=2, stages=3, team_ctas=2)


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("shape", [None, STAGED])
@pytest.mark.parametrize("count,n", [(24, 700), (3, 5000), (300, 60)])
def test_areas_are_those_in_use(shape, count, n):
    dim, batch = 128, 16384
    graphs = [gg.rmat_csr_n(n + i % 7, 4, seed=i)[1:] for i in range(count)]
    deg = max(int(np.diff(rp).max()) for rp, _ in graphs)
    parts = max(len(col) for _, col in graphs) // 16 + n + 7  # pieces and items of a graph at most
    with de.Batch(graphs, dim) as b:
        if shape:
            b.set_shape(**shape)
        b.run(1, 8, 5, 0.02)  # the kernel is loaded and the small buffers are there
        before = free_bytes()
        b.run(1, batch, 5, 0.02)
        used = before - free_bytes()
    # an area a graph at most: its staged rows, partial rows and item losses; 16 MiB for the
    # work lists and the allocator's rounding
    need = min(count, 152 * 8) * ((n + 7) * dim * 4 + parts * (dim * 4 + 4))
    assert deg > 16 and used <= need + (16 << 20), (used, need)


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_fewer_graphs_than_ctas(precision):
    dim, batch, ns = 64, 50, 5
    graphs = [gg.rmat_csr_n(n, 6, seed=n)[1:] for n in [2500, 1800] + [60 + 11 * i for i in range(20)]]
    x0s = [gg.init_embedding(len(rp) - 1, dim, seed=i).astype(np.float32) for i, (rp, _) in enumerate(graphs)]

    def train(which):
        with de.Batch([graphs[i] for i in which], dim, precision=precision) as b:
            b.set_shape(**STAGED)
            for k, i in enumerate(which):
                b.set_embeddings(k, x0s[i])
            loss = b.run(3, batch, ns, 0.02)
            return [b.get_embeddings(k) for k in range(len(which))], loss, b.trace()

    rows, loss, trace = train(range(len(graphs)))
    assert len(set(trace[:, 2])) > 2  # several teams at once
    for i in (0, 1, 2, 9, 21):
        alone, la, _ = train([i])
        assert np.array_equal(alone[0], rows[i]) and np.array_equal(la[0], loss[i]), i
