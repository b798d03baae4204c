"""Staged kernel of the batched form with four-CTA clusters compiled in (dim 128, at least as
many graphs as CTAs): every graph's bits are those of one-CTA teams, big graphs taken by a
whole cluster and small ones by its CTAs alone, with split rows and a ragged minibatch."""
import numpy as np
import pytest

import distembed_gb300 as de
from distembed_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("pairs,stages", [(1, 3), (2, 4)])
def test_four_ctas_give_the_bits_of_one(precision, pairs, stages):
    dim = 128
    graphs = [gg.rmat_csr_n(n, 5, seed=n)[1:] for n in [100 + 7 * (i % 20) for i in range(160)] + [20 + i for i in range(16)]]
    assert max(int(np.diff(rp).max()) for rp, _ in graphs) > 33
    x0s = [gg.init_embedding(len(rp) - 1, dim, seed=i).astype(np.float32) for i, (rp, _) in enumerate(graphs)]
    out = []
    for ctas in (1, 4):
        with de.Batch(graphs, dim, precision=precision) as b:
            b.set_shape("staged", team_warps=4, edge_cap=8, pairs=pairs, stages=stages, team_ctas=ctas)
            for i, x in enumerate(x0s):
                b.set_embeddings(i, x)
            loss = b.run(2, 100, 5, 0.02)
            out.append((b.get_embeddings(-1), loss))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
