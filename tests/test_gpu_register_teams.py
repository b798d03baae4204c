"""Register kernel of the batched form: as many teams are resident as the shape allows (an
SM's registers hold that many CTAs), and the CTAs that make a team follow the graphs: a
cluster where few graphs leave the GPU idle, one CTA where there are many and a CTA's
warps cover a minibatch in a round or two.  Read off the traced team of every graph."""
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


def blocks(count, n, dim, precision, batch, **shape):
    """The first CTA of every team that trained a graph."""
    graphs = [gg.rmat_csr_n(n + i % 13, 3, seed=i % 50)[1:] for i in range(count)]
    with de.Batch(graphs, dim, precision=precision) as b:
        b.set_shape("register", **shape)
        b.run(1, batch, 5, 0.02)
        return np.unique(b.trace()[:, 2])


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("dim,vpw,warps,per_sm", [(32, 4, 8, 2), (32, 2, 8, 2), (32, 4, 4, 4), (64, 4, 8, 2), (64, 2, 4, 4),
                                                  (64, 1, 8, 2), (128, 1, 4, 3), (128, 1, 8, 2), (128, 4, 4, 2)])
def test_resident_teams(dim, vpw, warps, per_sm, precision):
    # minibatches of one round, and far more graphs than teams: single CTAs, as many as fit
    got = blocks(2500, 40, dim, precision, 16, vertices_per_warp=vpw, team_warps=warps, edge_cap=32)
    assert got.max() + 1 == per_sm * sms()


@pytest.mark.parametrize("dim,precision", [(32, "fp32"), (64, "bf16"), (128, "fp32")])
@pytest.mark.parametrize("count,n,batch,vpw,warps,ctas", [
    (225, 380, 200, 4, 32, 1), (225, 380, 200, 4, 16, 1), (450, 200, 100, 2, 16, 1), (5, 2000, 256, 4, 8, 8),
    (5, 2000, 256, 2, 16, 8)])
def test_ctas_of_a_team(dim, precision, count, n, batch, vpw, warps, ctas):
    got = blocks(count, n, dim, precision, batch, vertices_per_warp=vpw, team_warps=warps, edge_cap=128)
    if ctas == 1:
        assert (got % 2 == 1).any()
    else:
        assert (got % ctas == 0).all() and len(got) > 1
