"""What a served job reserves: no more than its run allocates (a minibatch larger than the
graph reserves what the whole graph does), and enough: a job alone in an arena of exactly
its reservation runs to its end and gives the bits that it gives with room to spare."""
import numpy as np
import pytest

import distembed_gb300 as de
from distembed_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from distembed_gb300 import build
    build.build()


def serve(graph, dim, epochs, batch, ns, precision, hbm_bytes):
    rp, col = graph
    x0 = gg.init_embedding(len(rp) - 1, dim, seed=1).astype(np.float32)
    with de.Server(slots=1, hbm_bytes=hbm_bytes) as srv:
        return srv.wait(srv.submit(rp, col, x0, epochs, batch, ns, [0.02] * epochs, precision))


def graph(n):
    rp, col = gg.rmat_csr_n(n, 8, seed=n)[1:]
    assert np.diff(rp).max() > 64  # split rows
    return rp, col


@pytest.mark.parametrize("dim,ns,precision", [(32, 5, "fp32"), (128, 0, "fp32"), (128, 9, "bf16"), (256, 300, "bf16")])
def test_minibatch_larger_than_the_graph(dim, ns, precision):
    g = graph(1000)
    whole = serve(g, dim, 2, 1000, ns, precision, 64 << 20)
    large = serve(g, dim, 2, 16384, ns, precision, 64 << 20)
    assert large[2]["device_bytes"] == whole[2]["device_bytes"] <= (4 + 4 * 1000 * dim * 8) + (6 << 20)
    assert np.array_equal(large[0], whole[0]) and np.array_equal(large[1], whole[1])


# whole graph and many epochs, two to five minibatches, many minibatches with many draws
@pytest.mark.parametrize("n,dim,epochs,batch,ns,precision", [
    (1000, 32, 400, 16384, 5, "fp32"), (900, 128, 2, 900, 0, "fp32"), (2000, 64, 3, 700, 40, "fp32"),
    (2000, 256, 2, 401, 5, "fp32"), (5000, 32, 1, 8, 900, "fp32"), (1000, 64, 3, 16384, 64, "bf16"),
    (3000, 256, 1, 32, 1024, "bf16"), (2000, 128, 2, 701, 5, "bf16")])
def test_reservation_is_enough(n, dim, epochs, batch, ns, precision):
    g = graph(n)
    x, loss, info = serve(g, dim, epochs, batch, ns, precision, 1 << 30)
    x1, loss1, info1 = serve(g, dim, epochs, batch, ns, precision, (info["device_bytes"] + 255) & ~255)
    assert info1["device_bytes"] == info["device_bytes"]
    assert np.array_equal(x, x1) and np.array_equal(loss, loss1)
