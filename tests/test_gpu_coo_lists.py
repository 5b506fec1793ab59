"""The two item lists of the COO tiles: steps without an output cut tiles of
one and a half shares of a resident CTA, steps with one only from two shares."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spmv(gg, g, x, flags):
    n = g.n
    xd, yd = gg.DeviceArray(g, np.float32, x), gg.DeviceArray(g, np.float32, np.zeros(n, np.float32))
    g.edge_map(g.frontier_all(), gg.F_SPMV, gg.PairArgs(xd.ptr, yd.ptr), flags=flags).close()
    y = yd.download()
    xd.close()
    yd.close()
    return y


# shares of the largest tile: below one and a half, between, above two
@pytest.mark.parametrize("partitions,tile_edges", [(384, 1 << 15), (384, 1 << 16), (64, 1 << 17)])
def test_spmv_with_and_without_output(gg, partitions, tile_edges):
    hg = gg.HostGraph.er(1 << 20, 16 << 20, seed=2)
    g = gg.Graph(hg, partitions=partitions, tile_edges=tile_edges)
    x = np.random.default_rng(1).random(hg.n, dtype=np.float32) + np.float32(0.5)
    want = spmv(gg, g, x, gg.EM_FORCE_CSC)
    for _ in range(2):  # the slabs are clear again after a run
        for flags in (gg.EM_NO_OUTPUT, 0):
            # sums of about 16 terms in another order
            np.testing.assert_allclose(spmv(gg, g, x, flags), want, rtol=2e-5)
    g.close()
