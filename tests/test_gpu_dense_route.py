"""Dense steps below m/2 run on the partitioned COO by default
(dense_takes_coo): the same values, outputs and statistics as the CSC pull, for
every kind of graph, and the CSC pull where the COO does not stand for it.
(BellmanFord's step gathers distances that the same step lowers, so two runs of
one kernel differ already; its fixed point is tested with the applications.)"""
import ctypes as C

import numpy as np
import pytest

from conftest import ok_partitions

pytestmark = pytest.mark.gpu

BUILDS = {"default": {}, "hot": {"vertex_order": 1}, "csr_order": {"order": 0}, "window": {"coo_window": 512},
          "vertex": {"balance": 1}, "source": {"part_how": 1}, "small_tiles": {"tile_vertices": 64, "tile_edges": 512}}


def step(gg, g, n, fid, frontier, policy, rng):
    """One edgeMap of `fid` from `frontier`: (its arrays, output mask, stats)."""
    g.set_dense_policy(policy)
    a = rng.integers(0, n, n).astype(np.int32)
    if fid == gg.F_CC:
        ids, prev = gg.DeviceArray(g, np.int32, a), gg.DeviceArray(g, np.int32, a)
        args, arrays = gg.CcArgs(ids.ptr, prev.ptr), [ids]
    elif fid == gg.F_BC:
        val = gg.DeviceArray(g, np.float32, (a % 3).astype(np.float32))  # small integers: sums are exact
        # the members are visited, so no step changes a value that it gathers
        vis = gg.DeviceArray(g, np.uint8, (a % 2).astype(np.uint8) | frontier.mask())
        args, arrays = gg.PairArgs(val.ptr, vis.ptr), [val, vis]
    else:
        x = gg.DeviceArray(g, np.float32, (a % 5 - 2).astype(np.float32))
        y = gg.DeviceArray(g, np.float32, 1.0)
        args, arrays = gg.PairArgs(x.ptr, y.ptr), [y]
    out = g.edge_map(frontier, fid, args)
    st = g.last_edge_map_stats()
    return [d.download() for d in arrays], out.mask(), out.stats(), st.kind, (st.output_active, st.output_out_edges)


@pytest.mark.parametrize("sym", [True, False])
@pytest.mark.parametrize("build", sorted(BUILDS))
def test_mid_size_frontier(gg, build, sym):
    hg = gg.HostGraph.rmat(11, 12, seed=77, symmetric=sym).add_weights(gg.W_INT32, seed=3, lo=1, hi=9)
    kw = BUILDS[build]
    P = ok_partitions(hg, 8) if "part_how" not in kw else 4
    try:
        g = gg.Graph(hg, partitions=P, **kw)
    except gg.GGError:
        pytest.skip("the partitioner refuses this count")
    deg = hg.degrees().astype(np.int64)
    rng = np.random.default_rng(5)
    order = rng.permutation(hg.n)
    pick = order[:np.searchsorted(np.cumsum(deg[order] + 1), hg.m // 4)]
    new_of_old = g.vertex_order()
    mask = np.zeros(hg.n, np.uint8)
    mask[new_of_old[pick]] = 1
    for transposed in (False, True):
        if transposed:
            g.transpose()
        fm, oe = g.frontier_from_mask(mask).stats()
        dense = hg.m // 20 < fm + oe <= hg.m // 2
        for fid in (gg.F_CC, gg.F_SPMV, gg.F_PRDELTA, gg.F_BC):
            got = step(gg, g, hg.n, fid, g.frontier_from_mask(mask), 0, np.random.default_rng(9))
            want = step(gg, g, hg.n, fid, g.frontier_from_mask(mask), 1, np.random.default_rng(9))
            if dense:
                assert got[3] == want[3] == 2
            if fid == gg.F_PRDELTA:  # quotients: sums differ by their order alone
                for x, y in zip(got[0], want[0]):
                    np.testing.assert_allclose(x, y, rtol=0, atol=2e-4)
            else:
                for x, y in zip(got[0], want[0]):
                    np.testing.assert_array_equal(x, y)
            np.testing.assert_array_equal(got[1], want[1])
            assert got[2] == want[2] and got[4] == want[4]
    g.close()
