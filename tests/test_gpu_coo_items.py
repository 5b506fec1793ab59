"""COO tiles cut into several work items (build_coo_items): the items' sums
meet in the tile's slab, and the item that arrives last commits."""
import numpy as np
import pytest

from conftest import PR_MAX_ABS, PR_REL_L1, ok_partitions, rel_l1

pytestmark = pytest.mark.gpu


def star(gg, n, seed):
    """One destination with n - 1 in-edges beside a few scattered edges."""
    rng = np.random.default_rng(seed)
    src = np.concatenate([np.arange(1, n), rng.integers(0, n, 300)])
    dst = np.concatenate([np.zeros(n - 1, np.int64), rng.integers(0, n, 300)])
    key = np.unique(src * n + dst)
    src, dst = key // n, key % n
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return gg.HostGraph.from_csr(off, dst, rng.integers(1, 101, len(dst)), symmetric=False)


# one tile per partition of up to 2^20 edges: whole tiles, tiles of several
# items, items that end inside a 256-edge block row, a tile of one destination
@pytest.mark.parametrize("kernel", [6, 7])
@pytest.mark.parametrize("shape", ["rmat8", "rmat13", "rmat15", "star"])
def test_split_tiles(gg, orc, shape, kernel):
    if shape == "star":
        hg = star(gg, 40_001, 5)
    else:
        hg = gg.HostGraph.rmat(int(shape[4:]), 16, seed=31, symmetric=False).add_weights(gg.W_INT32, seed=2, lo=1, hi=100)
    g = gg.Graph(hg, partitions=ok_partitions(hg, 3), tile_edges=1 << 20)
    g.set_tuning(gg.TUNE_COO_KERNEL, kernel)
    g.set_dense_policy(2)
    og = orc.Graph.from_host(hg)
    start = int(np.argmax(hg.degrees()))
    for _ in range(2):  # the slabs are clear again after a run
        np.testing.assert_array_equal(g.components()[0], og.cc()[0])
        np.testing.assert_array_equal(g.bellman_ford(start)[0], og.bellman_ford(start)[0])
        np.testing.assert_array_equal(g.bfs(start)[1], og.bfs(start)[1])
        if shape == "star":  # its frontier empties, where the reference aborts
            with pytest.raises(gg.GGError, match="Sizes Don't match"):
                g.pagerank(10)
        else:
            r, o = g.pagerank(10)[0], og.pagerank(10)[0]
            assert rel_l1(r, o) <= PR_REL_L1 and np.abs(r - o).max() <= PR_MAX_ABS
        assert rel_l1(g.pagerank_delta()[0], og.pagerank_delta()[0]) <= 1e-4
        assert rel_l1(g.spmv()[0], og.spmv()[0]) <= 1e-6
        dep, paths, _ = g.bc(start)
        odep, opaths, _ = og.bc(start)
        np.testing.assert_allclose(paths, opaths, rtol=1e-6)
        ok = np.isfinite(odep)
        assert rel_l1(dep[ok], odep[ok]) <= 1e-4
    g.close()
