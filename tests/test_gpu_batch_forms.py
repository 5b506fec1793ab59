"""The forms a batch runs in: the union graph's whole-GPU loop first, one CTA
per graph on the union's numbering, one CTA per graph on separate numberings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def edgeless(gg, n):
    return gg.HostGraph.from_csr(np.zeros(n + 1, np.uint32), np.zeros(0, np.uint32))


def graphs(gg):
    return [gg.HostGraph.rmat(13, 16, seed=3), edgeless(gg, 1), gg.HostGraph.grid(33, 0.01, seed=2), edgeless(gg, 300),
            gg.HostGraph.rmat(4, 2, seed=9, symmetric=False), gg.HostGraph.rmat(10, 8, seed=1, symmetric=False)]


@pytest.mark.parametrize("form", ["AUTO", "PER_CTA", "SEPARATE"])
def test_forms(gg, orc, form):
    hgs = graphs(gg)
    b = gg.GraphBatch(hgs, getattr(gg, "BATCH_" + form))
    keep = gg.PinnedArray(b.total_vertices, np.int32)
    for rep in range(2):
        src = np.array([0 if rep == 0 else h.n - 1 for h in hgs], np.uint32)
        for out in (np.full(b.total_vertices, -7, np.int32), keep.array):
            _, run = b.bfs(src, out)
            assert (run.kernels > 1) == (form == "AUTO")
            trav = 0
            for h, s, lv in zip(hgs, src, b.split(out)):
                _, olev, ost = orc.Graph.from_host(h).bfs(int(s))
                np.testing.assert_array_equal(lv, olev)
                trav += ost.edges_traversed
            assert run.edges_traversed == trav
    b.close()


@pytest.mark.parametrize("form", [-1, 3])
def test_unknown_form(gg, form):
    with pytest.raises(gg.GGError) as e:
        gg.GraphBatch([edgeless(gg, 3)], form)
    assert e.value.code == gg.ERR_INVALID_ARG


@pytest.mark.parametrize("pinned", [False, True])
def test_barrier_timeout_runs_without_barriers(gg, orc, pinned):
    """With no probe at all, the CTAs that reach the first grid barrier before
    the last one return at once; the call then gives the result all the same."""
    hgs = [gg.HostGraph.rmat(15, 16, seed=3), gg.HostGraph.rmat(12, 16, seed=4, symmetric=False), edgeless(gg, 40)]
    b = gg.GraphBatch(hgs, wait_budget=-1)
    keep = gg.PinnedArray(b.total_vertices, np.int32)
    out = keep.array if pinned else np.empty(b.total_vertices, np.int32)
    for s in (0, 7, 0):
        out[:] = -7
        _, run = b.bfs(np.full(3, s, np.uint32), out)
        assert run.kernels == 5
        trav = 0
        for h, lv in zip(hgs, b.split(out)):
            _, olev, ost = orc.Graph.from_host(h).bfs(s)
            np.testing.assert_array_equal(lv, olev)
            trav += ost.edges_traversed
        assert run.edges_traversed == trav
    b.close()


@pytest.mark.parametrize("n,kernels", [(3072, 1), (3073, 4)])
def test_small_graphs_skip_the_union(gg, orc, n, kernels):
    """n vertices in a path: n + m = 2 n - 1, on both sides of 6144."""
    off = np.minimum(np.arange(n + 1), n - 1).astype(np.uint32)
    hgs = [gg.HostGraph.from_csr(off, np.arange(1, n, dtype=np.uint32)), edgeless(gg, 5)]
    b = gg.GraphBatch(hgs)
    lev, run = b.bfs([n - 40, 2])
    assert run.kernels == kernels
    for h, s, lv in zip(hgs, (n - 40, 2), b.split(lev)):
        np.testing.assert_array_equal(lv, orc.Graph.from_host(h).bfs(s)[1])
    b.close()
