"""Batches as one union graph: levels that finish in the whole-GPU loop and
levels handed to one CTA per graph, into pageable and page-locked arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def edgeless(gg, n):
    return gg.HostGraph.from_csr(np.zeros(n + 1, np.uint32), np.zeros(0, np.uint32))


def graphs(gg, kind):
    if kind == "deep":  # handed over after the first level
        return [gg.HostGraph.grid(s, 0.0, seed=s) for s in (2, 17, 33, 64)]
    if kind == "wide":  # ends in the whole-GPU loop
        return [gg.HostGraph.rmat(13, 16, seed=7, symmetric=False)]
    if kind == "edgeless":
        return [edgeless(gg, n) for n in (1, 2, 31, 32, 33, 257)]
    return [gg.HostGraph.rmat(14, 24, seed=3), gg.HostGraph.grid(40, 0.01, seed=2), edgeless(gg, 300),
            gg.HostGraph.rmat(4, 2, seed=9, symmetric=False), edgeless(gg, 1)]


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("kind", ["deep", "wide", "edgeless", "mixed"])
def test_union_levels(gg, orc, kind, pinned):
    hgs = graphs(gg, kind)
    b = gg.GraphBatch(hgs)
    keep = gg.PinnedArray(b.total_vertices, np.int32)
    out = keep.array if pinned else np.empty(b.total_vertices, np.int32)
    for rep in range(2):
        src = np.array([0 if rep == 0 else h.n - 1 for h in hgs], np.uint32)
        out[:] = -7
        _, run = b.bfs(src, out)
        trav = 0
        for h, s, lv in zip(hgs, src, b.split(out)):
            _, olev, ost = orc.Graph.from_host(h).bfs(int(s))
            np.testing.assert_array_equal(lv, olev)
            trav += ost.edges_traversed
        assert run.edges_traversed == trav
    b.close()
