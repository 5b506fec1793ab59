"""Batches right after their creation: the copies of the host arrays, the
kernels that renumber them and the first traversal are one sequence."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(gg, orc, hgs, b):
    src = np.array([h.n // 2 for h in hgs], np.uint32)
    lev, run = b.bfs(src)
    trav = 0
    for h, s, lv in zip(hgs, src, b.split(lev)):
        _, olev, ost = orc.Graph.from_host(h).bfs(int(s))
        np.testing.assert_array_equal(lv, olev)
        trav += ost.edges_traversed
    assert run.edges_traversed == trav


@pytest.mark.parametrize("count", [1, 3, 700])
def test_first_traversal_after_creation(gg, orc, count):
    hgs = [gg.HostGraph.rmat(17 if count == 1 else 5 + i % 4, 12, seed=i, symmetric=False) for i in range(count)]
    for _ in range(3):
        b = gg.GraphBatch(hgs)
        check(gg, orc, hgs, b)
        b.close()


class Late:
    """hg with `lead` more entries before its first edge: offsets[0] = lead."""

    def __init__(self, gg, hg, lead):
        self.hg = hg
        self.offsets = hg.offsets + np.uint32(lead)
        self.indices = np.concatenate([np.full(lead, hg.n - 1, np.uint32), hg.indices])
        p = C.POINTER(C.c_uint32)
        self.c = gg.HostGraphC(hg.n, len(self.indices), 0, gg.W_NONE, self.offsets.ctypes.data_as(p),
                               self.indices.ctypes.data_as(p), None)


@pytest.mark.parametrize("leads", [(5, 0, 0), (0, 7, 300), (1, 1, 1)])
def test_offsets_that_start_late(gg, orc, leads):
    hgs = [gg.HostGraph.rmat(9, 8, seed=i, symmetric=False) for i in range(len(leads))]
    late = [Late(gg, h, k) for h, k in zip(hgs, leads)]
    b = gg.GraphBatch(late)
    assert b.total_edges == sum(h.m for h in hgs) + sum(leads)
    check(gg, orc, hgs, b)
    b.close()
    late[0].c.offsets[0] = late[0].c.m + 1
    with pytest.raises(gg.GGError) as e:
        gg.GraphBatch(late)
    assert e.value.code == gg.ERR_INVALID_ARG


def test_runs_of_vertices_without_in_edges(gg, orc):
    """In-lists at the ends of long empty runs: before the first edge, between
    two, behind the last, and graphs with none at all."""
    def fan(n, u, dst):
        off = np.zeros(n + 1, np.uint32)
        off[u + 1:] = len(dst)
        return gg.HostGraph.from_csr(off, np.array(dst, np.uint32))
    n = 70_001
    none = gg.HostGraph.from_csr(np.zeros(n + 1, np.uint32), np.zeros(0, np.uint32))
    every = np.arange(0, n, 3)  # a first level dense enough for the bottom-up walk
    hgs = [none, fan(n, n // 2, [n - 1]), fan(n, n // 2, [0, n - 1]), none, fan(n, n // 2, every), none]
    b = gg.GraphBatch(hgs)
    check(gg, orc, hgs, b)
    b.close()
