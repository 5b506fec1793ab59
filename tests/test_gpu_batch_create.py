"""Batches right after their creation: the copies of the host arrays, the
kernels that renumber them and the first traversal are one sequence."""
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
