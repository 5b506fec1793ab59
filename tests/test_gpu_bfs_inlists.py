"""The copy of the in-lists with hub sources first is built where the program
asks for it, by its next BFS, and not otherwise."""
import numpy as np
import pytest

from conftest import ok_partitions

pytestmark = pytest.mark.gpu


def test_copy_is_built_on_request(gg, orc):
    hg = gg.HostGraph.rmat(14, 16, seed=5, symmetric=False)
    g = gg.Graph(hg, partitions=ok_partitions(hg, 16))
    og = orc.Graph.from_host(hg)
    assert g.get_tuning(gg.TUNE_EARLY_KERNEL) == 3

    def bfs(s):
        np.testing.assert_array_equal(g.bfs(s)[1], og.bfs(s)[1])
        return g.info().device_bytes

    plain = bfs(0)
    assert [bfs(s) for s in (0, 100, 0, 7)] == [plain] * 4
    g.set_tuning(gg.TUNE_EARLY_KERNEL, 3)
    assert g.info().device_bytes == plain  # the call that uses it builds it
    held = bfs(0)
    assert held >= plain + 4 * hg.m
    g.set_tuning(gg.TUNE_EARLY_KERNEL, 2)
    assert bfs(100) == held
    g.set_tuning(gg.TUNE_EARLY_KERNEL, 3)
    assert [bfs(s) for s in (100, 0)] == [held] * 2
    g.close()
