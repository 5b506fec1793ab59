"""A BFS whose loop gives up (its barrier waits driven to expiry, as in
test_gpu_timeout.py) leaves the caller's arrays as they were."""
import ctypes as C

import numpy as np
import pytest

from conftest import ok_partitions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["pageable", "pinned", "asynchronous"])
@pytest.mark.parametrize("order", [0, 1])
def test_arrays_untouched_after_a_timeout(gg, orc, mode, order):
    hg = gg.HostGraph.rmat(14, 16, seed=3, symmetric=True)
    g = gg.Graph(hg, partitions=ok_partitions(hg, 16), vertex_order=order)
    keep = [gg.PinnedArray(hg.n, np.int32) for _ in range(2)]
    par, lev = [k.array for k in keep] if mode != "pageable" else [np.empty(hg.n, np.int32) for _ in range(2)]
    g.set_tuning(gg.TUNE_ASYNC_RESULTS, int(mode == "asynchronous"))
    for want_par, want_lev in ((1, 1), (1, 0), (0, 1)):
        par[:], lev[:] = -7, -8
        g.set_tuning(gg.TUNE_LOOP_WAIT_BUDGET, 0)
        st = gg.RunStats()
        args = [C.c_void_p(a.ctypes.data) if w else None for a, w in ((par, want_par), (lev, want_lev))]
        assert gg.lib.gg_bfs(g.h, 100, *args, C.byref(st)) == gg.ERR_TIMEOUT
        g.synchronize()
        assert (par == -7).all() and (lev == -8).all()
        g.set_tuning(gg.TUNE_LOOP_WAIT_BUDGET, 1 << 22)
        gg.check(gg.lib.gg_bfs(g.h, 100, *args, C.byref(st)), "gg_bfs")
        g.synchronize()
        _, olev, _ = orc.Graph.from_host(hg).bfs(100)
        if want_lev:
            np.testing.assert_array_equal(lev, olev)
        if want_par:
            np.testing.assert_array_equal(par >= 0, olev >= 0)
            v = np.flatnonzero(olev > 0)
            np.testing.assert_array_equal(olev[par[v]], olev[v] - 1)
    g.set_tuning(gg.TUNE_ASYNC_RESULTS, 0)
    g.close()
