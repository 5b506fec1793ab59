"""The sparse push step (k_push, k_scan_one) at the borders of its queue scan
and edge windows, with runs of members that have no out-edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 12_000


@pytest.fixture(scope="module")
def graph(gg):
    rng = np.random.default_rng(11)
    deg = np.where(rng.random(N) < 0.15, rng.integers(1, 12, N), 0)  # most vertices have no out-edges
    deg[[0, 5000, N - 1]] = [700, 256, 1]
    dst = np.concatenate([rng.choice(N, d, replace=False) for d in deg])
    off = np.concatenate([[0], np.cumsum(deg)])
    w = rng.integers(1, 9, len(dst))
    hg = gg.HostGraph.from_csr(off, dst, w)
    return gg.Graph(hg, partitions=4), off, dst, w


@pytest.mark.parametrize("members", [1, 2, 255, 256, 257, 511, 2049, 8191, 8192, 8193, N])
@pytest.mark.parametrize("front", [True, False])
def test_push_sums(gg, graph, members, front):
    g, off, dst, w = graph
    rng = np.random.default_rng(members)
    rest = rng.permutation(np.arange(1, N))
    # the hub first in the queue, or last behind members most of which have no out-edges
    queue = np.concatenate([[0], rest[:members - 1]] if front else [rest[:members - 1], [0]]).astype(np.uint32)
    x = rng.integers(-4, 5, N).astype(np.float32)  # small integers: every sum is exact
    xd, yd = gg.DeviceArray(g, np.float32, x), gg.DeviceArray(g, np.float32, 0.0)
    out = g.edge_map(g.frontier_from_list(queue), gg.F_SPMV, gg.PairArgs(xd.ptr, yd.ptr), flags=gg.EM_FORCE_SPARSE)
    want, touched = np.zeros(N), np.zeros(N, np.uint8)
    for s in queue:
        e = slice(off[s], off[s + 1])
        want[dst[e]] += x[s] * w[e]
        touched[dst[e]] = 1
    np.testing.assert_array_equal(yd.download(), want)
    np.testing.assert_array_equal(out.mask(), touched)
    assert out.stats() == (int(touched.sum()), int(np.diff(off)[touched == 1].sum()))
    assert g.last_edge_map_stats().kind == 1
