"""The sparse push step where a CTA takes several 256-edge windows: the next
window's first slot follows from the staged ones, unless a run of members
without out-edges reaches past them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 300_000


def degrees(kind):
    rng = np.random.default_rng(5)
    if kind == "ones":  # a window is exactly a stage of slots
        return np.ones(N, np.int64)
    if kind == "mixed":
        deg = rng.integers(0, 13, N)
        deg[rng.integers(0, N, 40)] = rng.integers(200, 4000, 40)
        return deg
    if kind == "aligned":  # slots that start at window borders
        return np.tile([256, 1, 255, 0, 512, 128, 128, 0, 0, 3, 253], N // 11 + 1)[:N] * (np.arange(N) < 60_000)
    deg = np.where(rng.random(N) < 0.3, rng.integers(1, 30, N), 0)  # "gaps": runs of several stages
    for a in rng.integers(0, N - 2000, 30):
        deg[a:a + rng.integers(200, 1500)] = 0
    return deg


@pytest.mark.parametrize("kind", ["ones", "mixed", "aligned", "gaps"])
@pytest.mark.parametrize("part", [1.0, 0.6])
def test_push_sums(gg, kind, part):
    rng = np.random.default_rng(int(part * 10))
    deg = degrees(kind)
    dst = rng.integers(0, N, int(deg.sum()))
    off = np.concatenate([[0], np.cumsum(deg)])
    hg = gg.HostGraph.from_csr(off.astype(np.uint32), dst.astype(np.uint32))
    g = gg.Graph(hg, partitions=4)
    queue = np.arange(N) if part == 1.0 else np.sort(rng.permutation(N)[:int(part * N)])
    x = rng.integers(-4, 5, N).astype(np.float32)  # small integers: every sum is exact
    xd, yd = gg.DeviceArray(g, np.float32, x), gg.DeviceArray(g, np.float32, np.zeros(N, np.float32))
    out = g.edge_map(g.frontier_from_list(queue.astype(np.uint32)), gg.F_SPMV, gg.PairArgs(xd.ptr, yd.ptr),
                     flags=gg.EM_FORCE_SPARSE)
    src = np.repeat(np.arange(N), deg)
    on = np.zeros(N, bool)
    on[queue] = True
    keep = on[src]
    want = np.bincount(dst[keep], weights=x[src[keep]], minlength=N)
    touched = np.bincount(dst[keep], minlength=N) > 0
    np.testing.assert_array_equal(yd.download(), want)
    np.testing.assert_array_equal(out.mask(), touched)
    assert out.stats() == (int(touched.sum()), int(deg[touched].sum()))
    out.close()
    g.close()
