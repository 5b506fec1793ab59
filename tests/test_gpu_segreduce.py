"""Row reductions over 256-edge blocks (k_seg_reduce) through weighted
PageRank: rows that end at lane and block borders, and blocks with a ragged
end, against FP64."""
import numpy as np
import pytest

from conftest import ok_partitions

pytestmark = pytest.mark.gpu


def graph(gg, degrees):
    """Vertex v has degrees[v] in-edges, from the vertices after it."""
    n = len(degrees)
    dst = np.repeat(np.arange(n), degrees)
    src = np.concatenate([(v + 1 + np.arange(d)) % n for v, d in enumerate(degrees)]).astype(np.int64)
    order = np.lexsort((dst, src))
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return gg.HostGraph.from_csr(off, dst[order])


@pytest.mark.parametrize("degrees", [
    [1], [2, 0, 3], [255, 1] + [0] * 300, [256] + [0] * 300, [257, 0, 255] + [0] * 300, [8] * 33, [7, 9] * 40, [1] * 600,
    [300] * 5 + [1] * 301, [700] + [1] * 800, [31, 33, 1, 0, 64] * 30])
def test_rows_at_borders(gg, orc, degrees):
    hg = graph(gg, degrees)
    n, m = hg.n, hg.m
    rng = np.random.default_rng(n + m)
    w, tele, x0, c = (rng.uniform(0.1, 1, k).astype(np.float32) for k in (m, n, n, n))
    g = gg.Graph(hg, partitions=ok_partitions(hg, 4))
    og = orc.Graph.from_host(hg)
    wpr = gg.WeightedPageRank(g, 1, 1.0, 1, False)  # one step: a plain row sum of positive terms
    x, _ = wpr.forward(w, tele, x0=x0)
    gw, _, gx, _ = wpr.backward(c)
    ox = og.wpr_forward(w, tele, 1, 1.0, x0=x0)
    ogw, _, ogx = og.wpr_backward(w, tele, 1, 1.0, c, x0=x0)
    # at most 800 positive FP32 terms a row: 800 * 2^-24 = 4.8e-5 relative
    for a, b in ((x, ox), (gw, ogw), (gx, ogx)):
        np.testing.assert_allclose(a, b, rtol=5e-5, atol=0)
    wpr.close()
