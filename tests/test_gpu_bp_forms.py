"""gg_bp's two reduction kernels: streams that both finish in one wave of
warps, that only k_seg_scan does, and that neither does, with rows up to a
block and one longer."""
import numpy as np
import pytest

from conftest import ok_partitions

pytestmark = pytest.mark.gpu


def graph(gg, degrees):
    """Vertex v has degrees[v] in-edges, from the vertices after it."""
    n = len(degrees)
    dst = np.repeat(np.arange(n), degrees)
    src = (dst + 1 + np.arange(len(dst)) - np.repeat(np.cumsum(degrees) - degrees, degrees)) % n
    order = np.lexsort((dst, src))
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return gg.HostGraph.from_csr(off, dst[order])


@pytest.mark.parametrize("blocks", [4000, 6000, 11000])
@pytest.mark.parametrize("longest", [256, 257])
def test_products(gg, orc, blocks, longest):
    pattern = np.array([3, 0, 31, 33, 1, 64, 255, 7, 9, 0, 2, 8, 8, 8, 1, 1, 1, 128, 5, 40])
    reps = blocks * 256 // int(pattern.sum())
    degrees = np.concatenate([np.tile(pattern, reps), [longest, 1]])
    hg = graph(gg, degrees)
    rng = np.random.default_rng(blocks)
    vp = rng.uniform(0.6, 0.8, (hg.n, 2)).astype(np.float32)
    ep = rng.uniform(0.65, 0.75, (hg.m, 2, 2)).astype(np.float32)
    g = gg.Graph(hg, partitions=ok_partitions(hg, 4))
    out, _ = g.bp(1, vp, ep)
    # iteration 1 starts from products of 1: belief_e[i] = sum_k vp[d][k] ep[e][i][k]
    # over d's in-edges, in order of their slots
    belief = np.einsum("ek,eik->ei", np.repeat(vp.astype(np.float64), degrees, axis=0), ep.astype(np.float64))
    logs = np.concatenate([np.zeros((1, 2)), np.cumsum(np.log(belief), axis=0)])
    end = np.cumsum(degrees)
    want = np.exp(logs[end] - logs[end - degrees])
    # 257 factors of 3 roundings each, 257 products: 1028 * 2^-24 = 6.2e-5
    np.testing.assert_allclose(out, want, rtol=1e-4)
    g.close()
