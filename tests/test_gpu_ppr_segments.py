"""The k-column pull's segments (128 edges of a block at 64 columns, 64 at 32):
rows that end at, cross and span segment and block boundaries, against FP64."""
import numpy as np
import pytest

from conftest import ok_partitions, rel_l1
from test_gpu_segreduce import graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [32, 64])
@pytest.mark.parametrize("degrees", [
    [1, 1], [63, 1] + [1] * 70, [64, 64, 128, 0, 1] + [0] * 140, [65, 63, 127, 129] + [2] * 140, [256, 256] + [0] * 300,
    [257, 255, 700] + [1] * 700, [7, 9] * 40, [1] * 600])
def test_rows_at_segment_borders(gg, orc, degrees, k):
    hg = graph(gg, degrees)
    g = gg.Graph(hg, partitions=ok_partitions(hg, 4))
    og = orc.Graph.from_host(hg)
    rng = np.random.default_rng(hg.n)
    tele = np.where(rng.random((hg.n, 1)) < 0.3, 0, rng.random((hg.n, k))).astype(np.float32)  # some rows are zero
    seeds = rng.integers(0, hg.n, k).astype(np.uint32)
    onehot = np.zeros((hg.n, k), np.float32)
    onehot[seeds, np.arange(k)] = 1
    for iters in (0, 1, 2, 3, 8):
        for given, x in ((tele, g.ppr_k(k, iters=iters, damping=0.85, tele=tele)[0]),
                         (onehot, g.ppr_k(k, iters=iters, damping=0.85, seeds=seeds)[0])):
            for j in (0, 1, 3, k // 2, k - 1):
                o = og.ppr(iters, 0.85, given[:, j].astype(np.float64))
                # rows of at most 700 positive FP32 terms, 8 iterations: 8 * 700 * 2^-24 = 3.3e-4 at worst, 1e-5 as
                # the other k-column tests have it
                assert rel_l1(x[:, j], o) <= 1e-5
    g.close()
