"""Hubs in sparse BFS levels: a frontier vertex whose edges span many of the
windows a level is cut into (512 edges each), appended by a push level, by the
seeding of a traversal and where a bitmap level turns into a queue."""
import numpy as np
import pytest

from conftest import ok_partitions

pytestmark = pytest.mark.gpu

ER = 200_000  # vertices of the random part, where levels turn dense


def csr(gg, n, src, dst):
    order = np.argsort(src, kind="stable")
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(src, minlength=n))
    return gg.HostGraph.from_csr(off, dst[order].astype(np.uint32))


def hub_graph(gg, degree):
    """A random part; six chains of 1..6 vertices out of it that end in a hub of
    `degree` out-edges each; one more hub behind a vertex of its own (the
    start of the sparse traversal), with two leaves that go on."""
    rng = np.random.default_rng(degree)
    edges = (24 if degree > 50_000 else 8) * ER
    src, dst = [rng.integers(0, ER, edges)], [rng.integers(0, ER, edges)]
    nxt = ER
    def edge(u, v):
        src.append(np.atleast_1d(u))
        dst.append(np.atleast_1d(v))
    def hub(u, tail):
        nonlocal nxt
        h, nxt = nxt, nxt + 1
        edge(u, h)
        edge(np.full(degree, h), nxt + np.arange(degree))
        if tail:
            edge(nxt + degree - 1, nxt + degree)
            edge(nxt + degree, nxt + degree + 1)
        nxt += degree + 2
        return h
    for length in range(1, 7):
        u = int(rng.integers(0, ER))
        for _ in range(length):
            edge(u, nxt)
            u, nxt = nxt, nxt + 1
        hub(u, length % 2)
    start, nxt = nxt, nxt + 1
    lone = hub(start, True)
    return csr(gg, nxt, np.concatenate(src), np.concatenate(dst)), start, lone


@pytest.mark.parametrize("loop", [1, 2])
@pytest.mark.parametrize("degree", [512, 513, 40 * 512 - 1, 256 * 512, 256 * 512 + 1, 300 * 512 + 7])
def test_hubs(gg, orc, degree, loop):
    hg, start, lone = hub_graph(gg, degree)
    assert degree + 2 <= hg.m // 20  # the hub's level stays sparse
    g = gg.Graph(hg, partitions=ok_partitions(hg, 16))
    g.set_tuning(gg.TUNE_DEVICE_LOOP, loop)
    og = orc.Graph.from_host(hg)
    for s in (start, lone, 5):
        par, lev, run = g.bfs(s)
        _, olev, ost = og.bfs(s)
        np.testing.assert_array_equal(lev, olev)
        assert run.edges_traversed == ost.edges_traversed
        v = np.flatnonzero(olev > 0)
        np.testing.assert_array_equal(olev[par[v]], olev[v] - 1)
    g.close()


@pytest.mark.parametrize("degree", [4 * 512 + 1, 300 * 512 + 7])
def test_hubs_of_a_batch(gg, orc, degree):
    hg, start, lone = hub_graph(gg, degree)
    hgs = [hg, gg.HostGraph.rmat(8, 8, seed=1), hg, hg]
    b = gg.GraphBatch(hgs)
    src = [lone, 0, start, 5]
    lev, _ = b.bfs(src)
    for h, s, lv in zip(hgs, src, b.split(lev)):
        np.testing.assert_array_equal(lv, orc.Graph.from_host(h).bfs(s)[1])
    b.close()
