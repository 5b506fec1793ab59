"""What the last edgeMap of a call reports does not depend on whether its
rounds ran in the captured graph."""
import pytest

from conftest import ok_partitions

pytestmark = pytest.mark.gpu

FIELDS = ("kind", "frontier_active", "frontier_out_edges", "output_active", "output_out_edges")


@pytest.mark.parametrize("policy,kind", [(0, 2), (2, 3)])
@pytest.mark.parametrize("shape", ["rmat", "er"])
def test_last_round(gg, shape, policy, kind):
    hg = gg.HostGraph.rmat(13, 16, seed=62) if shape == "rmat" else gg.HostGraph.er(1 << 13, 1 << 16, seed=7, symmetric=True)
    g = gg.Graph(hg, partitions=ok_partitions(hg, 16))
    g.set_tuning(gg.TUNE_SPARSE_DIV, 1 << 20)  # every round is dense, the last one below m / 2
    g.set_dense_policy(policy)
    seen = []
    for graph in (0, 1):
        g.set_tuning(gg.TUNE_ROUND_GRAPH, graph)
        _, run = g.components()  # its pull reads the previous labels alone: the rounds are the same
        s = g.last_edge_map_stats()
        seen.append((run.rounds, run.edges_traversed) + tuple(getattr(s, f) for f in FIELDS))
    assert seen[0] == seen[1]
    assert seen[1][2] == kind and 0 < seen[1][4] <= hg.m // 2
    g.close()
