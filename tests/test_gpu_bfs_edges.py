"""BFS where a step's shared-memory structures reach their limits: a first
bottom-up frontier from one vertex to a third of the graph, blocks that claim
more vertices than their local queue holds, and hubs whose edges are dealt to
the grid.  Levels are compared exactly with the oracle's or the known ones."""
import numpy as np
import pytest

from graphs import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 8191, 8192, 8193, 20000])
def test_first_bottom_up_frontier(gpu, orc, n):
    """The source has n neighbours; a bottom-up step follows at once."""
    rng = np.random.default_rng(n)
    V, m = 60000, 400
    a = np.concatenate([np.zeros(n, np.int64), rng.integers(1, V, m * 10), rng.integers(1, n + 1, 20000)])
    b = np.concatenate([np.arange(1, n + 1), rng.integers(1, V, m * 10), rng.integers(1, V, 20000)])
    src, dst = np.concatenate([a, b]).astype(np.uint32), np.concatenate([b, a]).astype(np.uint32)
    g, o = pair(gpu, orc, gpu.Graph.from_edges(src, dst, num_vertices=V))
    dg = gpu.DeviceGraph(g, gpu.MAP_IN | gpu.MAP_OUT)
    for mode, om in (("do", 2), ("push", 1)):
        parents, dist, res = dg.bfs(0, mode)
        _, rd, info = orc.bfs(o, om, 0)
        np.testing.assert_array_equal(dist, rd)
        assert res["processed_nodes"] == info["processed_nodes"]
        assert res["edges_examined"] == info["edges_examined"]
        reached = np.flatnonzero((parents >= 0) & (np.arange(V) != 0))
        assert (dist[parents[reached]] + 1 == dist[reached]).all()


@pytest.mark.parametrize("mids,each", [(3, 5000), (4200, 1000), (5000, 65)])
def test_two_levels_of_many_claims(gpu, mids, each):
    """0 -> mids -> mids * each leaves: with more hubs than the deferred list
    holds, single warps claim thousands of vertices each."""
    leaves = mids * each
    V = 1 + mids + leaves
    src = np.concatenate([np.zeros(mids, np.uint32), np.repeat(np.arange(1, mids + 1, dtype=np.uint32), each)])
    dst = np.arange(1, V, dtype=np.uint32)
    rng = np.random.default_rng(mids)
    perm = rng.permutation(leaves).astype(np.uint32) + np.uint32(1 + mids)
    dst[mids:] = perm
    g = gpu.Graph.from_edges(src, dst, num_vertices=V)
    dg = gpu.DeviceGraph(g, gpu.MAP_IN | gpu.MAP_OUT)
    want = np.full(V, 2, np.uint32)
    want[0], want[1:1 + mids] = 0, 1
    parent = np.empty(V, np.int32)
    parent[0], parent[1:1 + mids] = 0, 0
    parent[dst[mids:]] = src[mids:]
    for mode in ("push", "do", "push_bitmap"):
        parents, dist, res = dg.bfs(0, mode)
        np.testing.assert_array_equal(dist, want)
        np.testing.assert_array_equal(parents, parent)
        assert res["processed_nodes"] == V


@pytest.mark.parametrize("hubs,degree", [(4200, 65), (4096, 600), (4097, 513), (9000, 520)])
def test_more_hubs_than_the_first_list(gpu, orc, hubs, degree):
    """A frontier of `hubs` vertices with `degree` edges each, past the first
    list's 4,096 and the second's chunks of as many."""
    rng = np.random.default_rng(hubs)
    V = 60000
    a = np.concatenate([np.zeros(hubs, np.int64), np.repeat(np.arange(1, hubs + 1), degree)])
    b = np.concatenate([np.arange(1, hubs + 1), rng.integers(hubs + 1, V, hubs * degree)])
    g, o = pair(gpu, orc, gpu.Graph.from_edges(a.astype(np.uint32), b.astype(np.uint32), num_vertices=V))
    dg = gpu.DeviceGraph(g, gpu.MAP_IN | gpu.MAP_OUT)
    for mode, om in (("push", 1), ("push_bitmap", 3), ("do", 2)):
        parents, dist, res = dg.bfs(0, mode)
        _, rd, info = orc.bfs(o, om, 0)
        np.testing.assert_array_equal(dist, rd)
        assert res["processed_nodes"] == info["processed_nodes"]
        reached = np.flatnonzero((parents >= 0) & (np.arange(V) != 0))
        assert (dist[parents[reached]] + 1 == dist[reached]).all()
    dg.free()
