"""GG_PR_CUDA_GRAPH in the modes that run as several launches: the captured call, its
repeats, other parameters, and a capture after a buffer was regrown in between all
give the launches' ranks (fixed-point and quantised ranks to the bit); and the
one-launch pull stops where the launches stop."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EXACT = ("pull_q16", "pull_fx64", "pull_q8")


@pytest.mark.parametrize("mode,kw", [("pull", dict(storage="bf16")), ("pull_q16", {}), ("pull_q8", {}), ("pull_fx64", {}),
                                     ("push", {}), ("pull", dict(hot=True))])
def test_replayed_graph_gives_the_launches_ranks(gpu, mode, kw):
    g = gpu.Graph.rmat(14, 16)
    dg = gpu.DeviceGraph(g, gpu.MAP_IN | gpu.MAP_OUT)
    # sums in arrival order: 20 iterations of rows of at most n terms, and four roundings
    # more each (16-bit deltas carry on what they round)
    tol = 20 * (int(np.diff(g.arrays()["in_off"].astype(np.int64)).max()) + 4) * 2.0 ** -24

    def check(**more):
        plain, rp = dg.pagerank(mode, **kw, **more)
        for _ in range(3):  # captured (or replayed), then replayed
            got, rg = dg.pagerank(mode, cuda_graph=True, **kw, **more)
            assert (rg["iterations"], rg["launches"]) == (rp["iterations"], rp["launches"])
            if mode in EXACT:
                np.testing.assert_array_equal(got, plain)
            else:
                np.testing.assert_allclose(got, plain, rtol=tol, atol=0)

    check(iterations=20, epsilon=0.0)
    check(iterations=7, epsilon=0.0)
    dg.bfs(0, "push")  # regrows work buffers that the captured graph writes
    check(iterations=7, epsilon=0.0)
    check(iterations=20, epsilon=0.0)
    dg.free()
    g.free()


@pytest.mark.parametrize("V,E", [(300, 3000), (3000, 40000), (40000, 300000)])
def test_one_launch_stops_where_the_launches_stop(gpu, V, E):
    """Unit out-degrees and damping that halves: every rank is a dyadic number and
    every sum exact in FP32, so the one launch and the launches agree to the bit, in
    the ranks, the active count and the iteration at which no rank moves by epsilon."""
    src = np.arange(V)
    dst = np.arange(V) // 2
    g = gpu.Graph.from_edges(src.astype(np.uint32), dst.astype(np.uint32), num_vertices=V)
    dg = gpu.DeviceGraph(g, gpu.MAP_IN)
    for its, eps in ((30, 2.0 ** -9), (30, 2.0 ** -5), (30, 0.0), (3, 2.0 ** -9)):
        a, ra = dg.pagerank("pull", iterations=its, epsilon=eps, damp=0.5)
        b, rb = dg.pagerank("pull", iterations=its, epsilon=eps, damp=0.5, profile=True)
        assert ra["launches"] == 1 < rb["launches"]
        np.testing.assert_array_equal(a, b)
        assert (ra["iterations"], ra["active"]) == (rb["iterations"], rb["active"])
        assert ra["error_total"] == rb["error_total"] and ra["rank_sum"] == rb["rank_sum"]
    dg.free()
    g.free()
