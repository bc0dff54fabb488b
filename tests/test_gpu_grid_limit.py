"""The one-launch pull's grid barriers wait up to gg_set_barrier_limit_us.  When a
wait runs out the kernel ends early and the call runs as separate launches: it
still succeeds, with their ranks, and the next call is one launch again."""
import numpy as np
import pytest

from fpcheck import assert_fp_as_accurate
from graphs import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iterations", [20, 12000])  # the records with the results, and on their own
def test_barrier_wait_runs_out_and_the_launches_take_over(gpu, orc, iterations):
    rng = np.random.default_rng(5)
    V, E = 40001, 2000003
    src, dst = (rng.random(E) ** 3 * V).astype(np.uint32), (rng.random(E) ** 2 * V).astype(np.uint32)
    g, o = pair(gpu, orc, gpu.Graph.from_edges(src, dst, num_vertices=V))
    dg = gpu.DeviceGraph(g, gpu.MAP_IN)

    def check(ranks, res, what):
        """as accurate as the reference's loop after as many iterations"""
        done = min(res["iterations"] + 1, iterations)
        assert done <= 200
        ref, _ = orc.pagerank(o, 0, done, 0.0)
        assert_fp_as_accurate(ranks, ref, orc.pagerank_f64(o, done), what)

    L = gpu.lib()
    L.gg_set_barrier_limit_us(1)
    try:
        ranks, res = dg.pagerank("pull", iterations=iterations, epsilon=1e-4)
    finally:
        L.gg_set_barrier_limit_us(0)
    assert res["launches"] > 2
    check(ranks, res, "by launches")
    ranks, res = dg.pagerank("pull", iterations=iterations, epsilon=1e-4)
    assert res["launches"] == 1
    check(ranks, res, "one launch")
    dg.free()
    g.free()
