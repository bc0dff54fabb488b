"""PageRank pull in one cooperative launch (a CTA per SM) where its shares
change: the smallest graph it takes, edges per thread at and past multiples of
four, the largest it takes and the first it leaves to the launches; one row
over all CTAs, rows of one edge, more vertices than edges, long runs of empty
rows inside a CTA's edges, no iteration and one.

Iteration counts equal the reference loop's; ranks are as accurate against
FP64 as the reference's FP32 loop (fpcheck)."""
import numpy as np
import pytest

from fpcheck import assert_fp_as_accurate
from graphs import pair

pytestmark = pytest.mark.gpu


def edges(shape, E):
    rng = np.random.default_rng(E)
    if shape == "one_row":
        return rng.integers(0, 60000, E), np.full(E, 777), 60000
    if shape == "degree_1":
        return rng.permutation(E), np.arange(E), E
    if shape == "sparse":
        V = 2 * E + 7
        return rng.integers(0, V, E), rng.integers(0, V, E), V
    if shape == "gaps":  # rows in two clusters, 5,000 empty rows between every pair of dense blocks
        V = 400000
        d = rng.integers(0, 40, E) * 10000 + rng.integers(0, 5000, E)
        return rng.integers(0, V, E), d, V
    if shape == "gaps_in":  # the same within the vertices it takes: 3,000 empty rows between blocks, one of 60,000
        V = 200000
        d = rng.integers(0, 20, E) * 7000 + rng.integers(0, 4000, E)
        return rng.integers(0, V, E), np.where(d < 70000, d, d + 57000), V
    V = max(3, E // 16) | 1
    return rng.integers(0, V, E), (rng.random(E) ** 3 * V).astype(np.int64), V


S = 152 * 1024  # threads
CASES = ([("skewed", E) for E in (163841, 4 * S, 4 * S + 1, 8 * S - 3, 8 * S + 1, 12 * S + 1, 16 * S, 20 * S + 1)] +
         [("one_row", E) for E in (200001, 8 * S + 5)] + [("degree_1", 200001), ("degree_1", 4 * S + 33)] +
         [("sparse", E) for E in (170000, 300001)] + [("gaps", E) for E in (180000, 900000)] +
         [("gaps_in", E) for E in (1000, 50000, 180000, 900000)] + [("sparse", E) for E in (40000, 109990)] +
         [("sparse", 20), ("degree_1", 219999)])


@pytest.mark.parametrize("shape,E", CASES)
def test_grid_pull(gpu, orc, shape, E):
    src, dst, V = edges(shape, E)
    g, o = pair(gpu, orc, gpu.Graph.from_edges(src.astype(np.uint32), dst.astype(np.uint32), num_vertices=V))
    dg = gpu.DeviceGraph(g, gpu.MAP_IN)
    for its, eps in ((20, 1e-4), (1, 0.0), (5, 0.0)):
        ranks, res = dg.pagerank("pull", iterations=its, epsilon=eps)
        ref, info = orc.pagerank(o, 0, its, eps)
        assert res["iterations"] == info["iterations"]
        assert_fp_as_accurate(ranks, ref, orc.pagerank_f64(o, info["executed"]), f"{its} iterations")
        assert abs(res["rank_sum"] - ranks.astype(np.float64).sum()) <= 1e-9 * res["rank_sum"]
    none, _ = dg.pagerank("pull", iterations=0)
    np.testing.assert_array_equal(none, np.full(V, (np.float32(1.0) - np.float32(0.85)) / np.float32(V), np.float32))
    dg.free()
