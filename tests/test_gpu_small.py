"""PageRank pull of small graphs (every iteration in one CTA or one cluster) at
the sizes where its shares change: edges per thread (4, 12, 20), one CTA or
eight, the largest graph it takes and the first it leaves to the launches; rows
of one edge, one row over all CTAs, empty rows, both formulations, no iteration
and one.

Iteration counts equal the reference loop's; ranks are as accurate against
FP64 as the reference's FP32 loop (fpcheck); in the 1/N formulation within the
error of six FP32 sums of the longest row's terms in any order (n * 2^-24 each,
and four roundings more)."""
import numpy as np
import pytest

from fpcheck import assert_fp_as_accurate
from graphs import pair

pytestmark = pytest.mark.gpu

DAMP = float(np.float32(0.85))


def edges(shape, E):
    rng = np.random.default_rng(E)
    if shape == "one_row":
        return rng.integers(0, 500, E), np.full(E, 77), 500
    if shape == "degree_1":
        return rng.permutation(E), np.arange(E), E
    if shape == "sparse":
        V = 2 * E + 7
        return rng.integers(0, V, E), rng.integers(0, V, E), V
    V = max(3, E // 16) | 1
    return rng.integers(0, V, E), (rng.random(E) ** 3 * V).astype(np.int64), V


CASES = ([("skewed", E) for E in (1, 31, 127, 4096, 4097, 12289, 16384, 16385, 32769, 98305, 163840, 163841)] +
         [("one_row", E) for E in (5, 4097, 16400, 100001)] + [("degree_1", E) for E in (2, 4097, 20001)] +
         [("sparse", E) for E in (3, 4500, 9000)])


@pytest.mark.parametrize("shape,E", CASES)
def test_small_pull(gpu, orc, shape, E):
    src, dst, V = edges(shape, E)
    g, o = pair(gpu, orc, gpu.Graph.from_edges(src.astype(np.uint32), dst.astype(np.uint32), num_vertices=V))
    dg = gpu.DeviceGraph(g, gpu.MAP_IN)
    for its, eps in ((20, 1e-4), (1, 0.0), (7, 0.0)):
        ranks, res = dg.pagerank("pull", iterations=its, epsilon=eps)
        ref, info = orc.pagerank(o, 0, its, eps)
        assert res["iterations"] == info["iterations"]
        assert_fp_as_accurate(ranks, ref, orc.pagerank_f64(o, info["executed"]), f"{its} iterations")
        again, r2 = dg.pagerank("pull", iterations=its, epsilon=eps, cuda_graph=True)
        np.testing.assert_allclose(again, ranks, rtol=2e-6, atol=0)
        _, plain = dg.pagerank("pull", iterations=its, epsilon=eps, profile=True)  # the launches
        assert (res["iterations"], res["active"]) == (plain["iterations"], plain["active"]) or eps
        assert abs(res["rank_sum"] - ranks.astype(np.float64).sum()) <= 1e-9 * res["rank_sum"]
    one, _ = dg.pagerank("pull", iterations=6, epsilon=0.0, init_one_over_n=True)
    r = np.full(V, 1.0 / V)
    deg = np.bincount(src, minlength=V)
    for _ in range(6):
        c = np.where(deg > 0, r / np.maximum(deg, 1), 0.0)
        r = (1.0 - DAMP) / V + DAMP * np.bincount(dst, c[src], minlength=V)
    assert (np.abs(one - r) <= 6 * (np.bincount(dst).max() + 4) * 2.0 ** -24 * r).all()
    none, _ = dg.pagerank("pull", iterations=0)
    np.testing.assert_array_equal(none, np.full(V, (np.float32(1.0) - np.float32(0.85)) / np.float32(V), np.float32))
    dg.free()
