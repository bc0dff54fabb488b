"""Push scatters through the table of frequent destinations where it can go
wrong: the fewest edges it is made for and one less, samples with and without
gaps, one destination for all edges, several frequent ones with one hash, no
frequent ones (the table stays off), CUDA graphs.

Integer sums equal the oracle's bits; FP32 as accurate against FP64 as the
reference's own FP32 loop (fpcheck); 8-bit pushes within the bound of their
other tests (5e-3 of the L1 norm)."""
import numpy as np
import pytest

from fpcheck import assert_fp_as_accurate
from graphs import pair

pytestmark = pytest.mark.gpu

MIN_E = 1 << 16


def edges(shape, E):
    rng = np.random.default_rng(E)
    V = 30011
    src, dst = rng.integers(0, V, E), rng.integers(0, V, E)
    if shape == "one":
        dst = np.full(E, 12345)
    elif shape == "skewed":
        dst = (rng.random(E) ** 6 * V).astype(np.int64)
    elif shape == "one_hash":  # the vertices whose 12-bit hash is that of vertex 1
        h = (np.arange(V, dtype=np.uint64) * 0x9E3779B1 % (1 << 32)) >> 20
        same = np.flatnonzero(h == h[1])
        assert same.size > 3
        dst = np.where(rng.random(E) < 0.5, same[rng.integers(0, same.size, E)], dst)
    return src.astype(np.uint32), dst.astype(np.uint32), V


@pytest.mark.parametrize("shape,E", [("skewed", MIN_E - 1), ("skewed", MIN_E), ("one", MIN_E + 1), ("one_hash", 70001),
                                     ("none", 100000), ("skewed", 262145), ("one_hash", 700001), ("skewed", 700033)])
def test_push_table(gpu, orc, shape, E):
    src, dst, V = edges(shape, E)
    w = np.random.default_rng(1).random(E).astype(np.float32)
    g, o = pair(gpu, orc, gpu.Graph.from_edges(src, dst, w, num_vertices=V))
    dg = gpu.DeviceGraph(g, gpu.MAP_OUT | gpu.MAP_OUT_W)
    its = 40  # makes the table before the first scatter
    for mode in (1, 3, 5):
        for graph in (False, True):
            ranks, res = dg.pagerank(mode, iterations=its, epsilon=0.0, cuda_graph=graph)
            ref, info = orc.pagerank(o, mode, its, 0.0)
            assert res["iterations"] == info["iterations"]
            if mode == 3:
                np.testing.assert_array_equal(ranks.view(np.uint32), ref.view(np.uint32))
            elif mode == 1:
                assert_fp_as_accurate(ranks, ref, orc.pagerank_f64(o, info["executed"]), "push")
            else:
                assert float(np.abs(ranks - ref).sum()) <= 5e-3 * float(np.abs(ref).sum())
    for mode in (1, 3):
        x, y, _ = dg.spmv(mode, iterations=3)
        _, ry, _ = orc.spmv(o, mode, 3)
        if mode == 3:
            np.testing.assert_array_equal(y.view(np.uint32), ry.view(np.uint32))
        else:
            assert_fp_as_accurate(y, ry, 3 * orc.spmv_f64(o, x), "spmv")
    dg.free()
