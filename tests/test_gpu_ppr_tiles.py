"""Batched personalised PageRank at the edges of its tiles and chunks: edge
counts around multiples of 16, 32, 256 and 512, rows of one edge, one row over
many tiles, mostly empty rows, and every row width and storage.

FP32 storage: within L1 <= 1e-6 of FP64 per vector, plus (a row of n edges
summed in FP32 in any order) n * 2^-24 of the largest entry.  BF16: bit-equal
to the same call with each iteration launched on its own, and FP32 results do
not depend on the row width."""
import numpy as np
import pytest

from graphs import pair

pytestmark = pytest.mark.gpu

DAMP = float(np.float32(0.85))


def edges(shape, E):
    rng = np.random.default_rng(E)
    if shape == "one_row":
        return rng.integers(0, 90, E), np.full(E, 7), 90
    if shape == "degree_1":
        return rng.permutation(E), np.arange(E), E
    if shape == "sparse":
        V = 5 * E + 40
        return rng.integers(0, V, E), rng.integers(0, V, E), V
    V = max(2, E // 20)
    return rng.integers(0, V, E), rng.integers(0, V, E), V


CASES = ([("one_row", E) for E in (1, 15, 16, 17, 33, 255, 257, 1023, 9001)] +
         [("degree_1", E) for E in (3, 64, 513, 20011)] + [("sparse", E) for E in (31, 512, 5003)] +
         [("rows_20", E) for E in (40, 256, 4097, 60013)])


@pytest.mark.parametrize("shape,E", CASES)
def test_ppr_shapes(gpu, orc, shape, E):
    src, dst, V = edges(shape, E)
    g, o = pair(gpu, orc, gpu.Graph.from_edges(src.astype(np.uint32), dst.astype(np.uint32), num_vertices=V))
    rng = np.random.default_rng(E + 1)
    sets = [rng.integers(0, V, int(rng.integers(1, 6))) for _ in range(64)]
    sets[1] = [int(src[0]), int(src[0]), int(dst[0])]
    dg = gpu.DeviceGraph(g, gpu.MAP_IN)
    wide, _ = dg.ppr(sets, iterations=5, storage="f32")
    ex = np.stack([orc.ppr_f64_multi(o, s, 5, DAMP) for s in sets], 1)
    longest = int(np.bincount(dst).max())
    assert (np.abs(wide - ex).sum(0) <= 1e-6 + longest * 2.0 ** -24 * ex.max()).all()
    for K in (1, 16, 17, 32, 33):
        part, _ = dg.ppr(sets[:K], iterations=5, storage="f32")
        np.testing.assert_array_equal(part, wide[:, :K], err_msg=f"K={K}")
    for K in (2, 20, 64):
        one, r = dg.ppr(sets[:K], iterations=5, storage="bf16")
        many, _ = dg.ppr(sets[:K], iterations=5, storage="bf16", profile=True)
        assert r["persistent"] == 1
        np.testing.assert_array_equal(one, many, err_msg=f"K={K}")
    dg.free()
