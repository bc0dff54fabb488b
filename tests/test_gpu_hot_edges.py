"""The hot-vertex gather at the sizes where its steps of 128 edges and tiles of
256 to 2048 edges can go wrong: edge counts around their multiples and of every
remainder, rows of one edge (128 row ends in a step), one row over many tiles,
empty rows between, and more vertices than the table holds.

Integer formats: bit-equal to the gather without the table.  FP32: as accurate
against FP64 as the reference's own FP32 loop (fpcheck)."""
import numpy as np
import pytest

from fpcheck import assert_fp_as_accurate
from graphs import pair

pytestmark = pytest.mark.gpu

INT_MODES = ["pull_fx64", "pull_q32", "pull_fx32", "pull_fx16", "pull_fx8", "pull_q16", "pull_q8"]


def edges(shape, E):
    rng = np.random.default_rng(E)
    if shape == "one_row":  # every edge ends at one vertex
        V = 300
        return rng.integers(0, V, E), np.full(E, 7), V
    if shape == "degree_1":  # a permutation: every row one edge
        return rng.permutation(E), np.arange(E), E
    if shape == "sparse":  # mostly empty rows, more vertices than table slots
        V = 3 * E + 100000
        return rng.integers(0, V, E), rng.integers(0, V, E), V
    V = max(2, E // 40)  # rows of about 40 edges
    return rng.integers(0, V, E), rng.integers(0, V, E), V


CASES = ([("one_row", E) for E in (1, 3, 127, 128, 130, 255, 256, 257, 2047, 2049, 70001)] +
         [("degree_1", E) for E in (5, 128, 1023, 100003)] +
         [("sparse", E) for E in (33, 4097, 150002)] + [("rows_40", E) for E in (81, 4096, 50005, 200000)])


@pytest.mark.parametrize("shape,E", CASES)
def test_hot_gather(gpu, orc, shape, E):
    src, dst, V = edges(shape, E)
    w = np.random.default_rng(1).random(E).astype(np.float32)
    g, o = pair(gpu, orc, gpu.Graph.from_edges(src.astype(np.uint32), dst.astype(np.uint32), w, num_vertices=V))
    dg = gpu.DeviceGraph(g, gpu.MAP_IN | gpu.MAP_IN_W)
    for mode in INT_MODES:
        hot, rh = dg.pagerank(mode, iterations=3, epsilon=0.0, hot=True)
        plain, rp = dg.pagerank(mode, iterations=3, epsilon=0.0, hot=False)
        assert (rh["hot_table"], rp["hot_table"]) == (1, 0)
        np.testing.assert_array_equal(hot.view(np.uint32), plain.view(np.uint32), err_msg=mode)
    hot, _ = dg.pagerank("pull", iterations=3, epsilon=0.0, hot=True)
    ref, info = orc.pagerank(o, 0, 3, 0.0)
    assert_fp_as_accurate(hot, ref, orc.pagerank_f64(o, 3), "pagerank")
    x = np.random.default_rng(2).random(V).astype(np.float32)
    _, y, _ = dg.spmv("pull", x=x, hot=True)
    _, y32, _ = orc.spmv(o, 0, 1, x=x)
    assert_fp_as_accurate(y, y32, orc.spmv_f64(o, x), "spmv")
