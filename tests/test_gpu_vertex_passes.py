"""Vertex passes of PageRank and SpMV at the sizes where they can go wrong:
one vertex, odd and even counts (passes take two or four vertices per step),
and sums across the range of each number format.

Integer formats are compared bit by bit with the oracle; the SpMV checksum is
a sum of whole hundredths, so it is compared with the same sum in Python
integers (one FP64 rounding: 1e-15 relative)."""
import numpy as np
import pytest

from graphs import pair

pytestmark = pytest.mark.gpu

MODES = {"pull_fx64": 2, "push_fx64": 3, "pull_q32": 4, "pull_fx32": 9, "pull_fx16": 10, "pull_fx8": 11,
         "pull_q16": 12, "pull_q8": 13}


def random_edges(V, E, seed):
    rng = np.random.default_rng(seed)
    # half of the edges end at one vertex: long rows beside empty ones
    dst = np.where(rng.random(E) < 0.5, V // 2, rng.integers(0, V, E))
    return rng.integers(0, V, E).astype(np.uint32), dst.astype(np.uint32)


@pytest.mark.parametrize("V", [1, 2, 3, 257, 4096, 70001])
def test_integer_formats_bit_exact(gpu, orc, V):
    src, dst = random_edges(V, 9 * V, V)
    g, o = pair(gpu, orc, gpu.Graph.from_edges(src, dst, num_vertices=V))
    dg = gpu.DeviceGraph(g, gpu.MAP_ALL)
    for name, mode in MODES.items():
        ranks, res = dg.pagerank(name, iterations=6, epsilon=1e-4)
        ref, info = orc.pagerank(o, mode, 6, 1e-4)
        assert res["iterations"] == info["iterations"], name
        np.testing.assert_array_equal(ranks.view(np.uint32), ref.view(np.uint32), err_msg=name)
        assert abs(res["error_total"] - info["error_total"]) <= 1e-9 * info["error_total"] + 1e-15, name


@pytest.mark.parametrize("V,scale", [(1, 1.0), (5, 1e6), (1023, 1e-3), (1024, 1.0), (70002, 3e4)])
def test_spmv_checksum(gpu, V, scale):
    src, dst = random_edges(V, 4 * V, V + 1)
    w = (np.random.default_rng(V).standard_normal(4 * V) * scale).astype(np.float32)
    g = gpu.Graph.from_edges(src, dst, w, num_vertices=V)
    dg = gpu.DeviceGraph(g, gpu.MAP_ALL)
    _, y, res = dg.spmv("pull", iterations=1)
    t = (y * np.float32(100.0)).astype(np.float64) + 0.5
    want = int(np.trunc(np.clip(t, -2.0 ** 31, 2.0 ** 31 - 1)).astype(np.int64).sum()) / 100.0
    assert abs(res["checksum"] - want) <= 1e-15 * abs(want)
