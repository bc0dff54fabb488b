"""The default choice between the plain gather and the one through the hot-vertex
table, from 8M edges: the table on graphs with hubs and on uniform random ones, the
plain gather where neighbours lie close together (a band, a mesh, many small
blocks), for every value size; both give the same ranks and products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

V, EF = 1 << 20, 9


def edges(kind):
    rng = np.random.default_rng(7)
    E = V * EF
    src = rng.integers(0, V, E)
    if kind == "uniform":
        dst = rng.integers(0, V, E)
    elif kind == "skewed":
        src, dst = (rng.random(E) ** 6 * V).astype(np.int64), rng.integers(0, V, E)
    elif kind == "band":
        dst = (src + rng.integers(-500, 501, E)) % V
    elif kind == "blocks":
        dst = src // 1024 * 1024 + rng.integers(0, 1024, E)
    else:  # a mesh of 1024 x 1024 with nine neighbours
        v = np.arange(V)
        src = np.repeat(v, EF)
        dst = (src + np.tile([-1025, -1024, -1023, -1, 1, 1023, 1024, 1025, 2], V)) % V
    return src.astype(np.uint32), dst.astype(np.uint32)


@pytest.mark.parametrize("kind,table", [("uniform", 1), ("skewed", 1), ("band", 0), ("blocks", 0), ("mesh", 0)])
def test_default_gather(gpu, kind, table):
    src, dst = edges(kind)
    w = np.random.default_rng(8).random(len(src)).astype(np.float32)
    dg = gpu.DeviceGraph.build(src, dst, weights=w, num_vertices=V, what=gpu.MAP_IN | gpu.MAP_IN_W)
    for mode, storage in (("pull", "f32"), ("pull", "bf16"), ("pull_q16", "f32"), ("pull_q8", "f32"), ("pull_fx64", "f32")):
        ranks, res = dg.pagerank(mode, storage=storage, iterations=10, epsilon=0.0)
        assert res["hot_table"] == table, (mode, storage)
        other, res = dg.pagerank(mode, storage=storage, iterations=10, epsilon=0.0, hot=not table)
        assert res["hot_table"] == 1 - table
        if storage == "f32" and mode == "pull":
            np.testing.assert_allclose(ranks, other, rtol=2e-6 * 10, atol=0)
        elif storage == "f32":
            np.testing.assert_array_equal(ranks, other)
    _, y, res = dg.spmv("pull", iterations=10)
    _, y2, same = dg.spmv("pull", iterations=10, hot=bool(table))
    assert res["launches"] == same["launches"]
    _, y3, other = dg.spmv("pull", iterations=10, hot=not table)
    assert other["launches"] == res["launches"] + (1 if not table else -1)  # the table's fill
    np.testing.assert_allclose(y, y3, rtol=2e-5, atol=0)
    dg.free()


def test_union_of_small_graphs(gpu):
    """Many graphs in one call, as the pull of their union."""
    n, size = 1024, 1 << 10
    src, dst = edges("blocks")
    dg = gpu.DeviceGraph.build(src, dst, num_vertices=V, what=gpu.MAP_IN)
    voff = np.arange(n + 1, dtype=np.uint32) * size
    ranks, res = dg.pagerank_batch(voff, iterations=10, epsilon=0.0, union=True)
    assert res["hot_table"] == 0
    other, res = dg.pagerank_batch(voff, iterations=10, epsilon=0.0, union=True, hot=True)
    assert res["hot_table"] == 1
    np.testing.assert_allclose(ranks, other, rtol=2e-5, atol=0)
    dg.free()
