"""The residual and the rank sum are results in double: no bit of an FP64 sum
is lost and none overflows FP32.

With damp 1 and ranks of 1/V at first, every rank after t iterations is the flow
along paths of t edges.  Three chains of fans leave, after six iterations, ranks
of r, 2^-25 r and 2^-50 r at three vertices of one warp and zero elsewhere: their
sum needs 51 bits and is exact in FP64 in any order.  One iteration later all
three are gone, and their differences are the residual."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chains(extra):
    """Edges of the chains, ending at vertices 0, 1 and 2 (22 vertices), and
    `extra` edges from a vertex without in-edges into one without out-edges."""
    src, dst, at, sink = [], [], 4, 3
    for end, fans in ((0, (0, 0, 0, 0, 0, 0)), (1, (10, 10, 5, 0, 0, 0)), (2, (10, 10, 10, 10, 10, 0))):
        ids = list(range(at, at + 6)) + [end]
        at += 6
        for i, f in enumerate(fans):
            src += [ids[i]] * (1 << f)
            dst += [ids[i + 1]] + [sink] * ((1 << f) - 1)
    return np.array(src + [at] * extra, np.uint32), np.array(dst + [sink] * extra, np.uint32)


# one CTA, a cluster, the whole chip, the launches, push
CASES = [(64, 0, "pull", {}), (64, 20000, "pull", {}), (1 << 14, 100000, "pull", {}),
         (64, 0, "pull", dict(profile=True)), (1 << 14, 100000, "pull", dict(hot=True)), (64, 0, "push", {})]


@pytest.mark.parametrize("V,extra,mode,kw", CASES)
def test_sums_keep_the_bits_of_fp64(gpu, V, extra, mode, kw):
    src, dst = chains(extra)
    g = gpu.Graph.from_edges(src, dst, num_vertices=V)
    dg = gpu.DeviceGraph(g, gpu.MAP_IN | gpu.MAP_OUT)
    want = (1.0 + 2.0 ** -25 + 2.0 ** -50) / V
    opts = dict(epsilon=0.0, damp=1.0, init_one_over_n=True, **kw)
    ranks, res = dg.pagerank(mode, iterations=6, **opts)
    np.testing.assert_array_equal(ranks[:3] * V, np.array([1.0, 2.0 ** -25, 2.0 ** -50], np.float32))
    assert not ranks[3:].any()
    assert res["rank_sum"] == want
    none, res = dg.pagerank(mode, iterations=7, **opts)
    assert not none.any()
    assert res["error_total"] == want / V
    dg.free()
    g.free()


@pytest.mark.parametrize("V,kw", [(1000, {}), (20000, {}), (40000, {}), (1000, dict(profile=True))])
def test_sums_past_the_range_of_fp32(gpu, V, kw):
    """A ring with damp 1e19: ranks near -1e38 after one iteration, whose
    differences add up past FP32's largest number in every warp."""
    v = np.arange(V, dtype=np.uint32)
    g = gpu.Graph.from_edges(v, np.roll(v, 1), num_vertices=V)
    dg = gpu.DeviceGraph(g, gpu.MAP_IN)
    damp = np.float32(1e19)
    base = np.float32(1.0) - damp
    rank = base + damp * base
    ranks, res = dg.pagerank("pull", iterations=1, epsilon=0.0, damp=float(damp), **kw)
    np.testing.assert_array_equal(ranks, np.full(V, rank / np.float32(V), np.float32))
    assert res["error_total"] == pytest.approx(float(np.abs(rank - base)), rel=1e-12)
    assert res["rank_sum"] == pytest.approx(float(rank / np.float32(V)) * V, rel=1e-12)
    dg.free()
    g.free()
