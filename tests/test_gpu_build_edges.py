"""The device build where its sort can go wrong: edge counts around a tile
(4096 and 8192 edges) and around the size from which the column scan takes
three launches, vertex counts whose ids need one to three digits of 5 to 8
bits, all edges in one row, either direction alone, weights of one direction,
and callers' arrays that start at any element.  Every array equals the stable
lexicographic sort; whole numbers and copies, so exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def edges(E, V, kind):
    rng = np.random.default_rng(E + V)
    s, d = rng.integers(0, V, E), rng.integers(0, V, E)
    if kind == "one_row":
        s = np.full(E, V - 1)
    elif kind == "dups":
        s, d = s % 3 % V, d % 2 % V
    return s.astype(np.uint32), d.astype(np.uint32), rng.standard_normal(E).astype(np.float32)


def expect(key, other, w, V):
    order = np.lexsort((other, key))
    off = np.zeros(V + 1, np.int64)
    np.cumsum(np.bincount(key, minlength=V), out=off[1:])
    return off.astype(np.uint32), other[order], w[order]


CASES = [(1, 1, "rand"), (4095, 33, "rand"), (4096, 129, "rand"), (4097, 256, "dups"), (8191, 257, "one_row"),
         (8192, 4097, "rand"), (8193, 70000, "rand"), (16384, (1 << 17) + 1, "rand"), (100001, 3, "dups"),
         (256 * 4096 + 1, 1 << 16, "rand"), (256 * 8192, (1 << 20) + 1, "rand"), (256 * 8192 + 5, 1 << 20, "one_row")]


@pytest.mark.parametrize("E,V,kind", CASES)
def test_build_equals_stable_sort(gpu, E, V, kind):
    torch = pytest.importorskip("torch")
    s, d, w = edges(E, V, kind)
    out, inn = expect(s, d, w, V), expect(d, s, w, V)

    def dev(a, at):  # the array from element `at` of an allocation
        t = torch.zeros(E + at, dtype=torch.int32 if a.dtype == np.uint32 else torch.float32, device="cuda")
        t[at:] = torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()
        return t[at:]

    for at in (0, 3):
        dg = gpu.DeviceGraph.build(dev(s, at), dev(d, at), dev(w, at), num_vertices=V)
        got = dg.download()
        for name, (off, adj, ww) in (("out", out), ("in", inn)):
            np.testing.assert_array_equal(got[name + "_off"], off)
            np.testing.assert_array_equal(got[name + "_adj"], adj)
            np.testing.assert_array_equal(got[name + "_w"].view(np.uint32), ww.view(np.uint32))
        assert got["max_weight"] == max(0.0, float(w.max()))
        dg.free()
    dg = gpu.DeviceGraph.build(s, d, None, num_vertices=V, what=gpu.MAP_IN | gpu.MAP_OUT)
    got = dg.download(weights=False)
    for name, (off, adj, _) in (("out", out), ("in", inn)):
        np.testing.assert_array_equal(got[name + "_off"], off)
        np.testing.assert_array_equal(got[name + "_adj"], adj)
    dg.free()
    # one direction: the products of a pull (in) and a push (out)
    x = np.ones(V, np.float32)
    ref = np.zeros(V)
    np.add.at(ref, d, w.astype(np.float64))
    bound = np.zeros(V)
    np.add.at(bound, d, np.abs(w.astype(np.float64)))
    deg = np.bincount(d, minlength=V)
    for mode, what in (("pull", gpu.MAP_IN | gpu.MAP_IN_W), ("push", gpu.MAP_OUT | gpu.MAP_OUT_W)):
        dg = gpu.DeviceGraph.build(s, d, w, num_vertices=V, what=what)
        _, y, _ = dg.spmv(mode, x=x)
        # FP32 sums of deg terms in any order: deg * 2^-24 of the sum of magnitudes
        assert (np.abs(y - ref) <= deg * 2.0**-24 * bound + 1e-30).all(), mode
        dg.free()


def test_build_refuses_ids_out_of_range(gpu):
    for s, d in (([0, 1, 5], [0, 1, 2]), ([0, 1, 2], [0, 0xffffffff, 2])):
        with pytest.raises(gpu.GgError):
            gpu.DeviceGraph.build(np.array(s, np.uint32), np.array(d, np.uint32), None, num_vertices=5)
