"""Connected components at the sizes where Afforest's passes can go wrong: vertex
counts of every remainder of four (they take four vertices per step), two large
components so that one is not skipped, hubs on either side of the row length
that is spread over the grid, many small components, and samples counted on the
device and on the host.  Labels are compared exactly with scipy's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def expected(V, src, dst):
    sp = pytest.importorskip("scipy.sparse")
    g = sp.coo_matrix((np.ones(len(src), np.int8), (src, dst)), shape=(V, V)).tocsr()
    _, lab = sp.csgraph.connected_components(g, directed=True, connection="weak")
    first = np.full(lab.max() + 1, V, np.int64)
    np.minimum.at(first, lab, np.arange(V))
    return first[lab].astype(np.uint32)


def two_halves(V, hub_edges, seed):
    """Edges inside the even and inside the odd vertices, each half with an out-
    hub and an in-hub, and the last tenth of the ids left alone."""
    rng = np.random.default_rng(seed)
    n = max(2, V - V // 10)
    s = rng.integers(0, n, 2 * V)
    d = rng.integers(0, n, 2 * V)
    d = np.minimum(d - d % 2 + s % 2, n - 1 - (n - 1 - s) % 2)
    out = [(s, d)]
    if hub_edges:
        for hub in (n // 2, n // 2 + 1):
            other = rng.integers(0, n // 2, hub_edges) * 2 + hub % 2
            other = np.where(other < n, other, hub)
            out += [(np.full(hub_edges, hub), other), (other, np.full(hub_edges, hub))]
    return (np.concatenate([a for a, _ in out]).astype(np.uint32),
            np.concatenate([b for _, b in out]).astype(np.uint32))


@pytest.mark.parametrize("V,hub", [(2, 0), (3, 0), (5, 0), (33, 40), (4096, 2040), (4097, 2060), (10002, 9000),
                                   (70003, 5000)])
@pytest.mark.parametrize("samples", [0, 3000])
def test_afforest(gpu, V, hub, samples):
    src, dst = two_halves(V, hub, V)
    want = expected(V, src, dst)
    g = gpu.Graph.from_edges(src, dst, num_vertices=V)
    dg = gpu.DeviceGraph(g, gpu.MAP_IN | gpu.MAP_OUT)
    for use_in in (1, 2):
        lab, r = dg.cc("afforest", use_in_edges=use_in, samples=samples)
        np.testing.assert_array_equal(lab, want)
        assert r["components"] == len(np.unique(want))
    out_only = gpu.DeviceGraph(g, gpu.MAP_OUT)
    lab, r = out_only.cc("afforest", samples=samples)
    np.testing.assert_array_equal(lab, want)
    assert r["skipped_label"] == 0xFFFFFFFF
    for rounds in (1, 3):
        lab, _ = dg.cc("afforest", neighbor_rounds=rounds, samples=samples)
        np.testing.assert_array_equal(lab, want)
    for algorithm in ("sv", "weakly"):
        lab, _ = dg.cc(algorithm)
        np.testing.assert_array_equal(lab, want)
