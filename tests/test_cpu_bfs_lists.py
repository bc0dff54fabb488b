"""The second list of a top-down step's hubs is chosen by the step's own frontier,
not by what an earlier call left in the mapping's page-locked scratch: a step over a
frontier whose edges are not known has it from more than 4,096 vertices on."""
import pytest

import fake_cuda

CODE = """
V, E = 20000, 100000
rng = np.random.default_rng(1)
g = gg.Graph.from_edges(rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32), num_vertices=V)
dg = gg.DeviceGraph(g, gg.MAP_ALL)
if {before!r}:
    eval({before!r})  # leaves other words in the scratch
u32p = C.POINTER(C.c_uint32)
for n, second in ((4096, False), (4097, True), (9000, True)):
    parents = np.full(V, -1, np.int32)
    dist = np.zeros(V, np.uint32)
    q = np.arange(n, dtype=np.uint32)
    nq = np.zeros(V, np.uint32)
    nlen, cnt = C.c_uint32(), C.c_uint32()
    F.fake_log_clear()
    F.gg_bfs_step_host.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_uint32, C.c_int] + [C.c_void_p] * 7
    st = F.gg_bfs_step_host(dg.h, 0, q.ctypes.data, n, 0, parents.ctypes.data, dist.ctypes.data, nq.ctypes.data, None,
                            C.addressof(nlen), C.addressof(cnt), None)
    assert st == 0
    assert any("k_td_huge" in k for k in launches()) == second, (n, launches())
print("ok")
"""


@pytest.mark.parametrize("before", ["", "dg.pagerank('push', iterations=30)"])
def test_second_list_by_the_frontier(before):
    assert "ok" in fake_cuda.run(CODE.format(before=before))
