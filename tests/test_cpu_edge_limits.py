"""Host arithmetic at the largest edge counts that a mapping takes (2^32 - 1):
calls on graphs whose arrays are address space only, with the fake runtime."""
import pytest

import fake_cuda

CODE = """
V, E = 1000, {E}
small = np.zeros(V + 16, np.uint32)
u32 = small.ctypes.data_as(C.POINTER(C.c_uint32))
vert = gg.Vertex(u32, u32, u32)
edges = gg.EdgeList(E, V, 1.0, u32, u32, None, None, None)  # ids that nothing reads: the copy is left out
graph = gg.GraphCSR(E, V, 1.0, 1, C.pointer(vert), C.pointer(vert), C.pointer(edges), C.pointer(edges))
gg.set_host_copy_mode("driver")
dg = gg.DeviceGraph(gg.Graph(C.pointer(graph)), gg.MAP_OUT)
F.fake_log_clear()
dg.pagerank("push", iterations=40, copy_out=False)
assert any("k_push_sample" in k for k in launches()), launches()
dg.graph.ptr = None
print("ok")
"""


@pytest.mark.parametrize("E", [1 << 24, (1 << 32) - 64, (1 << 32) - 33, (1 << 32) - 32, (1 << 32) - 31, (1 << 32) - 1])
def test_push_sampling_at_edge_limits(E):
    assert "ok" in fake_cuda.run(CODE.format(E=E))
