"""GG_PR_CUDA_GRAPH: a first call captures and instantiates, a repeat launches the
instance and queues no kernel of its own, other parameters and a buffer freed in
between capture again; FP32 pulls that are one launch anyway capture nothing."""
import pytest

import fake_cuda

CODE = """
V, E = {V}, {E}
rng = np.random.default_rng(1)
g = gg.Graph.from_edges(rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32), num_vertices=V)
dg = gg.DeviceGraph(g, gg.MAP_ALL)

def call(its):
    F.fake_log_clear()
    _, res = dg.pagerank({args}, iterations=its, cuda_graph=True)
    log = launches()
    return log.count("<instantiate>"), log.count("<graph>"), sum("k_pr_" in k for k in log), res["launches"]

first = call(20)
assert first[:2] == (1, 1) and first[2] > 20, first
again = call(20)
assert again == (0, 1, 0, first[3]), again
other = call(7)
assert other[:2] == (1, 1) and other[3] < first[3], other
assert call(7) == (0, 1, 0, other[3])
dg.bfs(0, "push")  # regrows work buffers that the captured graph writes
assert call(7)[:2] == (1, 1)
assert call(7) == (0, 1, 0, other[3])
print("ok")
"""

MODES = ["'pull', storage='bf16'", "'pull_q16'", "'pull_fx64'", "'push'", "'pull', hot=True"]


@pytest.mark.parametrize("args", MODES)
def test_capture_replay_and_recapture(args):
    assert "ok" in fake_cuda.run(CODE.format(args=args, V=5000, E=70000))


def test_larger_fp32_pull_is_captured():
    assert "ok" in fake_cuda.run(CODE.format(args="'pull'", V=300000, E=600000))


def test_small_fp32_pull_is_one_launch_without_a_graph():
    code = CODE[:CODE.index("first =")].format(args="'pull'", V=5000, E=70000)
    assert "ok" in fake_cuda.run(code + "\nassert call(20) == (0, 0, 1, 1) and call(20) == (0, 0, 1, 1)\nprint('ok')\n")
