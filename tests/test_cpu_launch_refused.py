"""A device that does not take the cooperative launch of the one-launch pull
(too few blocks resident at once): the call runs as separate launches."""
import fake_cuda

CODE = """
rng = np.random.default_rng(1)
V, E = 50000, 200000
g = gg.Graph.from_edges(rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32), num_vertices=V)
dg = gg.DeviceGraph(g, gg.MAP_IN)
F.fake_log_clear()
dg.pagerank("pull", iterations=3)
assert sum("k_pr_grid" in k for k in launches()) == 1, launches()
F.fake_log_clear()
F.fake_coop_error(720)  # cudaErrorCooperativeLaunchTooLarge
_, res = dg.pagerank("pull", iterations=3)
assert sum("k_pr_update" in k for k in launches()) == 3, launches()
assert res["launches"] > 3, res
print("ok")
"""


def test_refused_cooperative_launch_runs_as_launches():
    assert "ok" in fake_cuda.run(CODE)
