"""A tuned shape chooses between gather launches; a graph that runs in one launch
uses none of them, whatever was tuned for its class."""
import fake_cuda

CODE = """
with open({path!r}, "w") as f:
    for v in range(1, 32):
        for d in range(0, 12):
            for k in range(0, 26):
                f.write(f"{{gg.TUNE_PR}} 0 {{v}} {{d}} {{k}} 152 0 : 1 5 32 0 0\\n")  # with the table
gg.tune_load({path!r})
rng = np.random.default_rng(1)
for V, E, kernel in ((500, 5000, "k_pr_small"), (5000, 60000, "k_pr_small"), (50000, 800000, "k_pr_grid")):
    g = gg.Graph.from_edges(rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32), num_vertices=V)
    dg = gg.DeviceGraph(g, gg.MAP_IN)
    F.fake_log_clear()
    _, res = dg.pagerank("pull", iterations=20)
    assert dg.tuned(gg.TUNE_PR)[0] == 1
    assert res["launches"] == 1 and any(kernel in k for k in launches()), (res, launches())
    F.fake_log_clear()
    _, res = dg.pagerank("pull", iterations=20, hot=True)
    assert res["hot_table"] == 1 and any("k_pr_pull_hot" in k for k in launches())
    F.fake_log_clear()
    _, res = dg.pagerank("pull", iterations=20, storage="bf16")
    assert res["hot_table"] == 1  # the tuned shape
print("ok")
"""


def test_one_launch_whatever_was_tuned(tmp_path):
    assert "ok" in fake_cuda.run(CODE.format(path=str(tmp_path / "plan.txt")))
