"""Dependent launches of the plain pull gathers: exactly the CTAs per SM that the
launch is sized for fit the carve-out that it selects (a share in percent selects
the smallest carve-out at least as large), so that no SM takes more of them."""
import pytest

import fake_cuda

CODE = """
CTAS = {ctas}
STATIC = {static}
F.fake_shared_size(STATIC)
with open("/tmp/carveout_plan_{ctas}_{static}.txt", "w") as f:
    for fam in (gg.TUNE_PR, gg.TUNE_SPMV):
        for v in range(1, 32):
            for d in range(0, 12):
                for k in range(0, 26):
                    f.write(f"{{fam}} 0 {{v}} {{d}} {{k}} 152 0 : 0 {{CTAS}} 32 0 0\\n")
gg.tune_load("/tmp/carveout_plan_{ctas}_{static}.txt")
rng = np.random.default_rng(1)
V, E = 300000, 3000000
g = gg.Graph.from_edges(rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32), num_vertices=V)
dg = gg.DeviceGraph(g, gg.MAP_ALL)
dg.pagerank("pull", iterations=2, hot=False)
dg.spmv("pull", iterations=2, hot=False)
SM = 233472
for name in (b"k_pr_pullILi0E", b"k_spmv_pullIf"):
    pct, pad = F.fake_carveout(name), F.fake_smem(name)
    config = min(k * 1024 for k in (8, 16, 32, 64, 100, 132, 164, 196, 228) if k * 1024 * 100 >= pct * SM)
    block = STATIC + 1024 + pad
    assert STATIC + pad <= 48 * 1024
    assert CTAS * block <= config < (CTAS + 1) * block, (name, pct, pad, config, block)
print("ok")
"""


@pytest.mark.parametrize("ctas", [3, 4, 5, 6, 8])
@pytest.mark.parametrize("static", [19456, 12800])
def test_carveout_holds_the_ctas_and_no_more(ctas, static, tmp_path):
    code = CODE.replace("/tmp/carveout", str(tmp_path) + "/carveout")
    assert "ok" in fake_cuda.run(code.format(ctas=ctas, static=static))
