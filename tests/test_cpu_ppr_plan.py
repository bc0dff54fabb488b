"""Tile sizes of the batched PageRank from a plan file: whatever the file holds, the
gather gets a power of two that it can run (its tiles and chunks are masked)."""
import pytest

import fake_cuda

CODE = """
with open({path!r}, "w") as f:
    for v in range(1, 32):
        for d in range(0, 12):
            for k in range(0, 26):
                f.write(f"{{gg.TUNE_PPR}} 0 {{v}} {{d}} {{k}} 152 0 : {tile} 0 0 0 0\\n")
gg.tune_load({path!r})
rng = np.random.default_rng(1)
for V, E in ((500, 5000), (50000, 2000000)):
    g = gg.Graph.from_edges(rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32), num_vertices=V)
    dg = gg.DeviceGraph(g, gg.MAP_IN)
    dg.ppr([[1], [2, 3]], iterations=2)
    tile = dg.tuned(gg.TUNE_PPR)[0]
    assert tile >= 32 and tile & (tile - 1) == 0, tile
    assert tile >= 256 or tile * 152 * 20 >= E, tile
    if {tile} >= 256 and {tile} & ({tile} - 1) == 0:
        assert tile == {tile}
print("ok")
"""


@pytest.mark.parametrize("tile", [1, 16, 48, 255, 256, 300, 384, 512, 1000, 1024, 4294967295])
def test_tile_from_a_plan(tile, tmp_path):
    assert "ok" in fake_cuda.run(CODE.format(path=str(tmp_path / "plan.txt"), tile=tile))
