"""Pull products repeated in one call: they alternate between two buffers, so
every count of them has to leave the same y (or zeros, for none), on mappings
used before with another count, with the hot-vertex table and without."""
import numpy as np
import pytest

from fpcheck import assert_fp_as_accurate
from graphs import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hot", [False, True])
@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_repeated_products(gpu, orc, hot, storage):
    g, o = pair(gpu, orc, gpu.Graph.rmat(13, 16, weighted=True))
    dg = gpu.DeviceGraph(g, gpu.MAP_IN | gpu.MAP_IN_W)
    x = np.random.default_rng(3).random(g.V).astype(np.float32)
    _, ry, _ = orc.spmv(o, 0, 1, x=x)
    ex = orc.spmv_f64(o, x)
    for its in (3, 2, 1, 0, 4, 1):
        _, y, res = dg.spmv("pull", storage=storage, iterations=its, x=x, hot=hot)
        if its == 0:
            assert not y.any()
        elif storage == "f32":
            assert_fp_as_accurate(y, ry, ex, f"{its} products")
        else:  # both factors rounded to 8 bits, non-negative (2^-8), and the FP32 sums
            assert np.abs(y - ex).sum() <= (2.0**-8 + 2e-4) * np.abs(ex).sum()
    dg.free()
