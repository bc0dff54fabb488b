"""Device allocations that fail part way through a call: the call reports it,
and what it left behind is not used by the next call.  After every failure the
same call succeeds and launches what it launches on a mapping where nothing
had failed (the kernels that fill an array run for every array that is read)."""
import pytest

import fake_cuda

HEAD = """
rng = np.random.default_rng(1)
V, E = 5000, 70000
g = gg.Graph.from_edges(rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32), num_vertices=V)
"""

TAIL = """
dg = gg.DeviceGraph(g, gg.MAP_ALL)
F.fake_fail_mallocs_from(-1)
F.fake_log_clear()
call(dg)
want, allocs = sorted(launches()), F.fake_mallocs()
dg.free()
gg.device_cache_trim()
assert want and allocs
for n in range(allocs):
    dg = gg.DeviceGraph(g, gg.MAP_ALL)
    gg.device_cache_trim()
    F.fake_fail_mallocs_from(n)
    try:
        call(dg)
        raise SystemExit(f"allocation {n} of {allocs} failed unnoticed")
    except gg.GgError:
        pass
    F.fake_fail_mallocs_from(-1)
    done = launches()
    F.fake_log_clear()
    call(dg)
    again = done + launches()  # what the failed call finished need not be done again
    missing = [k for k in set(want) if again.count(k) < want.count(k)]
    assert not missing, (n, missing)
    dg.free()
    gg.device_cache_trim()
    F.fake_log_clear()
print("ok")
"""


@pytest.mark.parametrize("call", ["dg.pagerank('pull', iterations=3, hot=True)",
                                  "dg.pagerank('pull_q16', iterations=3, hot=True)",
                                  "dg.pagerank('push', iterations=40)", "dg.pagerank('pull', iterations=3)",
                                  "dg.spmv('pull', iterations=3)", "dg.ppr([[1], [2, 3]], iterations=3)",
                                  "dg.cc('afforest')"])
def test_call_after_a_failed_allocation(call):
    code = HEAD + f"def call(dg):\n    {call}\n" + TAIL
    assert "ok" in fake_cuda.run(code)
