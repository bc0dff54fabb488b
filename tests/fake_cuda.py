"""The product library linked with tests/fake_cuda.c in place of cudart: its
host code runs without a GPU, and allocations and launches can be made to fail.

run(code) executes `code` in a process of its own (a second copy of the library
cannot share one with the real one), with `gg` the package on the fake library
and `F` the library's handle with the fake's own functions."""
import glob
import os
import subprocess
import sys
import tempfile
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PRELUDE = """
import ctypes as C, sys
import numpy as np
import accelgraph_express_gb300 as gg
gg.LIB_PATH = sys.argv[1]
F = gg.lib()
F.fake_mallocs.restype = C.c_long
F.fake_fail_mallocs_from.argtypes = [C.c_long]
F.fake_log.restype = C.c_char_p
F.fake_smem.restype = C.c_long
F.fake_shared_size.argtypes = [C.c_long]

def launches():
    return F.fake_log().decode().split()

gg.device_init(0)
"""


def run(code, timeout=300):
    import accelgraph_express_gb300 as gg

    gg.build()
    objs = sorted(glob.glob(os.path.join(ROOT, "accelgraph_express_gb300", "_build", "*.o")))
    assert objs
    with tempfile.TemporaryDirectory() as d:
        so = os.path.join(d, "libfake.so")
        subprocess.check_call(["gcc", "-O1", "-fPIC", f"-I{CUDA}/include", "-c", os.path.join(ROOT, "tests", "fake_cuda.c"),
                               "-o", os.path.join(d, "fake.o")])
        subprocess.check_call(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, os.path.join(d, "fake.o"), *objs, "-fopenmp",
                               "-lpthread", "-ldl"])
        script = PRELUDE + textwrap.dedent(code)
        r = subprocess.run([sys.executable, "-c", script, so], cwd=ROOT, capture_output=True, text=True, timeout=timeout,
                           env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0, f"exit {r.returncode}\n{r.stdout}\n{r.stderr}"
    return r.stdout
