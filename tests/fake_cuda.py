"""Runs a script in a child process whose CUDA runtime is fake_cudart.c, so
that the library's host code can be tested where there is no GPU, or whose
device allocations limit_cudart.c refuses."""
import os
import subprocess
import sys
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "fake_cudart.c")
LIMIT_SRC = os.path.join(ROOT, "tests", "limit_cudart.c")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

PRELUDE = """
import ctypes as C
import numpy as np
import kclistpp_gb300 as K
fake = C.CDLL(None)
fake.fake_launches.restype = fake.fake_instantiations.restype = fake.fake_allocations.restype = C.c_ulong
fake.fake_malloc_limit.argtypes = fake.fake_allocations.argtypes = [C.c_size_t]
COST = C.CFUNCTYPE(C.c_double, C.c_char_p, C.c_uint, C.c_uint, C.c_ulong)
ctx = K.Context(0)
"""


LIMIT_PRELUDE = """
import ctypes as C
import numpy as np
import kclistpp_gb300 as K
limit = C.CDLL(None)
limit.limit_exact.argtypes = [C.c_size_t, C.c_long]
limit.limit_refused.restype = C.c_ulong
ctx = K.Context(0)
"""


def _child(tmp_path, src: str, prelude: str, script: str) -> str:
    so = os.path.join(str(tmp_path), os.path.basename(src) + ".so")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-I" + CUDA_INCLUDE, src, "-o", so, "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", prelude + textwrap.dedent(script)], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def run(tmp_path, script: str) -> str:
    """The script's output; it finds K, np, ctx and fake (the fake_* functions)."""
    return _child(tmp_path, SRC, PRELUDE, script)


def run_limited(tmp_path, script: str) -> str:
    """The script's output on the GPU; it finds K, np, ctx and limit (the limit_*
    functions of limit_cudart.c)."""
    return _child(tmp_path, LIMIT_SRC, LIMIT_PRELUDE, script)
