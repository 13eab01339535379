"""Runs a script in a child process whose CUDA runtime is fake_cudart.c, so
that the library's host code can be tested where there is no GPU."""
import os
import subprocess
import sys
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "fake_cudart.c")
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


def run(tmp_path, script: str) -> str:
    """The script's output; it finds K, np, ctx and fake (the fake_* functions)."""
    so = os.path.join(str(tmp_path), "libfakecudart.so")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-I" + CUDA_INCLUDE, SRC, "-o", so], check=True)
    env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(script)], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
