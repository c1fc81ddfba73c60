"""The engine's host code on a fake CUDA runtime of two devices (tests/cpp/fake_cudart.cpp): the objects of the built
library, linked with the fake in place of the runtime.  Scripts run in a process of their own, as
`ed` (the package on that library) and `fake` (the library, for the fake's own calls)."""

import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROLOGUE = """
import ctypes, sys
import numpy as np
import alps_b200 as ed
ed.LIB_PATH = sys.argv[1]
fake = ed.lib()
fake.fake_set_cost.argtypes = [ctypes.c_char_p, ctypes.c_double]
fake.fake_pool_bytes.restype = ctypes.c_size_t
"""


def link(folder):
    from alps_b200 import build as b

    b.build()
    lib = os.path.join(folder, "libaed_fake.so")
    objs = [os.path.join(b.BUILD, s + ".o") for s in b.CU_SOURCES + b.CPP_SOURCES]
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I" + os.path.join(b.CUDA_HOME, "include"),
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp")] + objs + ["-o", lib, "-lpthread"], check=True)
    return lib


def run(lib, script, env=None):
    r = subprocess.run([sys.executable, "-c", PROLOGUE + script, lib], cwd=ROOT, capture_output=True, text=True,
                       timeout=300, env={**os.environ, **(env or {})})
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
