"""Runs a script in a process of its own whose calls of the CUDA runtime pass
through fake_cuda.c: allocations above a limit fail with the runtime's own error
code, cooperative launches can be refused; nothing reaches the GPU that would not
be valid there.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))

PRELUDE = """
import ctypes, os
fake = ctypes.CDLL(os.environ["FAKE_CUDA"])
for f, a, r in (("fake_limit", [ctypes.c_size_t], None), ("fake_no_cooperative", [ctypes.c_int], None),
                ("fake_used", [], ctypes.c_size_t), ("fake_peak", [ctypes.c_int], ctypes.c_size_t),
                ("fake_refused", [], ctypes.c_long), ("fake_allocs", [], ctypes.c_long),
                ("fake_copies", [], ctypes.c_long)):
    getattr(fake, f).argtypes, getattr(fake, f).restype = a, r
import numpy as np
import fortran_airtools_gb300 as fair
from fortran_airtools_gb300._clib import FairError, check, lib, FAIR_ERR_ALLOC
"""


def run(tmp_path, script):
    """The script's standard output; a failed assertion in it fails the test."""
    from fortran_airtools_gb300.build import cuda_home, nvcc_path
    so, cuda = str(tmp_path / "fake_cuda.so"), cuda_home(nvcc_path())
    # linked against the runtime, which is then loaded right behind it
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"), "-o", so,
                    os.path.join(HERE, "fake_cuda.c"), "-L", os.path.join(cuda, "lib64"), "-Wl,--no-as-needed",
                    "-lcudart", "-Wl,-rpath," + os.path.join(cuda, "lib64"), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=so, FAKE_CUDA=so, PYTHONPATH=os.path.dirname(HERE))
    r = subprocess.run([sys.executable, "-c", PRELUDE + script], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout + r.stderr)
    return r.stdout
