"""Builds native_calls.cpp against the library and loads it (ctypes)."""
import ctypes
import functools
import os
import subprocess
import tempfile

from conftest import PKG

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@functools.lru_cache(maxsize=None)
def load():
    import sadmrg
    lib = sadmrg.LIB_PATH
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native_calls.cpp")
    out = os.path.join(tempfile.mkdtemp(prefix="sadmrg_native_"), "native_calls.so")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I" + os.path.join(PKG, "csrc"),
                        "-I" + os.path.join(CUDA, "include"), src, lib,
                        "-Wl,-rpath," + os.path.dirname(os.path.abspath(lib)), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def ptr(x):
    """The address of a torch tensor's or numpy array's data."""
    return ctypes.c_void_p(x.data_ptr() if hasattr(x, "data_ptr") else x.ctypes.data)
