"""Builds device_math_check.cu with the library's flags, once per process, and
loads it."""
import ctypes as C
import functools
import os
import subprocess
import tempfile

from rkdg3d_gb300 import buildlib

HERE = os.path.dirname(os.path.abspath(__file__))


@functools.lru_cache(None)
def load():
    with tempfile.TemporaryDirectory() as tmp:
        out = os.path.join(tmp, "device_math_check.so")
        subprocess.run([buildlib.nvcc_path(), *buildlib.ARCH, "-O3", "-std=c++17", "-ftz=true", "-Xcompiler", "-fPIC",
                        "-shared", "-I", buildlib.INCLUDE, "-I", buildlib.CSRC, os.path.join(HERE, "device_math_check.cu"),
                        "-o", out], check=True)
        return C.CDLL(out)


def ptr(t):
    return C.c_void_p(t.data_ptr())
