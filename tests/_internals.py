"""internals.cu, compiled once per session for the tests that look inside the library."""
import ctypes as C
import functools
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "peridigm_b200", "csrc")


@functools.lru_cache(maxsize=None)
def load():
    so = os.path.join(tempfile.mkdtemp(prefix="internals_"), "internals.so")
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", CSRC, os.path.join(HERE, "internals.cu"), "-o", so],
                   check=True)
    return C.CDLL(so)
