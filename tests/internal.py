"""Builds internal_probe.cu against the engine's library and loads it."""
import ctypes
import functools
import os
import subprocess
import tempfile
from pathlib import Path

import dmrg2

HERE = Path(__file__).resolve().parent
PKG = Path(dmrg2.__file__).resolve().parent.parent


@functools.lru_cache(maxsize=1)
def load():
    lib = dmrg2.load_library()
    so = Path(tempfile.mkdtemp(prefix="dmrg2_probe_")) / "probe.so"
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                    "-shared", "-I", str(PKG / "csrc"), str(HERE / "internal_probe.cu"), "-o", str(so),
                    "-L", str(PKG / "dmrg2"), "-ldmrg2_b200", f"-Xlinker=-rpath={PKG / 'dmrg2'}", "-lcudart"],
                   check=True, capture_output=True, text=True)
    assert lib is not None
    return ctypes.CDLL(str(so))


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)
