"""Compiles and loads native_shim.cpp against the built library."""
import ctypes
import functools
import os
import subprocess
import tempfile

from votca_gb300 import _lib, build

HERE = os.path.dirname(os.path.abspath(__file__))


@functools.lru_cache(maxsize=None)
def load():
    _lib.load()
    so = os.path.join(tempfile.mkdtemp(prefix="native_shim"), "native_shim.so")
    d = os.path.dirname(_lib.library_path())
    subprocess.run([build.nvcc(), "-std=c++17", "-O1", "-shared", "-Xcompiler", "-fPIC",
                    os.path.join(HERE, "native_shim.cpp"), "-o", so, "-L" + d, "-lvotca_gb300",
                    "-Xlinker", "-rpath=" + d], check=True)
    L = ctypes.CDLL(so)
    L.shim_last_error.restype = ctypes.c_char_p
    return L
