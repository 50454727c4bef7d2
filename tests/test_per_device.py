"""CPU test of the per-device setup of kernels (csrc/per_device.hpp): the attributes that a kernel needs for
its shared memory belong to a device, so a second device of the process needs them set again."""
import ctypes
import os
import re
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "votca_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("pd") / "per_device_shim.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread",
                    os.path.join(HERE, "per_device_shim.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def test_once_per_device(lib):
    n = ctypes.c_int(0)
    run = lambda dev, fail=0: (lib.per_device_run(dev, fail, ctypes.byref(n)), n.value)
    assert run(0) == (0, 1) and run(0) == (0, 1)
    assert run(1) == (0, 2) and run(0) == (0, 2) and run(1) == (0, 2)
    assert run(63) == (0, 3) and run(63) == (0, 3)
    assert run(2, 1) == (1, 3) and run(2) == (0, 4) and run(2) == (0, 4)  # again after a failure
    assert run(64) == (0, 5) and run(64) == (0, 6)  # beyond the counted ones: every time
    lib.per_device_threads(7, 16, ctypes.byref(n))
    assert n.value == 7


def test_no_kernel_is_set_up_once_per_process():
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        src = open(os.path.join(CSRC, f)).read()
        for m in re.finditer(r"cudaFuncSetAttribute\(", src):
            before = src[max(0, m.start() - 400):m.start()]
            assert "call_once" not in before, f
            assert "PerDevice" in before or "configured[dev]" in before, f
