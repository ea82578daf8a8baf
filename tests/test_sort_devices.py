"""The radix sorts' host side with two devices in one process, on the CPU (tests/cpp/
test_sort_devices.cpp): sort.cu linked against a stand-in for the CUDA runtime, so that what a
launch needs of its device is checked where there is one GPU or none."""
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_sorts_opt_in_on_every_device(tmp_path):
    from nbody_gb300 import build
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    csrc, include = ROOT / "nbody_gb300" / "csrc", ROOT / "include"
    obj, exe = tmp_path / "sort.o", tmp_path / "test_sort_devices"
    for cmd in ([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-I", str(include), "-I", str(csrc), "-c",
                 str(csrc / "sort.cu"), "-o", str(obj)],
                ["g++", "-std=c++17", "-I", build.cuda_include(), "-I", str(include), "-I", str(csrc),
                 str(ROOT / "tests" / "cpp" / "test_sort_devices.cpp"), str(obj), "-o", str(exe)], [str(exe)]):
        r = subprocess.run([str(c) for c in cmd], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr[-3000:]
