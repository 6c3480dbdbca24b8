"""The FP64 transforms launch on every device of a process: the kernels'
shared-memory limits belong to the device that was current when they were
set (tests/cpp/fft_launch_check.cpp, against a stand-in for the runtime)."""
import glob
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

PKG = os.path.join(ROOT, "sledgehamr_gb300")


def test_transforms_launch_on_every_device(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    from sledgehamr_gb300 import build as pkg_build
    pkg_build.build()
    objs = sorted(glob.glob(os.path.join(PKG, "_build", "sh_fft*.o")))
    exe = str(tmp_path / "fft_launch_check")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    inc = ["-I" + d for d in (cuda, os.path.join(PKG, "csrc"), os.path.join(ROOT, "include"),
                              os.path.join(ROOT, "include", "sledgehamr"))]
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-w"] + inc +
                       [os.path.join(ROOT, "tests", "cpp", "fft_launch_check.cpp")] + objs +
                       ["-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
