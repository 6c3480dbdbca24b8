"""Tiles of the one-pass RKN4 steps (tests/cpp/fuse_plan_check.cpp)."""
import os
import subprocess

from tests.conftest import ROOT


def test_plan_equals_the_exhaustive_search(tmp_path):
    exe = str(tmp_path / "fuse_plan_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2",
                        "-I" + os.path.join(ROOT, "sledgehamr_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "fuse_plan_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
