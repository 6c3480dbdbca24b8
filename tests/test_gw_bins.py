"""The spectra's bin lists on the host (tests/cpp/gw_bins_check.cpp)."""
import os
import subprocess

from tests.conftest import ROOT


def test_bin_lists_of_even_and_odd_grids(tmp_path):
    exe = str(tmp_path / "gw_bins_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-fopenmp", "-D_GLIBCXX_ASSERTIONS",
                        "-I" + os.path.join(ROOT, "sledgehamr_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "gw_bins_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr[-500:]
