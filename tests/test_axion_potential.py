"""The axion-string potential is as accurate as the equation written out
(tests/cpp/axion_potential_check.cpp)."""
import os
import subprocess

from tests.conftest import ROOT


def test_rate_no_less_accurate_than_written_out(tmp_path):
    exe = str(tmp_path / "axion_potential_check")
    inc = ["-I" + os.path.join(ROOT, *p) for p in (("sledgehamr_gb300", "projects"),
                                                   ("include", "sledgehamr"))]
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-w"] + inc +
                       [os.path.join(ROOT, "tests", "cpp", "axion_potential_check.cpp"), "-o",
                        exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
