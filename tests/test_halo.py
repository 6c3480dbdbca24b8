"""The periodic halo of the ensembles' tiles stays inside the realisation
for every extent (tests/cpp/halo_check.cpp)."""
import os
import subprocess

from tests.conftest import ROOT


def test_halo_places_stay_inside(tmp_path):
    exe = str(tmp_path / "halo_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1",
                        "-I" + os.path.join(ROOT, "sledgehamr_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "halo_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
