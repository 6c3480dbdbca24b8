"""Projects of a user's own, compiled and linked with the library's objects,
stepped on the GPU in a process of their own."""
import glob
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

PKG = os.path.join(ROOT, "sledgehamr_gb300")


def library_with(source, tmp_path):
    """A copy of the library with the project of tests/cpp/<source> linked in."""
    from sledgehamr_gb300 import build as pkg_build
    pkg_build.build()
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    obj, so = str(tmp_path / "project.o"), str(tmp_path / "libwithproject.so")
    for cmd in ([nvcc] + pkg_build.ARCH + pkg_build.NVCC_FLAGS +
                ["-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(PKG, "projects"), "-c",
                 os.path.join(ROOT, "tests", "cpp", source), "-o", obj],
                [nvcc] + pkg_build.ARCH + ["-shared", "-o", so] +
                glob.glob(os.path.join(PKG, "_build", "*.o")) +
                [obj, "-lcufft", "-lcudart", "-Xcompiler", "-fopenmp"]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr[-3000:]
    return so


def run_with(so, body):
    """body in a process that has loaded the library `so`."""
    head = f"""
        import numpy as np
        from sledgehamr_gb300 import _lib
        _lib.LIB_PATH = {so!r}
        import sledgehamr_gb300 as sh
        from tests.conftest import rel_l2
        from tests.test_gpu_parity import axion_state
        ctx = sh.Context(0)
    """
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(head) + textwrap.dedent(body)],
                       capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr[-3000:]


def test_shipped_rhs_inside_a_users_project(tmp_path):
    """With its own term at zero the project is AxionStringsLap1, up to the
    rounding of the equation's constants (formed here in the hook, there on
    the host): 4 steps of 3 stages, each within some 1e-16; and the term acts.
    """
    run_with(library_with("reuse_project.cu", tmp_path), """
        N = 24
        st = axion_state(N, N * 0.25)
        kw = dict(t0=1.0, dt=0.05, dx=0.25, nsteps=4, nghost=1)
        for integ in (sh.RKN4, sh.LSSSPRK3, sh.LEAPFROG):
            want = ctx.evolve_periodic("AxionStringsLap1", integ, st, params=[0.8, 0.3], **kw)
            got = ctx.evolve_periodic("DrivenStrings", integ, st, params=[0.8, 0.3, 0.0], **kw)
            assert rel_l2(got, want) <= 1e-14, (integ, rel_l2(got, want))
            driven = ctx.evolve_periodic("DrivenStrings", integ, st, params=[0.8, 0.3, 5.0], **kw)
            assert rel_l2(driven, want) > 1e-3
    """)


def test_dissipation_of_an_odd_number_of_fields(tmp_path):
    """Three fields with one state and one strength stay equal, bit for bit,
    and are smoothed, for both orders."""
    run_with(library_with("odd_project.cu", tmp_path), """
        N = 16
        st = np.repeat(axion_state(N, N * 0.25)[:1], 3, axis=0)
        for order in (2, 3):
            got = ctx.evolve_periodic("ThreeFields", sh.LSSSPRK3, st, t0=1.0, dt=0.05, dx=0.25,
                                      nsteps=3, nghost=3, ko_order=order, ko_strength=[0.3] * 3)
            assert not np.array_equal(got[0], st[0])
            assert np.array_equal(got[1], got[0]) and np.array_equal(got[2], got[0]), order
    """)
