"""Admitting to and releasing from a pool of one-pass members costs about
what it does in a pool of the 13-point family, which plans no such tiles."""
import time

import pytest

import sledgehamr_gb300 as sh

pytestmark = pytest.mark.gpu


def test_admission_to_a_large_pool(ctx):
    took = {}
    for family in (sh.FAMILY_AXION_LAP1, sh.FAMILY_AXION_LAP2):
        E = sh.Ensemble.pool(ctx, family, sh.PREC_FP32_KAHAN, 25 * 128 ** 3)
        for _ in range(24):
            assert E.admit(128, 0.25, (1.0, 0.0, 0.0, 0.0)) is not None
        times = []
        for _ in range(15):
            ctx.synchronize()
            t = time.perf_counter()
            E.release(E.admit(128, 0.25, (1.0, 0.0, 0.0, 0.0)))
            times.append(time.perf_counter() - t)
        took[family] = sorted(times)[len(times) // 2]
        E.close()
    # 4.7 ms against 0.13 when every depth's tiles were listed and sorted
    assert took[sh.FAMILY_AXION_LAP1] <= 8 * took[sh.FAMILY_AXION_LAP2], took
