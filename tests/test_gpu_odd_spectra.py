"""Scalar spectra of levels with an odd number of cells a side against
numpy's full transform: every mode once, in the bin of its k^2.  Tolerance:
the repository's 1e-10 per bin, plus 1e-14 of the largest."""
import math

import numpy as np
import pytest

import sledgehamr_gb300 as sh
from tests.test_gpu_outputs import axion_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,max_grid", [(9, 0), (15, 8), (33, 0), (49, 16)])
def test_scalar_spectrum_of_odd_grids(ctx, N, max_grid):
    dx, t = 0.25, 1.3
    st = axion_state(N)
    lv = sh.Level.periodic(ctx, "AxionStringsLap1", N, 1, max_grid=max_grid)
    lv.write(st)
    lv.set_time(t)
    bins, ks = lv.scalar_spectrum(0, dx, 1)
    lv.close()
    k = np.rint(np.fft.fftfreq(N, 1 / N)).astype(np.int64) ** 2
    k2 = (k[:, None, None] + k[None, :, None] + k[None, None, :]).ravel()
    want_ks = np.unique(k2)
    assert np.array_equal(ks, want_ks)
    power = np.abs(np.fft.fftn(st[1])).ravel() ** 2
    pre = t / (float(N) ** 6 * 2 * math.pi / (N * dx))
    want = pre * np.bincount(np.searchsorted(want_ks, k2), power, len(want_ks))
    assert np.all(np.abs(bins - want) <= 1e-10 * want + 1e-14 * want.max())
