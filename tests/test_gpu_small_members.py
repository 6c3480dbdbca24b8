"""Ensembles of small realisations whose arrays end with an allocation (2 MiB
granules): tiles are wider than the realisations, and their halo must not
reach past the last one.  The last member gets the first one's state and has
to come out the same, bit for bit, as the only member of an ensemble."""
import numpy as np
import pytest

import sledgehamr_gb300 as sh
from tests.test_gpu_ensemble import axion_state, fopt_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,precision,N,members", [
    (sh.FAMILY_AXION_LAP1, sh.PREC_FP64, 8, 512),
    (sh.FAMILY_AXION_LAP2, sh.PREC_FP64, 16, 64),
    (sh.FAMILY_AXION_LAP1, sh.PREC_FP32_KAHAN, 16, 128),
    (sh.FAMILY_AXION_LAP2, sh.PREC_FP32_KAHAN, 8, 1024),
    (sh.FAMILY_AXION_LAP2, sh.PREC_FP32, 16, 128),
    (sh.FAMILY_FOPT_GW, sh.PREC_FP64, 16, 64),
    (sh.FAMILY_FOPT_GW, sh.PREC_FP32_KAHAN, 8, 1024),
])
def test_last_small_member_equals_the_first(ctx, family, precision, N, members):
    size = 8 if precision == sh.PREC_FP64 else 4
    assert members * N ** 3 * size % (1 << 21) == 0
    fopt = family == sh.FAMILY_FOPT_GW
    state = (fopt_state if fopt else axion_state)(N, 0.25 * N, 5)
    params = [-1.0, 1.0, -0.1, 0.0] if fopt else [0.8, 0.3, 0.0, 0.0]
    got = []
    for n in (1, members):
        with sh.Ensemble(ctx, family, precision, [N] * n, [0.25] * n, params * n) as E:
            for r in {0, n - 1}:
                E.write(r, state)
            E.set_time(1.0)
            E.step(0.03125, 3)
            got += [E.read(r) for r in (0, n - 1)]
    assert np.isfinite(got[0]).all() and not np.array_equal(got[0], state)
    for g in got[1:]:
        assert np.array_equal(g, got[0])


@pytest.mark.parametrize("precision", [sh.PREC_FP32, sh.PREC_FP32_KAHAN])
def test_one_pass_blocks_of_small_members(ctx, precision):
    """Members of up to 10^3 step in blocks of 16 x 16 threads, with a larger
    one beside them in blocks of 32 x 32: the same bits."""
    sizes = [8, 9, 10, 8]
    out = []
    for Ns in (sizes, sizes + [11]):
        with sh.Ensemble(ctx, sh.FAMILY_AXION_LAP1, precision, Ns, [0.25] * len(Ns),
                         [[0.5 + 0.1 * r, 0.2, 0, 0] for r in range(len(Ns))]) as E:
            for r, n in enumerate(Ns):
                E.write(r, axion_state(n, 0.25 * n, r))
            E.set_time(1.0)
            E.step(0.0625, 3)
            out.append([E.read(r) for r in range(len(sizes))])
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
