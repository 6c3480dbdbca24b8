"""What follows the creation of an ensemble at once is not undone by the
clearing of its arrays."""
import numpy as np
import pytest

import sledgehamr_gb300 as sh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,ncomp", [(sh.FAMILY_FOPT_GW, 14), (sh.FAMILY_AXION_LAP2, 4)])
def test_time_and_state_set_right_after_creation(ctx, family, ncomp):
    N = 96
    state = np.random.default_rng(1).standard_normal((ncomp, N, N, N)).astype(np.float32)
    for _ in range(5):
        with sh.Ensemble(ctx, family, sh.PREC_FP32_KAHAN, [N] * 4, [0.25] * 4) as E:
            E.set_time(3.0)
            E.write(3, state)
            assert E.time() == 3.0
            assert np.array_equal(E.read(3), state)
            assert not E.read(0).any()
