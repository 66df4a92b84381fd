"""finalise on grids at the edges of its panel chunks (32 rows, 32 phi panels, 256 theta panels),
odd and even lengths, against the CPU oracle (1e-12, the bar of the FP64 epilogue)."""
import numpy as np
import pytest

import abt_b200
from oracle import oracle as O
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,nphi", [(3, 3), (4, 4), (31, 65), (32, 66), (33, 67), (514, 5), (515, 6), (1027, 130)])
@pytest.mark.parametrize("scaling", [False, True])
def test_grid_edges(ctx, nt, nphi, scaling):
    rng = np.random.default_rng(nt + nphi)
    # uneven spacing, near enough to even for the rule's weights to stay positive
    th = 0.02 + 3.0 * (np.arange(nt) + rng.uniform(0, 0.2, size=nt)) / nt
    ph = 6.2 * (np.arange(nphi) + rng.uniform(0, 0.2, size=nphi)) / nphi
    a, b = (np.asfortranarray(rng.normal(size=(nphi, nt, 2, 2)) + 1j * rng.normal(size=(nphi, nt, 2, 2)))
            for _ in range(2))
    pin = abt_b200.params(abs=0.4, geo_cross_sec=7.0, beam_energy_out=3.0, ext_energy_out=5.0)
    mu, m1, p = ctx.finalise(a, b, th, ph, 0.532, pin, scaling=scaling)
    rmu, rm1, want = O.finalise(a, b, th, ph, 0.532, np.array(pin.tolist()), scaling=scaling)
    assert rel_err(mu, rmu) <= 1e-12
    assert rel_err(m1, rm1) <= 1e-12
    got = np.array([p[n] for n in abt_b200.PARAM_NAMES])
    # the integrals cancel between panels of random data: relative to the largest parameter
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
