"""Facets far smaller than the wavelength, where the contour's differences of cosines near 1 lose
most of their digits: the short forms give way to it, so the result keeps the reference's own
rounding.  1e-10 of the largest amplitude, the drop-in's bar, in the median of six meshes
(CUDA's and the C library's cosines differ by a unit in the last place now and then, which
alone can make 7e-10 of it at a radius of a 2,000th of the wavelength)."""
import numpy as np
import pytest

import abt_b200
from oracle import oracle as O
from tests.helpers import outbeams, rel_err
from tests.test_gpu_fp64_forms import _polygon

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lam,radius", [(20.0, 0.01), (20.0, 0.1), (0.532, 0.001)])
@pytest.mark.parametrize("nv", [3, 4, 6])
def test_small_facets(ctx, lam, radius, nv):
    th = np.linspace(5.0, 175.0, 61) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(60) * 6.0) * abt_b200.PI_REF / 180.0
    err = []
    for seed in range(6):
        rng = np.random.default_rng(100 * nv + seed)
        polys = [_polygon(rng, nv, radius) for _ in range(8)]
        geo = abt_b200.make_geometry(np.concatenate(polys), [list(range(i * nv + 1, (i + 1) * nv + 1)) for i in range(8)])
        obs = outbeams(8, rng, 8)
        got = ctx.diff_main(obs, None, geo, th, ph, lam, precision="fp64")[0]
        err.append(rel_err(got, O.diff_main(th, ph, lam, geo, obs, obs[:0])[0]))
    assert np.median(err) <= 1e-10, err
