"""Batches whose field-of-view lists are put in order of direction (1e9 outbeam-bins and more a
run): several orientations with vertices of their own, odd, uneven and empty lists, in one run
and in several, against the FP64 batch, the same call under an explicit plan (which keeps the
lists' order), and itself.  Bars: the package's 1e-4 of a bin's M11 and 1e-5 of the cross sections."""
import numpy as np
import pytest

import abt_b200
from tests.helpers import mueller_rel_err, outbeams
from tests.test_gpu_fp32_edges import LAM, _polygon_mesh

pytestmark = pytest.mark.gpu

TILT = (np.sin(0.3), 0, -np.cos(0.3))


@pytest.mark.parametrize("nb,beams,exts,scaling", [
    ((259, 200), (9001, 0, 4003, 3, 3501), (1500, 777, 0, 2001, 35), False),
    ((65, 64), (130001, 90001, 7, 200003, 0, 130000), (1, 45000, 131, 0, 20001, 999), False),
    ((65, 64), (130001, 90001, 7, 200003, 1, 130000), (1, 45000, 131, 2, 20001, 999), True),
    ((65, 64), (130001, 90001, 7, 200003, 0, 130000), (1, 45000, 131, 0, 20001, 999), True)])
@pytest.mark.parametrize("nv", [[3] * 40, [3] * 35 + [7] * 5, [3, 4, 5, 6] * 10])
def test_orientations_in_order_of_direction(ctx, nb, beams, exts, scaling, nv):
    rng = np.random.default_rng(sum(nv))
    geo = _polygon_mesh(rng, nv)
    verts, bl, el = [], [], []
    for n, m in zip(beams, exts):
        q = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        verts.append(geo["verts"] @ q + rng.normal(size=3))
        bl.append(outbeams(n, rng, len(nv)))
        el.append(outbeams(m, rng, len(nv), prop=TILT))
    th = np.linspace(4.0, 180.0, nb[0]) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(nb[1]) * 360.0 / nb[1]) * abt_b200.PI_REF / 180.0
    pin = np.array([abt_b200.params(abs=0.3, geo_cross_sec=10.0, beam_energy_out=2.0)] * len(beams),
                   dtype=abt_b200.PARAMS_DTYPE)

    def run(**kw):
        return ctx.diff_batch(bl, el, verts, geo, th, ph, LAM, pin, is_fast_diff=True, scaling=scaling, **kw)

    got, again, ref = run(precision="fp32"), run(precision="fp32"), run(precision="fp64")
    ctx.set_plan(1, 1, 2048)
    plain = run(precision="fp32")
    ctx.set_plan(-1)
    assert np.array_equal(got[0], again[0], equal_nan=True) and np.array_equal(got[1], again[1], equal_nan=True)
    # an empty list's energies, rescaled, are 0 / 0 in all three
    for r in (ref, plain):
        ok = np.isfinite(r[0]).all(axis=-1)
        assert np.array_equal(np.isfinite(got[0]).all(axis=-1), ok)
        if ok.any():
            assert mueller_rel_err(got[0][ok], r[0][ok]) <= 1e-4
        u, v = (p.view(np.float64).reshape(-1, 18) for p in (got[3], r[3]))
        assert np.array_equal(np.isnan(u), np.isnan(v))
        cols = [c for c in range(18) if c != 9]
        np.testing.assert_allclose(u[:, cols], v[:, cols], rtol=1e-5, atol=1e-5)
