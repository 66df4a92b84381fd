"""The FP64 sum's short forms against the CPU oracle where they can go wrong: list lengths
around the staged chunks and the facet runs, polygons of every corner count, wavelengths and
facet sizes that move every lane to the contour, clamped edge slopes, an empty list.

Bar: 1e-10 of the largest amplitude, as for the drop-in.  The short forms agree with the
contour to 5e-11 of a facet's own area by the rule that chooses between them.
"""
import numpy as np
import pytest

import abt_b200
from abt_b200 import workloads as W
from oracle import oracle as O
from tests.helpers import outbeams, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _grid(nt=19, nphi=13, lo=0.0):
    th = np.linspace(lo, 180.0 - lo, nt) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(nphi) * 360.0 / nphi) * abt_b200.PI_REF / 180.0
    return th, ph


def _polygon(rng, nv, radius):
    n = rng.normal(size=3)
    n /= np.linalg.norm(n)
    e1 = np.cross(n, rng.normal(size=3))
    e1 /= np.linalg.norm(e1)
    e2 = np.cross(n, e1)
    ang = 2 * np.pi * (np.arange(nv) + rng.uniform(0, 0.5, size=nv)) / nv
    return rng.uniform(-5, 5, size=3) + radius * (np.cos(ang)[:, None] * e1 + np.sin(ang)[:, None] * e2)


def _check(ctx, geo, beam, ext, th, ph, lam, fast=False):
    got = ctx.diff_main(beam, ext, geo, th, ph, lam, is_fast_diff=fast, precision="fp64")
    ref = O.diff_main(th, ph, lam, geo, beam, ext, is_fast_diff=fast)
    for g, r in zip(got, ref):
        ok = np.isfinite(r)
        assert np.array_equal(np.isfinite(g), ok)
        assert rel_err(g[ok], r[ok]) <= TOL
        if fast:
            assert np.array_equal(g == 0, r == 0)


@pytest.mark.parametrize("nbeam,next_", [(1, 0), (0, 1), (15, 2), (16, 17), (33, 47), (95, 16), (0, 0)])
def test_list_lengths(ctx, nbeam, next_):
    rng = np.random.default_rng(100 + nbeam)
    geo, _, _ = W.synthetic_beam_list(n_beams=4, facets_per_beam=10, seed=3, cube=10.0)
    beam, ext = outbeams(nbeam, rng, 40), outbeams(next_, rng, 40, prop=(0, 0, -1))
    for fast in (False, True):
        _check(ctx, geo, beam, ext, *_grid(), 0.532, fast)


@pytest.mark.parametrize("nv", [3, 4, 5, 8, 17])
@pytest.mark.parametrize("radius", [0.05, 0.8, 30.0])
def test_polygons(ctx, nv, radius):
    rng = np.random.default_rng(7 * nv)
    polys = [_polygon(rng, nv, radius) for _ in range(5)]
    geo = abt_b200.make_geometry(np.concatenate(polys), [list(range(i * nv + 1, (i + 1) * nv + 1)) for i in range(5)])
    _check(ctx, geo, outbeams(6, rng, 5), outbeams(3, rng, 5, prop=(0, 0, -1)), *_grid(lo=1.5), 0.532)


@pytest.mark.parametrize("lam", [0.005, 0.02, 12.0])
def test_wavelengths(ctx, lam):
    """0.005 um: phases beyond the kernel's argument reduction (the contour everywhere)."""
    rng = np.random.default_rng(5)
    geo, _, _ = W.synthetic_beam_list(n_beams=1, facets_per_beam=6, seed=9, cube=4.0)
    # the phase k |x| grows with 1/lambda, and with it what one ulp of it is worth
    th, ph = _grid(lo=4.0)
    got = ctx.diff_main(outbeams(6, rng, 6), None, geo, th, ph, lam, precision="fp64")[0]
    rng = np.random.default_rng(5)
    ref = O.diff_main(th, ph, lam, geo, outbeams(6, rng, 6), np.zeros(0, abt_b200.OUTBEAM_DTYPE))[0]
    assert rel_err(got, ref) <= TOL


def test_clamped_slopes(ctx):
    """Edges along the aperture axes: slopes 0 and infinity, clamped by the reference."""
    rng = np.random.default_rng(2)
    v = np.array([[0, 0, 0], [1.2, 0, 0], [0, 0.9, 0], [2, 2, 1], [3.1, 2, 1], [2, 3, 1]], float)
    geo = abt_b200.make_geometry(v, [[1, 2, 3], [4, 6, 5]])
    beam = outbeams(4, rng, 2, prop=(np.sin(0.4), 0.0, -np.cos(0.4)))
    _check(ctx, geo, beam, beam[:0], *_grid(lo=5.0), 0.532)


@pytest.mark.parametrize("lo,hi", [(0.0, 3.2), (1.0, 2.6), (176.8, 180.0)])
def test_forward_bodge(ctx, lo, hi):
    """Rows on both sides of the forward bodge's limit, acos(0.999) = 2.56 degrees from the
    incidence axis, in both hemispheres, and the rows at the axis itself."""
    rng = np.random.default_rng(31)
    geo, _, _ = W.synthetic_beam_list(n_beams=1, facets_per_beam=6, seed=9, cube=4.0)
    th = np.linspace(lo, hi, 33) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(7) * 51.0) * abt_b200.PI_REF / 180.0
    tilt = (np.sin(0.3), 0.0, -np.cos(0.3))
    for sign in (1, -1):
        prop = tuple(sign * x for x in tilt)
        _check(ctx, geo, outbeams(5, rng, 6, prop=prop), outbeams(3, rng, 6, prop=prop), th, ph, 0.532)
