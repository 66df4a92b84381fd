"""Edges of the packed FP32 kernel: record counts around its stages and work items (an item's
first and last pair half another's), grids that leave warps of a tile without bins, the
field-of-view cull per warp, and far-field phases beyond the fixed-point range.
"""
import numpy as np
import pytest
import torch

import abt_b200
from abt_b200 import workloads as W
from oracle import adjoint_ref as AR
from tests.helpers import mueller_rel_err, outbeams, rel_err

pytestmark = pytest.mark.gpu

LAM = 0.532


def _grid(nt, nphi):
    th = np.linspace(0.0, 180.0, nt) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(nphi) * 360.0 / nphi) * abt_b200.PI_REF / 180.0
    return th, ph


def _closed_form(obs, geo, th, ph, lam, fast, ext):
    """Sum of the facets' closed-form amplitudes (the contour of the FP64 drop-in cancels at
    theta = 0), each in the bins of its field of view."""
    X = np.stack(abt_b200.make_far_field_bins(th, ph), -1)
    phase = np.exp(2j * abt_b200.PI_REF / lam * np.linalg.norm(X, axis=-1))[:, :, None, None]
    V = torch.from_numpy(np.ascontiguousarray(geo["verts"]))
    F = (geo["face_vi"] - 1).reshape(-1, 3)
    total = np.zeros((len(ph), len(th), 2, 2), complex)
    for ob in obs:
        z = torch.from_numpy(ob["ampl"][0::2] + 1j * ob["ampl"][1::2])
        a = torch.stack([torch.stack([z[0], z[2]]), torch.stack([z[1], z[3]])])[None]
        S = AR.forward(V, F, [ob["fi"] - 1], a, [ob["prop_out"]], [ob["vk7"]], [], None, [], [], th, ph, lam)
        S = S.numpy().reshape(len(th), len(ph), 2, 2).transpose(1, 0, 2, 3) * phase
        if fast:
            d = X - geo["verts"][F[ob["fi"] - 1]].mean(0)
            u = d / np.linalg.norm(d, axis=-1, keepdims=True)
            fov = abt_b200.PI_REF / 2 if ext else ob["fov"]
            S = np.where((u @ ob["prop_out"] < np.cos(fov))[:, :, None, None], 0.0, S)
        total += S
    return total


@pytest.mark.parametrize("counts", [(1, 1), (63, 2), (64, 65), (87, 88), (89, 177), (263, 1)])
@pytest.mark.parametrize("fast", [False, True])
def test_record_counts(ctx, counts, fast):
    """2e-5 of the largest amplitude (FP32 sums of up to 263 facets with phases near 50 rad,
    2e-6 each)."""
    rng = np.random.default_rng(sum(counts))
    geo, _, _ = W.synthetic_beam_list(n_beams=30, facets_per_beam=10, seed=4, cube=10.0)
    beam = outbeams(counts[0], rng, 300)
    ext = outbeams(counts[1], rng, 300, prop=(0, 0, -1))
    th, ph = _grid(21, 37)
    ref = [_closed_form(obs, geo, th, ph, LAM, fast, k == 1) for k, obs in enumerate((beam, ext))]
    fp64 = ctx.diff_main(beam, ext, geo, th, ph, LAM, is_fast_diff=fast, precision="fp64")
    for rpi in (None, 32, 75):
        if rpi:
            ctx.set_plan(1, 1, rpi)
        got = ctx.diff_main(beam, ext, geo, th, ph, LAM, is_fast_diff=fast, precision="fp32")
        ctx.set_plan(-1)
        for g, r, f in zip(got, ref, fp64):
            assert rel_err(g, r) <= 2e-5
            if fast:
                assert np.array_equal(g == 0, f == 0)


@pytest.mark.parametrize("nt,nphi", [(5, 3), (9, 17), (8, 16), (33, 9), (4, 250)])
def test_fast_grids(ctx, nt, nphi):
    """Tiles with empty warps: the FP32 mask is the FP64 drop-in's in every bin."""
    rng = np.random.default_rng(nt * nphi)
    geo, _, _ = W.synthetic_beam_list(n_beams=10, facets_per_beam=10, seed=6, cube=20.0)
    beam = outbeams(80, rng, 100)
    th, ph = _grid(nt, nphi)
    ref = ctx.diff_main(beam, None, geo, th, ph, LAM, is_fast_diff=True, precision="fp64")[0]
    for bpt in (1, 2):
        ctx.set_plan(1, bpt, 64)
        got = ctx.diff_main(beam, None, geo, th, ph, LAM, is_fast_diff=True, precision="fp32")[0]
        ctx.set_plan(-1)
        assert rel_err(got, ref) <= 2e-5
        assert np.array_equal(got == 0, ref == 0)


@pytest.mark.parametrize("lam", [0.532, 1e-3, 1e-5])
def test_far_field_phase(ctx, lam):
    """One facet at c against the same facet at the origin: the amplitudes differ by the phase
    k (|X - c| - |X|) and by terms of order |c| / R = 2e-5.  At 1e-5 um the phase is beyond the
    fixed-point range (k |c| = 7e6 rad).  The FP32 phase is good to 3e-5 rad there (its second
    order, 90 rad, rounded to FP32); the bar of 1e-3 leaves room for the parallax."""
    rng = np.random.default_rng(12)
    c = np.array([7.0, -5.5, 6.1])
    # facet of about 0.1 / k, so that its own aperture integral hardly depends on the bin
    size = 0.1 * lam / (2 * np.pi)
    tri = size * np.array([[1.0, 0.1, 0.3], [-0.6, 0.8, -0.2], [-0.4, -0.9, -0.1]])
    ob = outbeams(1, rng, 1)
    th = np.linspace(20.0, 160.0, 36) * abt_b200.PI_REF / 180.0
    ph = (0.3 + 11.0 * np.arange(32)) * abt_b200.PI_REF / 180.0
    at, origin = (ctx.diff_main(ob, None, abt_b200.make_geometry(tri + o, [[1, 2, 3]]), th, ph, lam,
                                precision="fp32")[0] for o in (c, 0.0 * c))
    com = (tri + c).mean(0)
    X = np.stack([v for v in abt_b200.make_far_field_bins(th, ph)], -1)
    r = np.linalg.norm(X - com, axis=-1)
    phase = 2 * abt_b200.PI_REF / lam * ((com @ com - 2 * X @ com) / (r + 1e6))
    want = origin * np.exp(1j * phase)[:, :, None, None]
    scale = np.abs(origin).max(axis=(-1, -2), keepdims=True)
    # bins within a degree of the facet's y axis, where the polarisation matrix turns fast
    assert np.quantile(np.abs(at - want) / scale, 0.99) <= 1e-3


def test_batch_odd_segments(ctx):
    """Orientations whose lists start at odd records: the FP32 average against the FP64 one."""
    rng = np.random.default_rng(8)
    geo, _, _ = W.synthetic_beam_list(n_beams=10, facets_per_beam=10, seed=7, cube=10.0)
    beams = [outbeams(n, rng, 100) for n in (31, 7, 90, 1)]
    exts = [outbeams(n, rng, 100, prop=(0, 0, -1)) for n in (5, 12, 3, 9)]
    V = [geo["verts"]] * 4
    pin = np.array([abt_b200.params(geo_cross_sec=10.0)] * 4, dtype=abt_b200.PARAMS_DTYPE)
    th, ph = _grid(31, 24)
    a = ctx.diff_batch(beams, exts, V, geo, th, ph, LAM, pin, precision="fp32")
    b = ctx.diff_batch(beams, exts, V, geo, th, ph, LAM, pin, precision="fp64")
    assert mueller_rel_err(a[0], b[0]) <= 1e-4


@pytest.mark.parametrize("norient,nt,nphi", [(1, 5, 3), (3, 41, 33), (40, 7, 5), (70, 16, 16)])
@pytest.mark.parametrize("corners", [3, 4, 0])
@pytest.mark.parametrize("scaling", [False, True])
def test_many_orientations(ctx, norient, nt, nphi, corners, scaling):
    """Epilogue over several orientation groups, lists of triangles, of quads and mixed, some of
    them empty: FP32 average and per-orientation parameters against the FP64 path (1e-4 of a
    bin's M11, 1e-5 of the cross sections, the package's bars)."""
    rng = np.random.default_rng(norient + corners)
    nf = 12
    nv = np.full(nf, corners) if corners else rng.integers(3, 7, size=nf)
    verts, faces = [], []
    for n in nv:
        e = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        ang = 2 * np.pi * (np.arange(n) + rng.uniform(0, 0.5, size=n)) / n
        faces.append(list(range(len(verts) + 1, len(verts) + n + 1)))
        verts += list(rng.uniform(-3, 3, size=3) + np.cos(ang)[:, None] * e[0] + np.sin(ang)[:, None] * e[1])
    geo = abt_b200.make_geometry(np.array(verts), faces)
    beams = [outbeams(int(m), rng, nf) for m in rng.integers(1, 12, size=norient)]
    exts = [outbeams(int(m), rng, nf, prop=(0, 0, -1)) for m in rng.integers(1, 9, size=norient)]
    if norient > 2 and not scaling:
        exts[1] = exts[1][:0]
        beams[2] = beams[2][:0]
    V = [geo["verts"]] * norient
    pin = np.array([abt_b200.params(abs=0.3, geo_cross_sec=10.0, beam_energy_out=2.0)] * norient,
                   dtype=abt_b200.PARAMS_DTYPE)
    th = np.linspace(3.0, 180.0, nt) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(nphi) * 360.0 / nphi) * abt_b200.PI_REF / 180.0
    a = ctx.diff_batch(beams, exts, V, geo, th, ph, LAM, pin, precision="fp32", scaling=scaling)
    b = ctx.diff_batch(beams, exts, V, geo, th, ph, LAM, pin, precision="fp64", scaling=scaling)
    assert mueller_rel_err(a[0], b[0]) <= 1e-4
    for x, y in ((a[2], b[2]), (a[3], b[3])):
        u, v = (np.atleast_1d(p).view(np.float64).reshape(-1, 18) for p in (x, y))
        assert np.array_equal(np.isnan(u), np.isnan(v))
        # the parameters but the back-scattering one (a single bin's M11, under the Mueller bar)
        cols = [c for c in range(18) if c != 9]
        np.testing.assert_allclose(u[:, cols], v[:, cols], rtol=1e-5, atol=1e-5)


def _polygon_mesh(rng, nv):
    verts, faces = [], []
    for n in nv:
        e = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        ang = 2 * np.pi * (np.arange(n) + rng.uniform(0, 0.5, size=n)) / n
        faces.append(list(range(len(verts) + 1, len(verts) + n + 1)))
        verts += list(rng.uniform(-4, 4, size=3) + np.cos(ang)[:, None] * e[0] + np.sin(ang)[:, None] * e[1])
    return abt_b200.make_geometry(np.array(verts), faces)


@pytest.mark.parametrize("nv", [[4] * 30, [16] * 30, [3, 5] * 15, [3] * 25 + [16] * 5, [3] * 29 + [4],
                                list(range(3, 17)) * 2 + [3, 3], [3] * 29 + [40]])
@pytest.mark.parametrize("counts", [(1, 2), (57, 58), (130, 31)])
@pytest.mark.parametrize("fast", [False, True])
def test_polygon_records(ctx, nv, counts, fast):
    """Facets of 3 to 16 vertices as one record each or as fans, neighbours of unequal length,
    lists that begin and end within a pair and a stage (a face of 40 vertices that no outbeam
    uses beside them): 2e-5 of the largest amplitude of the FP64 drop-in, off the forward row
    (facets of radius 1, FP32 phases near 25 rad)."""
    rng = np.random.default_rng(len(nv) + sum(counts))
    geo = _polygon_mesh(rng, nv)
    usable = np.nonzero(np.asarray(nv) <= 16)[0] + 1
    beam, ext = outbeams(counts[0], rng, 1), outbeams(counts[1], rng, 1, prop=(0, 0, -1))
    for ob in (beam, ext):
        ob["fi"] = rng.choice(usable, size=len(ob))
    th = np.linspace(4.0, 180.0, 23) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(35) * 360.0 / 35) * abt_b200.PI_REF / 180.0
    ref = ctx.diff_main(beam, ext, geo, th, ph, LAM, is_fast_diff=fast, precision="fp64")
    for rpi in (None, 33):
        if rpi:
            ctx.set_plan(1, 1, rpi)
        got = ctx.diff_main(beam, ext, geo, th, ph, LAM, is_fast_diff=fast, precision="fp32")
        ctx.set_plan(-1)
        for g, r in zip(got, ref):
            assert rel_err(g, r) <= 2e-5
            if fast:
                assert np.array_equal(g == 0, r == 0)


def test_too_many_vertices(ctx):
    """A face above 16 vertices is refused in FP32 when an outbeam uses it."""
    rng = np.random.default_rng(1)
    th, ph = _grid(9, 8)
    for nv in ([4, 4, 17], [3] * 20 + [17]):
        geo = _polygon_mesh(rng, nv)
        ob = outbeams(3, rng, 1)
        ob["fi"] = len(nv)
        with pytest.raises(abt_b200.PbtError):
            ctx.diff_main(ob, None, geo, th, ph, LAM, precision="fp32")


@pytest.mark.parametrize("offset", [0.0, 55.0, 68.0, 160.0])
@pytest.mark.parametrize("rows", [(0.1, 3.2), (176.8, 179.9), (20.0, 160.0)])
@pytest.mark.parametrize("corners", [3, 5])
@pytest.mark.parametrize("fast", [False, True])
def test_reach_and_poles(ctx, offset, rows, corners, fast):
    """Facet centres within 61 um of the origin (the step without the direction's second order)
    and beyond, in rows around the forward bodge's limit (2.56 degrees from the axis) and away
    from it: 2e-5 of the largest amplitude of the FP64 drop-in (20 facets of radius 1)."""
    rng = np.random.default_rng(int(offset) + corners)
    geo = _polygon_mesh(rng, [corners] * 20)
    geo["verts"] = np.asfortranarray(geo["verts"] + offset / np.sqrt(3.0) * np.array([1.0, -1.0, 1.0]))
    beam, ext = outbeams(35, rng, 20), outbeams(18, rng, 20, prop=(np.sin(0.3), 0, -np.cos(0.3)))
    th = np.linspace(*rows, 23) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(35) * 360.0 / 35) * abt_b200.PI_REF / 180.0
    got = ctx.diff_main(beam, ext, geo, th, ph, LAM, is_fast_diff=fast, precision="fp32")
    ref = ctx.diff_main(beam, ext, geo, th, ph, LAM, is_fast_diff=fast, precision="fp64")
    for g, r in zip(got, ref):
        assert rel_err(g, r) <= 2e-5
        if fast:
            assert np.array_equal(g == 0, r == 0)


@pytest.mark.parametrize("nv", [[3] * 60, [3] * 55 + [7] * 5, [3, 4, 5] * 20])
@pytest.mark.parametrize("alike", [False, True])
def test_direction_order(ctx, nv, alike):
    """Field-of-view lists long enough (1e9 outbeam-bins) to be put in order of direction,
    records per face 1 or of a fan, and lists that look alike already and keep their order:
    the FP64 drop-in's masks, 2e-5 of its largest amplitude, the same bits again."""
    rng = np.random.default_rng(sum(nv) + alike)
    geo = _polygon_mesh(rng, nv)
    beam, ext = outbeams(12001, rng, 60), outbeams(8000, rng, 60, prop=(np.sin(0.3), 0, -np.cos(0.3)))
    if alike:
        beam["prop_out"] = beam["prop_out"][np.arange(len(beam)) // 100 * 100]
        beam["vk7"] = beam["vk7"][np.arange(len(beam)) // 100 * 100]
    th = np.linspace(4.0, 180.0, 259) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(200) * 360.0 / 200) * abt_b200.PI_REF / 180.0
    got = ctx.diff_main(beam, ext, geo, th, ph, LAM, is_fast_diff=True, precision="fp32")
    ref = ctx.diff_main(beam, ext, geo, th, ph, LAM, is_fast_diff=True, precision="fp64")
    again = ctx.diff_main(beam, ext, geo, th, ph, LAM, is_fast_diff=True, precision="fp32")
    for g, r, a in zip(got, ref, again):
        assert rel_err(g, r) <= 2e-5
        assert np.array_equal(g == 0, r == 0)
        assert np.array_equal(g, a)
