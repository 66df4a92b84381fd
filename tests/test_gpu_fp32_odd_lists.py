"""Field-of-view sums of lists that end, or begin, in the middle of a record pair: the other half
of such a pair belongs to another list or to nothing, and must not show in the result.  The bits
are those of a fresh context whatever the context summed before, and a list's grid does not
depend on the list beside it."""
import numpy as np
import pytest

import abt_b200
from tests.helpers import outbeams
from tests.test_gpu_fp32_edges import LAM, _grid, _polygon_mesh

pytestmark = pytest.mark.gpu

TILT = (np.sin(0.3), 0, -np.cos(0.3))


def _lists(counts, rng, nf):
    return outbeams(counts[0], rng, nf), outbeams(counts[1], rng, nf, prop=TILT)


@pytest.mark.parametrize("plan", [None, (1, 1, 33), (1, 2, 64)])
@pytest.mark.parametrize("nv", [[3] * 20, [5] * 20, [3, 6] * 10])
@pytest.mark.parametrize("counts", [(1, 0), (2, 1), (40, 27), (65, 64)])
def test_earlier_calls_leave_nothing(nv, counts, plan):
    """After a longer call whose amplitudes exceed FP32, or whose records are others."""
    geo = _polygon_mesh(np.random.default_rng(3), nv)
    beam, ext = _lists(counts, np.random.default_rng(sum(counts)), len(nv))
    # the whole sphere in view, so that every warp visits the last pair
    beam["fov"] = abt_b200.PI_REF
    long = _lists((150, 150), np.random.default_rng(9), len(nv))
    huge = [ob.copy() for ob in long]
    for ob in huge:
        ob["ampl"] *= 1e300
    th, ph = _grid(21, 37)

    def run(ctx, a, b):
        return ctx.diff_main(a, b, geo, th, ph, LAM, is_fast_diff=True, precision="fp32")

    want = None
    for before in (None, long, huge):
        with abt_b200.Context(0) as ctx:
            if plan:
                ctx.set_plan(*plan)
            if before:
                run(ctx, *before)
            got = run(ctx, beam, ext)
        want = want or got
        for g, w in zip(got, want):
            assert np.isfinite(g).all() and np.array_equal(g, w)


@pytest.mark.parametrize("nv", [[3] * 20, [5] * 20])
@pytest.mark.parametrize("plan", [None, (1, 2, 64)])
def test_lists_of_one_pair_do_not_mix(ctx, nv, plan):
    """27 beam records: the last pair's other half is the first external-diffraction record."""
    geo = _polygon_mesh(np.random.default_rng(4), nv)
    beam, ext = _lists((27, 8), np.random.default_rng(5), len(nv))
    beam["fov"] = abt_b200.PI_REF
    other = ext.copy()
    other["ampl"] *= 1e300
    th, ph = _grid(21, 37)
    if plan:
        ctx.set_plan(*plan)
    want, _ = ctx.diff_main(beam, ext, geo, th, ph, LAM, is_fast_diff=True, precision="fp32")
    got, _ = ctx.diff_main(beam, other, geo, th, ph, LAM, is_fast_diff=True, precision="fp32")
    ctx.set_plan(-1)
    assert np.isfinite(got).all() and np.array_equal(got, want)
