"""The FP64 sum without room for its partial grids: fewer runs, at last one a list."""
import numpy as np
import pytest

import abt_b200
from abt_b200 import _lib
from abt_b200._lib import PBT_ENOMEM, PbtError
from tests.helpers import outbeams, rel_err

pytestmark = pytest.mark.gpu

LAM = 0.532


@pytest.mark.parametrize("failures", [0, 1, 2, 1000])
def test_no_room_for_partial_grids(failures):
    """Every buffer but the partial grids' is large enough from the calls before, so the injected
    failures meet them alone.  The sum's order changes with its runs: 1e-13 of the largest
    amplitude (about 60 roundings of 1.1e-16 in a list of 64 facets)."""
    rng = np.random.default_rng(1)
    ang = 2 * np.pi * np.arange(60) / 60
    ring = np.stack([2.0 + np.cos(ang), np.sin(ang) - 1.0, 0.3 * np.ones(60)], 1)
    tri = rng.normal(size=(20, 3, 3)) + 3.0 * rng.normal(size=(20, 1, 3))
    geo = abt_b200.make_geometry(np.concatenate([ring, tri.reshape(-1, 3)]),
                                 [list(range(1, 61))] + [[61 + 3 * i, 62 + 3 * i, 63 + 3 * i] for i in range(20)])
    th = np.linspace(4.0, 176.0, 41) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(30) * 12.0) * abt_b200.PI_REF / 180.0
    beam, ext, ring_ob = outbeams(64, rng, 20), outbeams(48, rng, 20, prop=(0, 0, -1)), outbeams(8, rng, 1)
    beam["fi"] += 1
    ext["fi"] += 1
    L = _lib.lib()

    with abt_b200.Context(0) as ctx:
        want = ctx.diff_main(beam, ext, geo, th, ph, LAM, precision="fp64")
    with abt_b200.Context(0) as ctx:
        # facet records (128 B an outbeam here, 384 B each below); edges, and grids of results
        ctx.diff_main(np.repeat(beam, 4), np.repeat(ext, 4), geo, th, ph, LAM, precision="fp32")
        ctx.diff_main(ring_ob, ring_ob[:0], geo, th, ph, LAM, precision="fp64")
        assert L.pbt_test_fail_next_alloc(failures) == 0
        try:
            got = ctx.diff_main(beam, ext, geo, th, ph, LAM, precision="fp64")
        finally:
            left = L.pbt_test_fail_next_alloc(0)
        assert left < failures or not failures
        for g, w in zip(got, want):
            assert rel_err(g, w) <= 1e-13
            assert failures or np.array_equal(g, w)
        # elsewhere a failing allocation is an error as before
        with pytest.raises(PbtError) as e:
            L.pbt_test_fail_next_alloc(1)
            try:
                ctx.diff_main(beam, ext, geo, np.concatenate([th, th + 1e-3]), ph, LAM, precision="fp64")
            finally:
                L.pbt_test_fail_next_alloc(0)
        assert e.value.status == PBT_ENOMEM
