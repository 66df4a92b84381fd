"""Large host copies: a context's first ones by the driver, the later ones through its pinned
slots (512 KB chunks, four in flight).  The same call gives the same bits either way, at sizes
around the chunks, with fresh and with reused arrays, and from two threads."""
import threading

import numpy as np
import pytest

import abt_b200
from tests.helpers import one_triangle, outbeams

pytestmark = pytest.mark.gpu


# 64 bytes a bin: one chunk less a bin, exactly one, one more, exactly four slots, five and a bit
@pytest.mark.parametrize("nt,nphi", [(8191, 1 * 3), (128, 64), (8193, 3), (256, 128), (300, 141)])
def test_copies_repeat(nt, nphi):
    th = (1.2 + 170.0 * np.arange(nt) / nt) * abt_b200.PI_REF / 180.0
    ph = np.arange(nphi) * 360.0 / nphi * abt_b200.PI_REF / 180.0
    rng = np.random.default_rng(nt)
    geo, ob = one_triangle(), outbeams(1, rng, 1)
    pin = abt_b200.params(geo_cross_sec=3.0)
    with abt_b200.Context(0) as ctx:
        first = ctx.diffraction(ob, geo, th, ph, 0.532)
        fin = ctx.finalise(first, first, th, ph, 0.532, pin)
        for _ in range(8):
            again = ctx.diffraction(ob, geo, th, ph, 0.532)
            assert np.array_equal(again, first)
            fin2 = ctx.finalise(again, again, th, ph, 0.532, pin)
            assert np.array_equal(fin2[0], fin[0]) and np.array_equal(fin2[1], fin[1])


def test_two_threads_share_a_context():
    th = (1.2 + 170.0 * np.arange(200) / 200) * abt_b200.PI_REF / 180.0
    ph = np.arange(100) * 3.6 * abt_b200.PI_REF / 180.0
    geo = one_triangle()
    obs = [outbeams(1, np.random.default_rng(s), 1) for s in (1, 2)]
    with abt_b200.Context(0) as ctx:
        want = [ctx.diffraction(o, geo, th, ph, 0.532) for o in obs]
        bad = []

        def work(k):
            for _ in range(20):
                if not np.array_equal(ctx.diffraction(obs[k], geo, th, ph, 0.532), want[k]):
                    bad.append(k)

        threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad
