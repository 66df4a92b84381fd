"""Large host copies where their pinned slots or their helpers cannot be had."""
import os
import subprocess
import sys

import numpy as np
import pytest

import abt_b200
from abt_b200 import _lib
from tests.conftest import ROOT
from tests.helpers import one_triangle, outbeams

pytestmark = pytest.mark.gpu

LAM = 0.532


def _inputs():
    th = (1.2 + 170.0 * np.arange(200) / 200) * abt_b200.PI_REF / 180.0
    ph = np.arange(150) * 2.4 * abt_b200.PI_REF / 180.0
    return one_triangle(), outbeams(1, np.random.default_rng(2), 1), th, ph


def test_no_pinned_memory():
    """A failing allocation of the slots (injected) leaves the copies to the driver, for the
    context's lifetime: the same results, and no further attempt."""
    geo, ob, th, ph = _inputs()
    L = _lib.lib()
    with abt_b200.Context(0) as ctx:
        want = ctx.diffraction(ob, geo, th, ph, LAM)
        assert L.pbt_test_fail_next_host_alloc(1) == 0
        try:
            for _ in range(30):
                assert np.array_equal(ctx.diffraction(ob, geo, th, ph, LAM), want)
            assert L.pbt_test_fail_next_host_alloc(5) == 0  # the attempt was made
            pin = abt_b200.params(geo_cross_sec=3.0)
            for _ in range(30):
                mu = ctx.finalise(want, want, th, ph, LAM, pin)[0]
                assert np.isfinite(mu).all()
        finally:
            left = L.pbt_test_fail_next_host_alloc(0)
        assert left == 5


_BOUND = r"""
import os, sys
sys.path.insert(0, %r)
if sys.argv[1] == "one":
    os.sched_setaffinity(0, {sorted(os.sched_getaffinity(0))[0]})
import numpy as np
import abt_b200
from tests.test_gpu_host_copy_limits import LAM, _inputs
geo, ob, th, ph = _inputs()
with abt_b200.Context(0) as ctx:
    want = ctx.diffraction(ob, geo, th, ph, LAM)  # 1.9 MB
    before = len(os.listdir("/proc/self/task"))
    for _ in range(30):
        assert np.array_equal(ctx.diffraction(ob, geo, th, ph, LAM), want)
    print("THREADS", len(os.listdir("/proc/self/task")) - before)
"""


@pytest.mark.parametrize("how,env,most", [("one", {}, 0), ("all", {"OMP_NUM_THREADS": "1"}, 0),
                                          ("all", {"OMP_NUM_THREADS": "3"}, 2), ("all", {}, 7)])
def test_threads_that_the_process_may_use(how, env, most):
    """The copies start no more threads than the processors the process is bound to, and
    OpenMP's limit, allow."""
    e = {k: v for k, v in os.environ.items() if not k.startswith("OMP_")}
    r = subprocess.run([sys.executable, "-c", _BOUND % ROOT, how], env=dict(e, **env), capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert 0 <= int(r.stdout.split("THREADS")[1]) <= most
