"""A submission that arrives while the server's worker is between its admission pass and its idle wait
has to be picked up at once: the wait tests the queue before it sleeps.

48 small slices are submitted together and waited for, over and over, so that the worker goes idle and
is woken in every pass. A pass is a few milliseconds of work; a missed wake-up costs its full 50 ms."""
import time

import numpy as np
import pytest

import gct_b200 as g
from cases import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["parallel_1d", "fan_line"])
def test_submissions_wake_an_idle_server(kind):
    case = make_case(kind, nv=90, nc=96, n=64)
    proj = np.random.default_rng(1).random((90, 1, 96), dtype=np.float32)
    outs = [np.empty(case.vg.shape, np.float32) for _ in range(48)]
    times = []
    with g.FdkPlan(case.cg, case.vg) as plan, g.FdkServer(256 << 20) as srv:
        for _ in range(12):
            t = time.perf_counter()
            for ticket in [srv.submit(plan, proj, o) for o in outs]:
                srv.wait(ticket)
            times.append(time.perf_counter() - t)
        assert srv.stats()["completed"] == 12 * len(outs)
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])
    # a shared machine may delay single passes: the third quickest of the last ten
    assert sorted(times[2:])[2] < 0.025, times
