"""Steps under a gravity ramp, whose arguments change from step to step: within one call they are
launched without a graph, the plastic returns beside the next step's sort.  The same bits as single
steps, through the end of the ramp, and no dearer than those (a graph captured for
every step took five times as long as a step)."""
import time

import numpy as np
import pytest

from mpm_b200 import problems as P

pytestmark = pytest.mark.gpu

FIELDS = ("x", "u", "v", "stress", "strain", "F", "volume", "density", "cell", "svars")


def column(ramp, block=(6, 5, 5), **kw):
    prob = P.column_3d(shape=(2 * block[0], block[1], block[2] + 3), block=block, c=500.0, psi=5.0, dt=1e-5, **kw)
    prob.analysis["gravity_ramping_time"] = ramp
    return prob


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("scheme", ["usl", "usf", "musl"])
def test_ramp_within_a_call_equals_single_steps(precision, scheme):
    runs = []
    for calls in ([1] * 70, [70], [2, 30, 38]):
        s = P.build_solver(column(4e-4, scheme=scheme), precision=precision)  # 40 steps of ramp
        st = s.read()
        st["v"] = st["x"] * np.array([2.0, 0.0, -2.0])
        s.load(st)
        for n in calls:
            s.step(n)
        runs.append(s.read())
    assert np.count_nonzero(runs[0]["svars"][:, 0]) > 100
    for r in runs[1:]:
        for f in FIELDS:
            assert np.array_equal(runs[0][f], r[f], equal_nan=True), f


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_ramp_is_no_dearer_than_single_steps(precision):
    s = P.build_solver(column(1.0), precision=precision)
    s.step(20)
    call, single = [], []
    for _ in range(5):
        t = time.perf_counter()
        s.step(100)
        call.append(time.perf_counter() - t)
        t = time.perf_counter()
        for _ in range(100):
            s.step(1)
        single.append(time.perf_counter() - t)
    assert min(call) < 2 * min(single), (call, single)
