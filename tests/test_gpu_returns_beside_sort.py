"""Within one call of several USL steps the plastic returns of a step run beside the next
step's sort; called one step at a time they run at the step's end.  The same bits."""
import numpy as np
import pytest

from mpm_b200 import problems as P

pytestmark = pytest.mark.gpu

FIELDS = ("x", "u", "v", "stress", "strain", "F", "volume", "density", "cell", "svars")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("block", [(4, 3, 3), (16, 12, 10), (24, 20, 16)])  # both sorts; up to 61,440 points
def test_calls_of_many_steps_equal_single_steps(precision, block):
    runs = []
    for calls in ([1] * 25, [2, 23], [25]):
        prob = P.column_3d(shape=(2 * block[0], block[1], block[2] + 3), block=block, c=500.0, psi=5.0, dt=1e-5)
        s = P.build_solver(prob, precision=precision)
        st = s.read()
        st["v"] = st["x"] * np.array([2.0, 0.0, -2.0])
        s.load(st)
        for n in calls:
            s.step(n)
        runs.append(s.read())
    assert np.count_nonzero(runs[0]["svars"][:, 0]) > len(st["x"]) // 4, "the column was meant to yield"
    for r in runs[1:]:
        for f in FIELDS:
            assert np.array_equal(runs[0][f], r[f], equal_nan=True), f
