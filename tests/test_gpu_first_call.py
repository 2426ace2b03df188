"""The first call of a process: three 2D mixed MohrCoulomb solvers of one slope's size whose first
call has many steps (the plastic returns beside the next step's sort, the captured step),
then calls and reads in turn.  Every call succeeds, no solver falls back from the graph
(mpm_gpu_last_error stays empty), and the states are those of single steps, bit for bit."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys
import numpy as np
from mpm_b200 import ensemble as E
from mpm_b200 import problems as P

def solver(k):
    prob, _ = E.ensemble_problem([E.SlopeRun(height=48, width=48, phi=32.0, cohesion=3000.0, seed=100 + k)])
    return P.build_solver(prob, precision="mixed")

many, calls = [solver(k) for k in range(3)], 40
outs = [s.state_buffers(pinned=True) for s in many]
for c in range(calls):
    for s, o in zip(many, outs):
        s.step(50)
        state = s.read(out=o)
        assert not s.L.mpm_gpu_last_error(s.h), s.L.mpm_gpu_last_error(s.h)
plastic = 0
for k, o in enumerate(outs):
    one = solver(k)
    for n in range(50 * calls):
        one.step(1)
    ref = one.read()
    plastic += np.count_nonzero(ref["svars"][:, 0])
    for f in ("x", "u", "v", "stress", "strain", "F", "volume", "density", "cell", "svars"):
        assert np.array_equal(o[f][:, :2] if f in "xuv" else o[f], ref[f]), (k, f)
print("points", len(state["x"]), "plastic", plastic)
"""


def test_first_call_of_many_steps_in_a_fresh_process():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    _, points, _, plastic = r.stdout.split()
    assert 13000 < int(points) <= 16384 and int(plastic) > 0  # the one-cluster sort; some points return
