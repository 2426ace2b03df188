"""The cell sort on both sides of its size rule: the same run in a mesh whose cell count
selects the one-cluster sort and in a taller one that selects the passes, where the
added cells stay empty, must agree bit for bit (ids and cells keep their order)."""
import numpy as np
import pytest

from mpm_b200 import problems as P

pytestmark = pytest.mark.gpu

FIELDS = ("x", "u", "v", "stress", "strain", "F", "volume", "density", "cell", "svars")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("block", [(3, 3), (31, 33), (64, 63), (64, 64), (64, 65)])
def test_cluster_sort_equals_the_passes(precision, block):
    states = []
    for height in (80, 1100):  # 5,600 and 77,000 cells; 16,384 particles at 64 x 64
        prob = P.column_2d(shape=(70, height), block=block, scheme="usl", material="MohrCoulomb", dt=1e-4)
        prob.materials = [(0, "MohrCoulomb2D", P.mohr_coulomb(1e6, 0.3, 1800.0, 30.0, 1000.0, 5.0))]
        s = P.build_solver(prob, precision=precision)
        st = s.read()
        st["v"] = 5.0 * (st["x"] - st["x"].mean(axis=0)) * np.array([1.0, -0.5])
        s.load(st)
        s.step(60)
        states.append(s.read())
    a, b = states
    assert np.count_nonzero(a["x"] != st["x"]) > 0
    for f in FIELDS:
        assert np.array_equal(a[f], b[f], equal_nan=True), f


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("scheme", ["usl", "usf", "musl"])
def test_both_launches_of_p2g(precision, scheme):
    """P2G waits for the sort on the device up to 4,096 tiles and is launched after it above:
    the same run in meshes of 88, 4,095 and 4,098 tiles, the added ones empty."""
    states = []
    for height in (80, 3744, 3746):
        prob = P.column_2d(shape=(70, height), block=(31, 33), scheme=scheme, dt=1e-4)
        s = P.build_solver(prob, precision=precision)
        st = s.read()
        st["v"] = 5.0 * (st["x"] - st["x"].mean(axis=0)) * np.array([1.0, -0.5])
        s.load(st)
        s.step(1)
        s.step(39)
        states.append(s.read())
    for b in states[1:]:
        for f in FIELDS:
            assert np.array_equal(states[0][f], b[f], equal_nan=True), f


@pytest.mark.parametrize("height", [234, 235])  # 16,380 and 16,450 cells: the rule's line is 16,384
def test_both_sides_of_the_cell_line(height):
    prob = P.column_2d(shape=(70, height), block=(64, 64), scheme="usl", dt=1e-4)
    launches = []
    s = P.build_solver(prob, precision="mixed")
    for n in (1, 1):
        before = s.launch_count
        s.step(n)
        launches.append(s.launch_count - before)
    # sort, P2G, nodes, G2P
    assert launches == [4 if height == 234 else 8] * 2
    o = P.build_solver(prob)
    o.step(2)
    assert np.array_equal(s.read()["cell"], o.read()["cell"])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("scheme", ["usl", "usf", "musl"])
def test_particles_leaving_a_grid_are_found_or_removed(precision, scheme):
    """Moves of several cells a step (the search beyond the neighbours) and out of the mesh."""
    prob = P.column_2d(shape=(40, 30), block=(8, 8), E=1e3, scheme=scheme, dt=1e-3)
    prob.velocity_constraints = None
    prob.analysis["gravity"] = (0.0, 0.0)
    s = P.build_solver(prob, precision=precision, locate_particles=False)
    st = s.read()
    st["v"] = np.tile([45.0, 30.0], (len(st["x"]), 1))  # 4.5 and 3 cells a step
    s.load(st)
    s.step(2)
    a = s.read()
    ij = np.floor(a["x"] / prob.dx).astype(int)
    assert np.array_equal(a["cell"], ij[:, 0] + 40 * ij[:, 1])
    s.step(9)
    assert np.all(s.read()["cell"] == -1)
