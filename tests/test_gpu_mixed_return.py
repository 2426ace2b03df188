"""The mixed path's plastic return (the reciprocal form of the update, on the device) from stresses at the
triaxial corners, near them and in between, against the FP64 update of the same points."""
import numpy as np
import pytest

from mpm_b200 import problems as P
from mpm_b200.solver import Solver, material_stress_batch

pytestmark = pytest.mark.gpu


def stresses(dim, corner, n, rng):
    s = np.zeros((n, 6))
    k = 4 if dim == 2 else 6
    if corner == "between":
        s[:, :k] = rng.normal(0.0, 4000.0, (n, k))
    else:
        s[:, 0 if corner == "compression" else 1] = -9000.0 * rng.uniform(0.5, 2.0, n)
        if corner == "extension":
            s[:, 2] = s[:, 1]
        s[n // 4:, 3] = 10.0 ** rng.uniform(-2.0, 3.0, n - n // 4)  # the distance from the corner
    s[:, :3] += rng.choice([-2000.0, 500.0], n)[:, None]  # shear and tensile returns
    return s.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("corner", ["compression", "extension", "between"])
def test_returned_stress(dim, corner):
    rng = np.random.default_rng(4)
    shape, n = ((40, 25), 800) if dim == 2 else ((20, 10, 8), 1200)
    dx, E, c, dt = 0.1, 1e7, 1500.0, 1e-9
    props = P.mohr_coulomb(E, 0.3, 1800.0, 32.0, c, 5.0, tension_cutoff=300.0)
    coords, cells = P.structured_mesh(dim, shape, dx)
    s = Solver(dim, scheme="usl", dt=dt, precision="mixed")
    s.set_mesh(coords, cells)
    s.add_material(0, "MohrCoulomb%dD" % dim, props)
    ijk = rng.integers(0, shape, (n, dim))
    s.add_particles((ijk + rng.uniform(0.1, 0.9, (n, dim))) * dx, 0)
    s.initialise()
    st = s.read()
    sig = st["stress"] = stresses(dim, corner, n, rng)
    s.load(st)
    s.step(1)
    got = s.read()
    sv0 = st["svars"].copy()
    sv0[:, 1:5] = sv0[:, 1:5].astype(np.float32)  # the state as the mixed path holds it
    ref, sv = material_stress_batch(dim, "MohrCoulomb%dD" % dim, props, sig, np.zeros((n, 6)), 1800.0, state=sv0)
    assert np.count_nonzero(sv[:, 0] == 1) > n // 8
    # Rounding to FP32 (2^-24 of the stress) and the step's strain, from accelerations of at most |sigma| / (rho
    # dx) over light nodes (down to 1e-2 of a full one): dt^2 |sigma| / (rho dx^2 1e-2) times 4 E
    scale = np.abs(sig).max()
    bound = scale * (2 * 2.0 ** -24 + dt * dt / (1800.0 * dx * dx * 1e-2) * 4 * E)
    assert np.array_equal(got["svars"][:, 0], sv[:, 0])
    assert np.abs(got["stress"] - ref).max() < bound
    plastic = sv[:, 0] != 0
    assert np.abs(got["svars"][plastic, 5:7] - sv[plastic, 5:7]).max() < 4 * bound
    # the angle: the returned stress's FP32 rounding is not in it, FP64 rounding at a corner is (its square root)
    assert np.abs(got["svars"][plastic, 7] - sv[plastic, 7]).max() < 2.0 ** -22
