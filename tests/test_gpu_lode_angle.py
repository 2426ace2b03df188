"""The Lode angle and the other invariants of the MohrCoulomb update as the FP64 path takes them on
the device (acos of cos 3 theta): on the triaxial corners (compression, extension), at
growing distances from them and in between, against 80-bit arithmetic."""
import numpy as np
import pytest

from mpm_b200 import problems as P
from mpm_b200.solver import material_stress_batch

pytestmark = pytest.mark.gpu


def invariants(s):
    s = s.astype(np.longdouble)
    p = s[:, :3].mean(axis=1)
    d = s[:, :3] - p[:, None]
    j2 = (d ** 2).sum(axis=1) / 2 + (s[:, 3:] ** 2).sum(axis=1)
    j3 = (d[:, 0] * d[:, 1] * d[:, 2] - d[:, 2] * s[:, 3] ** 2 + 2 * s[:, 3] * s[:, 4] * s[:, 5]
          - d[:, 0] * s[:, 4] ** 2 - d[:, 1] * s[:, 5] ** 2)
    r = np.clip(1.5 * np.sqrt(np.longdouble(3)) * j3 / j2 ** np.longdouble(1.5), -1, 1)
    return p, j2, r


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("corner", ["compression", "extension", "between"])
def test_lode_angle(dim, corner):
    rng = np.random.default_rng(2)
    n = 400
    s = np.zeros((n, 6))
    if corner == "between":
        s[:, :4 if dim == 2 else 6] = rng.normal(0.0, 1000.0, (n, 4 if dim == 2 else 6))
    else:
        s[:, 0 if corner == "compression" else 1] = -1000.0 * rng.uniform(0.5, 2.0, n)
        if corner == "extension":
            s[:, 2] = s[:, 1]
        s[1:, 3] = 10.0 ** rng.uniform(-9.0, 2.0, n - 1)  # the distance from the corner
    s[:, :3] -= 5000.0
    props = P.mohr_coulomb(1e7, 0.3, 1800.0, 30.0, 1e6, 0.0, tension_cutoff=1e6)  # elastic throughout
    out, st = material_stress_batch(dim, f"MohrCoulomb{dim}D", props, s, np.zeros((n, 6)), 1800.0,
                                    state=np.tile([0, np.pi / 6, 0, 1e6, 1e6, 0, 0, 0, 0], (n, 1)))
    assert np.array_equal(out, s) and np.all(st[:, 0] == 0)
    p, j2, r = invariants(s)
    theta = np.arccos(r) / 3
    # cos 3 theta carries the rounding of j2 and j3, whose terms come from stresses around |s| = 7000: relative
    # error 16 * 2^-53 * |s| / sqrt(j2) (and it is rounded itself), amplified by d theta / d r
    e = 16 * 2.0 ** -53 * (1 + 7000.0 / np.sqrt(j2.astype(float)))
    lo, hi = np.clip(r - 3 * e, -1, 1), np.clip(r + 3 * e, -1, 1)
    bound = np.maximum(np.abs(np.arccos(lo) / 3 - theta), np.abs(np.arccos(hi) / 3 - theta)).astype(float) + 1e-15
    assert np.all(np.abs(st[:, 7] - theta.astype(float)) <= bound)
    assert np.allclose(st[:, 6], np.sqrt(2 * j2.astype(float)), rtol=1e-12)
    assert np.allclose(st[:, 5], (np.sqrt(3) * p).astype(float), rtol=1e-14)
