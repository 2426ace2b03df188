"""Tensor-product grids with graded axes: the box-cell kernels (axis tables, the
division-free locate, interpolation along the axes) against the CPU oracle, which
knows cells only by their nodes, and mixed against FP64.

Every other grid of the tests is uniform and cubic; here each axis has its own
spacings, the cell counts are odd and differ per axis, and the particles move
across cells.
"""
import numpy as np
import pytest

from mpm_b200 import problems as P
from oracle.oracle import build_oracle
from tests.parity import assert_parity, field_errors

pytestmark = pytest.mark.gpu


def graded(dim, scheme, update="flip"):
    """A free linear elastic block flying through a graded grid."""
    shape = (13, 9) if dim == 2 else (11, 7, 5)
    if dim == 2:
        prob = P.column_2d(shape=shape, block=(5, 4), E=5e5, scheme=scheme, dt=1e-4, velocity_update=update)
    else:
        prob = P.column_3d(shape=shape, block=(4, 3, 3), material="LinearElastic", E=5e5, scheme=scheme, dt=1e-4,
                           geostatic=False, velocity_update=update)
    rng = np.random.default_rng(5)
    axes = [np.concatenate([[0.0], np.cumsum(prob.dx * rng.uniform(0.6, 1.7, n))]) for n in shape]
    old = [np.arange(n + 1) * prob.dx for n in shape]
    stretch = lambda x: np.stack([np.interp(x[:, d], old[d], axes[d]) for d in range(dim)], axis=1)  # noqa: E731
    prob.coords = np.stack([axes[d][np.rint(prob.coords[:, d] / prob.dx).astype(int)] for d in range(dim)], axis=1)
    prob.particles = [(stretch(p + prob.dx), m) for p, m in prob.particles]
    prob.velocity_constraints = prob.friction_constraints = None
    prob.analysis["gravity"] = (0.0,) * dim
    return prob


def start_velocity(x):
    """Translation and a linear field (spin and stretch)."""
    dim = x.shape[1]
    grad = np.array([[0.5, 2.0, -1.0], [-1.5, -0.8, 0.7], [1.0, -0.6, 0.4]])[:dim, :dim]
    return np.array([0.9, 0.5, 0.4])[:dim] + x @ grad.T


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("scheme,update", [("usl", "flip"), ("usf", "pic"), ("musl", "flip"), ("usl", "apic")])
def test_graded_grid(dim, scheme, update):
    prob = graded(dim, scheme, update)
    g, m, o = (P.build_solver(prob), P.build_solver(prob, precision="mixed"), build_oracle(prob))
    st = g.read()
    st["v"] = v = start_velocity(st["x"])
    g.load(st)
    m.load(st)
    so = o.get()
    so["v"][:, :dim] = v
    o.set(so)
    start = st["cell"].copy()
    dx = min(np.diff(np.unique(prob.coords[:, d])).min() for d in range(dim))
    for n in (1, 100):
        for s in (g, m, o):
            s.step(n - (n > 1))
        a, b, c = g.read(), o.get(), m.read()
        assert_parity(a, b, label=f"{dim}D {scheme} {update}")
        # FP32 rounding of n steps.  Fields: at most a few 2^-24 of their scale a step.  Strain: a step adds dt
        # times velocity differences over a cell, of velocities off by up to 8 * 2^-24 each; stress: that times 3 K.
        # Later steps only where the velocities of nodes that a corner of the block hardly touches (FP32
        # momentum over a tiny mass) do not stay in the particles' velocities, as they do in FLIP and APIC.
        if n > 1 and scheme == "usl":
            continue
        errs = field_errors(c, a, ("x", "u", "v", "F", "volume", "density", "mass"))
        assert max(errs.values()) < n * 8 * 2.0 ** -24, errs
        strain = n * 1e-4 * 16 * 2.0 ** -24 * np.abs(a["v"]).max() / dx
        assert np.abs(c["strain"] - a["strain"]).max() < strain
        assert np.abs(c["stress"] - a["stress"]).max() < 5e5 / (1 - 2 * 0.3) * strain
    assert np.count_nonzero(a["cell"] != start) > len(start) // 4, "the block was meant to cross cells"
