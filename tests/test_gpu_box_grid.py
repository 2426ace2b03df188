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


def perturbed(st, prob, axes, seed):
    """The state moved by what one mixed step rounds: local coordinates and velocities to FP32 (2^-24 of a cell's
    half length, and of the largest velocity)."""
    rng, dim = np.random.default_rng(seed), prob.dim
    out = {k: v.copy() for k, v in st.items()}
    for d in range(dim):
        length = np.diff(axes[d])[np.searchsorted(axes[d], st["x"][:, d], side="right") - 1]
        out["x"][:, d] += rng.uniform(-1, 1, len(length)) * 2.0 ** -24 * length / 2
    out["v"][:, :dim] += rng.uniform(-1, 1, (len(st["x"]), dim)) * 2.0 ** -24 * np.abs(st["v"]).max()
    return out


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("scheme,update", [("usl", "flip"), ("usf", "pic"), ("musl", "flip"), ("usl", "apic"),
                                           ("usl", "asflip"), ("usl", "tpic")])
def test_graded_grid(dim, scheme, update):
    prob = graded(dim, scheme, update)
    axes = [np.unique(prob.coords[:, d]) for d in range(dim)]
    g, m, o = (P.build_solver(prob), P.build_solver(prob, precision="mixed"), build_oracle(prob))
    near = [P.build_solver(prob) for _ in range(4)]  # FP64 runs of inputs one mixed rounding away
    st = g.read()
    st["v"] = start_velocity(st["x"])
    g.load(st)
    m.load(st)
    for k, s in enumerate(near):
        s.load(perturbed(st, prob, axes, k))
    so = o.get()
    so["v"][:, :dim] = st["v"]
    o.set(so)
    start = st["cell"].copy()
    dx = min(np.diff(a).min() for a in axes)
    fields = ("x", "u", "v", "F", "volume", "density", "mass", "stress", "strain")
    # TPIC in 2D for 60 steps only: at 70 a corner that just entered a cell strains its point by 0.8, at 80 by 2.6,
    # and 1 / (1 + dV) carries the oracle's own rounding beyond 1e-10 of the density
    for n in (1, 60 if update == "tpic" else 100):
        for s in (g, m, o, *near):
            s.step(n - (n > 1))
        a, b, c = g.read(), o.get(), m.read()
        assert_parity(a, b, label=f"{dim}D {scheme} {update}")
        errs = field_errors(c, a, fields)
        if n == 1:
            # FP32 rounding of one step.  Fields: at most a few 2^-24 of their scale.  Strain: dt times velocity
            # differences over a cell, of velocities off by up to 8 * 2^-24 each; stress: that times 3 K.
            assert max(errs[f] for f in fields[:7]) < 8 * 2.0 ** -24, errs
            strain = 1e-4 * 16 * 2.0 ** -24 * np.abs(a["v"]).max() / dx
            assert np.abs(c["strain"] - a["strain"]).max() < strain
            assert np.abs(c["stress"] - a["stress"]).max() < 5e5 / (1 - 2 * 0.3) * strain
            continue
        # Each of n steps rounds as far as the perturbed runs start away, and what is rounded grows from there as
        # theirs has grown (most of it at nodes that a corner of the block hardly touches): n times the
        # largest of them, on top of n roundings of the result itself.
        floor = [field_errors(s.read(), a, fields) for s in near]
        for f in fields:
            assert errs[f] < n * (max(e[f] for e in floor) + 2.0 ** -24), (f, errs[f], [e[f] for e in floor])
        # the same cells, but for particles as close to a face as the runs are to each other
        apart = np.abs(c["x"] - a["x"]).max() + 1e-15
        face = np.min([np.abs(a["x"][:, d, None] - axes[d][None]).min(axis=1) for d in range(dim)], axis=0)
        assert np.array_equal(c["cell"][face > apart], a["cell"][face > apart])
    assert np.count_nonzero(a["cell"] != start) > len(start) // 4, "the block was meant to cross cells"
