"""P2G cell tiles at the sizes where they can go wrong: tiles with fewer, exactly and
more particles than are staged at once (T and 1.25 T rows of T threads), cells from
empty to 60 particles, ids scattered over the cells.  Mixed against FP64, and the
same bits from every tile size."""
import numpy as np
import pytest

from mpm_b200 import problems as P
from tests.parity import field_errors

pytestmark = pytest.mark.gpu


def ragged(dim, per_cell, scheme, seed=3):
    """A linear elastic block whose filled cells hold per_cell(rng) particles each, in shuffled id order."""
    rng = np.random.default_rng(seed)
    shape, block = ((23, 11), (17, 9)) if dim == 2 else ((9, 7, 6), (7, 5, 5))
    prob = (P.column_2d(shape=shape, block=block, scheme=scheme) if dim == 2 else
            P.column_3d(shape=shape, block=block, scheme=scheme, material="LinearElastic", E=1e6, dt=1e-5,
                        geostatic=False))
    cells = np.stack(np.meshgrid(*[np.arange(b) for b in block], indexing="ij"), axis=-1).reshape(-1, dim)
    pts = np.concatenate([(c + rng.uniform(0.02, 0.98, (per_cell(rng), dim))) * prob.dx for c in cells])
    prob.particles = [(rng.permutation(pts), prob.particles[0][1])]
    return prob


PER_CELL = {"one": lambda r: 1, "usual": lambda r: int(r.integers(6, 11)), "edge": lambda r: int(r.integers(8, 12)),
            "full": lambda r: int(r.integers(9, 14)), "ragged": lambda r: int(r.choice([0, 1, 3, 16, 17, 60]))}


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("scheme", ["usl", "usf"])
@pytest.mark.parametrize("cells", sorted(PER_CELL))
def test_tile_occupancy(dim, scheme, cells):
    prob = ragged(dim, PER_CELL[cells], scheme)
    f = P.build_solver(prob)
    f.step(20)
    ref, bits = f.read(), None
    for tile in (128, 256):
        s = P.build_solver(prob, precision="mixed")
        s.set_launch_shape(p2g_tile=tile)
        s.step(20)
        st = s.read()
        # FP32 rounding of 20 steps: each adds at most a few 2^-24 of the field's scale
        errs = field_errors(st, ref)
        assert max(errs.values()) < 20 * 8 * 2.0 ** -24, (tile, errs)
        assert np.array_equal(st["cell"], ref["cell"])
        if bits is not None:
            assert all(np.array_equal(st[k], bits[k]) for k in ("x", "v", "stress", "strain")), tile
        bits = st
