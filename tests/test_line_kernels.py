"""The derivative and adjoint line kernels at the block lengths where they
differ: 16 and 32 points (a line in registers), other lengths (run-time
sweeps in shared memory), lengths that lower the threads of a CTA (above 48
and 96 points) and the blocks a CTA takes side by side (200 points), line
counts that leave the last warp partly empty, and the adjoint on few lines
(groups of blocks, with a group left over) and on many (a walk of each
line).  Forward against the oracle at the
derivative bar; adjoint by <D x, y> = <x, D^T y> at 1e-13 of the sum of the
products' magnitudes (rounding of sums of 1e5 terms)."""
import numpy as np
import pytest

from css_b200 import problem
from css_b200.context import Simulation
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [((32, 32, 48), (2, 2, 3)), ((64, 64, 96), (2, 2, 3)), ((36, 52, 66), (2, 2, 3)),
          ((104, 36, 30), (2, 2, 3)), ((20, 200, 42), (2, 2, 3)), ((20, 400, 30), (2, 2, 3)),
          ((20, 30, 300), (2, 3, 3)), ((200, 20, 30), (2, 2, 3))]


def _sim(dims, decomp):
    p, prof, v0, dt, _ = problem.build(dims, decomp=decomp)
    return p, Simulation(p, prof), O.Oracle(p, prof), v0


@pytest.mark.parametrize("dims,decomp", SHAPES)
def test_derivatives_at_block_length(dims, decomp, gpu_available):
    p, sim, orc, v0 = _sim(dims, decomp)
    rng = np.random.default_rng(2)
    f = v0[4] + 1e-3 * rng.standard_normal(v0[4].shape)
    for direction in range(3):
        face = p.nth * p.nphi if direction == 0 else p.nphi * p.nr
        for order in (1, 2):
            for bdry in ((1, 4) if direction < 2 else (0,)):
                lo, hi = rng.standard_normal(face), rng.standard_normal(face)
                g = sim.deriv(direction, order, f, lo, hi, bdry)
                o = orc.deriv(direction, order, f, lo, hi, bdry)
                assert np.abs(g - o).max() <= 1e-12 * np.abs(o).max(), (direction, order, bdry)
    sim.close()


# adjoint alone: lines of 9 to 18 blocks (groups of 8 and a rest), and 40000 or
# more lines along r, theta and phi in turn, of 16 and 32 points and others
ADJOINT = SHAPES + [((90, 36, 40), (9, 2, 4)), ((36, 90, 40), (2, 9, 4)), ((36, 40, 180), (2, 4, 18)),
                    ((32, 192, 224), (2, 6, 7)), ((224, 32, 192), (7, 2, 6)), ((192, 224, 48), (6, 7, 3)),
                    ((64, 192, 224), (2, 6, 7)), ((224, 64, 192), (7, 2, 6)), ((192, 224, 96), (6, 7, 3)),
                    ((20, 200, 200), (2, 4, 5)), ((200, 24, 200), (4, 2, 5)), ((200, 200, 30), (4, 4, 3))]


@pytest.mark.parametrize("dims,decomp", ADJOINT)
def test_adjoint_at_block_length(dims, decomp, gpu_available):
    import torch
    from css_b200 import torch_ops  # noqa: F401
    p, sim, _, _ = _sim(dims, decomp)
    g = torch.Generator().manual_seed(1)
    x, y = (torch.randn(p.nr, p.nphi, p.nth, generator=g, dtype=torch.float64).cuda() for _ in range(2))
    for direction in range(3):
        for order in (1, 2):
            for bdry in (range(5) if direction < 2 else (0,)):
                dx = torch.ops.css.deriv(x, sim.h.value, direction, order, None, None, bdry)
                aty = torch.ops.css.deriv_adjoint(y, sim.h.value, direction, order, bdry)
                lhs, rhs = float((dx * y).sum()), float((x * aty).sum())
                scale = float((dx.abs() * y.abs()).sum())
                assert abs(lhs - rhs) <= 1e-13 * scale, (direction, order, bdry, lhs, rhs)
    sim.close()
