"""The slope limiter beside a non-finite cell.  The limited difference is q
times a ratio, so a NaN difference gives NaN, and an infinite one of the
opposite sign, whose ratio is zero, NaN too: a face next to such a cell is
not finite.  Which cells of the diffusion tendency are finite is compared
with the oracle's formula.  An infinite difference of the same sign is
limited to the other difference, where the oracle's rounded ratio makes it
inf * 0; so the NaN cell is put into a random state, the infinite one into a
field that grows away from it in every direction, where every neighbouring
difference has the opposite sign."""
import numpy as np
import pytest

from css_b200 import problem
from oracle import oracle as O


def state(kind, cell):
    p, prof, v0, _, _ = problem.build((32, 32, 48), decomp=(2, 2, 3))
    rng = np.random.default_rng(1)
    v = v0.copy()
    v[1:4] = 1e-3 * rng.standard_normal(v[1:4].shape)
    v[4] += 10 * rng.standard_normal(v[4].shape)
    iv, ir, ip, it = cell
    if kind == "bowl":
        r, ph, t = np.meshgrid(np.arange(p.nr) - ir, np.arange(p.nphi) - ip, np.arange(p.nth) - it, indexing="ij")
        bowl = np.abs(r) + np.minimum(np.abs(ph), p.nphi - np.abs(ph)) + np.abs(t)
        v[iv] = (1e-3 if iv < 4 else 1e5) * bowl
    return p, prof, v


@pytest.mark.gpu
@pytest.mark.parametrize("bad,kind", [(np.nan, "random"), (-np.nan, "random"), (np.nan, "bowl"), (np.inf, "bowl")])
@pytest.mark.parametrize("cell", [(4, 10, 20, 9), (2, 7, 5, 25), (4, 16, 16, 16)])
def test_faces_beside_a_non_finite_cell(bad, kind, cell, gpu_available):
    from css_b200.context import Simulation
    p, prof, v = state(kind, cell)
    v[cell] = bad
    sim = Simulation(p, prof)
    got = sim.diffusion(v)
    sim.close()
    want = O.Oracle(p, prof).diffusion(v)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    if np.isnan(bad):
        assert np.array_equal(np.isnan(got), np.isnan(want))
