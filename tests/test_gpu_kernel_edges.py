"""Kernel forms against each other at the sizes where tiles, chunks and copies end.

Tolerances: FP32 forms of one update (different summation order and FMA contraction), two steps
from a random state: max |diff| <= 2e-5 x max |ref| per component, as against the oracle. FP64 forms:
equal to double rounding, so their read-back floats differ by one unit in the last place at most:
1.2e-7 x max |ref|. Forms that only cut the work differently: bitwise.
"""
import numpy as np
import pytest

from cgfd_b200 import Simulation
from helpers import small_problem, random_wavefield

pytestmark = pytest.mark.gpu

# smaller than a tile, one point over a tile in x / y, several tiles with remainders
GRIDS = [(9, 8, 13), (33, 37, 21), (70, 41, 34)]


def _two_steps(p, shots=None, variant=None, setup=None):
    sim = Simulation(p, shots)
    if variant is not None:
        sim.set_bulk_variant(variant)
    if setup:
        setup(sim)
    for s in range(sim.nshot):
        sim.set_wavefield(random_wavefield(p, seed=3 + s), s)
    sim.run(2)
    return [sim.wavefield(s) for s in range(sim.nshot)]


@pytest.mark.parametrize("medium", ["iso", "vti", "aniso", "ac"])
@pytest.mark.parametrize("grid", GRIDS + [(101, 64, 48)])
def test_default_chunk_changes_no_result(medium, grid):
    p = small_problem(medium, *grid, nsteps=4, npml=3, nsrc=1)
    (a,), (b,) = _two_steps(p), _two_steps(p, setup=lambda s: s.set_zchunk(12))
    np.testing.assert_array_equal(a, b)


# a field below the staged copy's least size, one of a single chunk, one of a chunk and a remainder
@pytest.mark.parametrize("grid", [(40, 36, 30), (120, 100, 70), (300, 280, 210)])
def test_wavefield_readback_equals_box(grid):
    p = small_problem("iso", *grid, nsteps=2, npml=0, nsrc=0, sta_grid=None)
    sim = Simulation(p)
    rng = np.random.default_rng(1)
    w = np.zeros((9,) + tuple(n + 6 for n in grid[::-1]), np.float32)
    w[:, 3:-3, 3:-3, 3:-3] = rng.standard_normal((9,) + grid[::-1], dtype=np.float32)
    sim.set_wavefield(w)
    out = sim.wavefield()
    np.testing.assert_array_equal(out, w)
    np.testing.assert_array_equal(out[:, 3:-3, 3:-3, 3:-3], sim.wavefield_box((0, 0, 0), grid))
