"""The 2-D boundary solver at the sizes where its block elimination changes:
lines of 5 k and 5 k +- 1 unknowns, the most tiles a thread block takes (100
unknowns) and one more (band elimination), lines along either axis, and the
fewest lines (two, none on one side of the middle)."""
import numpy as np
import pytest

from helpers import random_model
from mt3d import capi, models

pytestmark = pytest.mark.gpu


# (nx, ny, nz): for mode 2 the slices are ny x nz, for mode 1 nx x nz cells
@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 3), (3, 4, 12), (4, 3, 6), (5, 7, 7), (6, 9, 16), (3, 38, 36),
                                      (40, 3, 41), (3, 61, 62), (3, 101, 101), (101, 3, 102), (3, 130, 101),
                                      (3, 101, 130), (3, 102, 102), (104, 3, 103)])
def test_lines(cuda, nx, ny, nz):
    """E0 against the oracle's sparse direct solves: 1e-10 of its largest
    entry, as the other tests of the boundary solver."""
    from oracle import bc2d
    rng = np.random.default_rng(nx + 1000 * ny + 1000000 * nz)
    na = max(1, nz // 6)
    g = models.Grid(rng.uniform(200.0, 900.0, nx), rng.uniform(200.0, 900.0, ny), rng.uniform(40.0, 400.0, nz), na)
    m = random_model(g, seed=nz)
    omega = 2 * np.pi * 0.7
    s = capi.Solver(g)
    s.update_cond(m.m_earth, m.air_cond)
    s.update_freq(omega)
    sig = bc2d.sigma_cells(g, m.m_earth, m.air_cond)
    for imode in (1, 2):
        want = bc2d.compute_bc(g, sig, omega, imode)
        assert np.max(np.abs(s.compute_bc(imode) - want)) < 1e-10 * np.max(np.abs(want))
