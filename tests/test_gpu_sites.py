"""The data functional where sites share edges and lie at the rims of their
interpolation: sites on nodes, edges, cell centres and past the last centre,
several in one cell and coincident ones, more sites than a tile of the
scatter's search, against oracle/datafunc.py.  The bound is 1e-10: sums of some
80 terms to 1e-14, times a condition number of B that reaches 1e3 to 1e4 at the
worst of 700 sites of a random field."""
import numpy as np
import pytest

from helpers import random_model, relerr, small_grid
from mt3d import capi

pytestmark = pytest.mark.gpu


def _sites(g, n, seed):
    rng = np.random.default_rng(seed)
    xe, ye = np.concatenate([[0.0], np.cumsum(g.dx)]), np.concatenate([[0.0], np.cumsum(g.dy)])
    rims = [(xe[3], ye[4], 0.0), (xe[3], (ye[4] + ye[5]) / 2, 0.0), ((xe[3] + xe[4]) / 2, (ye[4] + ye[5]) / 2, 0.0),
            (xe[0] + 1.0, ye[0] + 1.0, 0.0), (xe[-1] - 1.0, ye[-1] - 1.0, 0.0), (xe[3], ye[4], g.dz[g.nzAir] / 2),
            (xe[3], ye[4], 0.0)]
    rnd = np.stack([rng.uniform(xe[1], xe[-2], n), rng.uniform(ye[1], ye[-2], n),
                    rng.uniform(0.0, g.dz[g.nzAir], n)], 1)
    return np.concatenate([np.array(rims), rnd])[:n]


@pytest.mark.parametrize("n", [1, 5, 7, 33, 700])
def test_shared_edges(cuda, n):
    from oracle import datafunc as df
    g = small_grid()
    m = random_model(g, seed=3)
    omega = 2 * np.pi * 0.2
    s = capi.Solver(g)
    s.update_cond(m.m_earth, m.air_cond)
    rng = np.random.default_rng(n)
    e1, e2 = (rng.standard_normal(s.nE) + 1j * rng.standard_normal(s.nE) for _ in range(2))
    sites = _sites(g, n, 5)
    d = rng.standard_normal((n, 2, 2)) + 1j * rng.standard_normal((n, 2, 2))
    origin = (0.0, 0.0, 0.0)
    c = df.coords(g.dx, g.dy, g.dz, g.nzAir, origin)
    assert relerr(s.impedance(omega, sites, e1, e2, origin), df.impedance(c, omega, sites, e1, e2)) < 1e-10
    g1, g2 = s.lmult_t(omega, sites, e1, e2, d, origin)
    o1, o2 = df.lmult_t(c, omega, sites, e1, e2, d)
    assert relerr(g1, o1) < 1e-10 and relerr(g2, o2) < 1e-10
    assert np.array_equal(g1 != 0, o1 != 0)
    r1, r2 = s.lmult_t(omega, sites, e1, e2, d, origin)
    assert np.array_equal(r1, g1) and np.array_equal(r2, g2)
