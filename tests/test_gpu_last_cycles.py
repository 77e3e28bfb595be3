"""An FP32 cycle ends early (its own residual at 1e-7 of its start) only where
enough cycles are left to reach the tolerance.  A call that allows one or two
cycles has each of them run to the tolerance it was given: the residual history
holds it, as the returned field cannot (an FP32 cycle lowers the true residual by
some 1e-5 to 1e-7 at most)."""
import numpy as np
import pytest

from helpers import random_model, small_grid
from mt3d import bc as mbc
from mt3d import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cycles", [1, 2, 3])
@pytest.mark.parametrize("poly", [0.0, 0.9])
def test_few_cycles_run_to_the_tolerance(cuda, cycles, poly):
    g = small_grid()
    m = random_model(g, seed=3)
    omega = 2 * np.pi * 0.5
    tol = 1e-10
    s = capi.Solver(g)
    s.set_formulation(capi.FORM_CCGD)
    s.set_restart(0)
    s.set_poly(poly)
    s.update_cond(m.m_earth, m.air_cond)
    s.update_freq(omega)
    s.set_control(IterPerDivCor=1000, MaxDivCor=cycles, tolEMfwd=tol, precision=capi.PREC_MIXED)
    e, rc = s.fwdsolve(bc=mbc.boundary_1d(m, omega, 1))
    d = s.diagnostics()
    # the first cycle starts from a zero field, so its tolerance is the call's
    assert d["EMrelErr"].min() < tol
    assert (rc == 0) == (d["final_relres"] <= tol)
    assert d["nDivCor"] <= cycles


def test_many_cycles_end_early(cuda):
    """With cycles to spare the first one stops at 1e-7 of its start and the
    solve still reaches 1e-12."""
    g = small_grid()
    m = random_model(g, seed=3)
    omega = 2 * np.pi * 0.5
    s = capi.Solver(g)
    s.set_formulation(capi.FORM_CCGD)
    s.update_cond(m.m_earth, m.air_cond)
    s.update_freq(omega)
    s.set_control(IterPerDivCor=1000, MaxDivCor=20, tolEMfwd=1e-12, precision=capi.PREC_MIXED)
    e, rc = s.fwdsolve(bc=mbc.boundary_1d(m, omega, 1))
    d = s.diagnostics()
    assert rc == 0 and d["final_relres"] <= 1e-12
    h = d["EMrelErr"]
    first = h[: 1 + int(np.argmax(h < 1e-7))]
    assert first.size < h.size and first.min() > 1e-12
