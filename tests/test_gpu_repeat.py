"""The same call gives the same bits.  Every reduction of the solver sums in a
fixed order, so a solve that is repeated on one handle, or on another, differs
only if a kernel reads memory that another thread is writing.  Two did, with the
grad-div term.  In the staged FP64 stencil the copy of the node weights of the
third plane of a chunk went into the slot that slower warps were still reading
for the potentials of the first.  In the tensor-copy stencils nothing but a
barrier stood between the reads of a slot and the copy into it, which writes
through another proxy: node weights read before the barrier and used after it
were now and then those of two planes on.  The grid has tiles and plane chunks
enough for several waves of blocks; with either fault two repeats in three came
out different, in the first digits of the residual after 100 iterations."""
import numpy as np
import pytest

from helpers import random_model, relerr
from mt3d import bc as mbc
from mt3d import capi, models

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prob(cuda):
    g = models.make_grid(100, 100, 10, 50, core=500.0, n_pad=4, pad_growth=1.5, air_first=60.0, air_growth=1.6,
                         earth_first=60.0, earth_growth=1.1)
    m = random_model(g, seed=4)
    om = 2 * np.pi * np.repeat([0.01, 0.1, 1.0, 10.0], 2)
    bc = np.stack([mbc.boundary_1d(m, w, 1 + i % 2) for i, w in enumerate(om)])
    return g, m, om, bc


def _solver(g, m, form):
    s = capi.Solver(g)
    s.set_formulation(form)
    s.set_restart(0)
    s.update_cond(m.m_earth, m.air_cond)
    return s


@pytest.mark.parametrize("form,prec,poly", [(capi.FORM_CCDC, capi.PREC_MIXED, 0.9),
                                            (capi.FORM_CCDC, capi.PREC_MIXED, 0.0),
                                            (capi.FORM_CCDC, capi.PREC_FP64, 0.0),
                                            (capi.FORM_CCGD, capi.PREC_MIXED, 0.9),
                                            (capi.FORM_CCGD, capi.PREC_MIXED, 0.0),
                                            (capi.FORM_CCGD, capi.PREC_FP64, 0.0)],
                         ids=["ccdc-mixed-poly", "ccdc-mixed", "ccdc-fp64", "ccgd-mixed-poly", "ccgd-mixed", "ccgd-fp64"])
def test_repeated_solves_are_bitwise_equal(prob, form, prec, poly):
    g, m, om, bc = prob
    s = _solver(g, m, form)
    s.set_poly(poly)
    s.set_control(IterPerDivCor=100, MaxDivCor=2, tolEMfwd=1e-12, precision=prec)
    out = []
    for rep in range(4):
        if rep == 3:
            s = _solver(g, m, form)
            s.set_poly(poly)
            s.set_control(IterPerDivCor=100, MaxDivCor=2, tolEMfwd=1e-12, precision=prec)
        e, st, rc = s.fwdsolve_batch(om, bc=bc)
        out.append((e, *s.batch_diagnostics(om.size)))
    for e, it, rr in out[1:]:
        assert np.array_equal(it, out[0][1]) and np.array_equal(rr, out[0][2])
        assert np.array_equal(e, out[0][0])


@pytest.mark.parametrize("kernel", [1, 2, 3])
@pytest.mark.parametrize("form", [capi.FORM_CCDC, capi.FORM_CCGD], ids=["ccdc", "ccgd"])
def test_repeated_products_are_bitwise_equal(prob, form, kernel):
    g, m, om, bc = prob
    s = _solver(g, m, form)
    s.update_freq(om[0])
    s.set_control(precision=capi.PREC_MIXED)
    rng = np.random.default_rng(1)
    x = rng.standard_normal(g.n_edges) + 1j * rng.standard_normal(g.n_edges)
    x[np.setdiff1d(np.arange(g.n_edges), s.interior_index() - 1)] = 0
    y = s.apply_kernel(kernel, x)
    for _ in range(20):
        assert np.array_equal(s.apply_kernel(kernel, x), y)
    if kernel == 1:
        assert relerr(y, s.apply_kernel(0, x)) < 1e-13
