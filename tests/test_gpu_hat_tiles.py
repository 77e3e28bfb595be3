"""The fused FP32 stencil at the edges of its 16 x 16 tiles: grids whose last
tile holds one node row or column, all of them, or all but one, so that the
curls and potentials a thread takes from the lane, row or tile before it come
from every place they can, and plane counts down to a few.  The bound per edge
is that of an FP32 sum of the stencil's terms, 64 * 2^-24 (|A| |x|)_e / |D_e|,
with A assembled by oracle/sp2.py (grad-div) or tests/helpers.py."""
import numpy as np
import pytest

from helpers import assemble_A, random_model
from mt3d import capi, models
from oracle.oracle import interior_edge_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [capi.FORM_CCDC, capi.FORM_CCGD], ids=["ccdc", "ccgd"])
@pytest.mark.parametrize("dims", [(15, 16, 3, 4), (16, 15, 3, 5), (14, 31, 4, 6), (32, 17, 3, 30), (47, 33, 4, 9)])
def test_tile_edges(cuda, dims, form):
    g = models.make_grid(*dims, core=400.0, n_pad=3, pad_growth=1.5, air_first=60.0, air_growth=2.0, earth_first=60.0,
                         earth_growth=1.25)
    m = random_model(g, seed=dims[0])
    omega = 2 * np.pi * 3.0
    mask = interior_edge_mask(g)
    s = capi.Solver(g)
    s.set_formulation(form)
    s.update_cond(m.m_earth, m.air_cond)
    s.update_freq(omega)
    s.set_control(precision=capi.PREC_MIXED)
    if form == capi.FORM_CCGD:
        from oracle.sp2 import SP2
        ref = SP2(g, m)
        ref.set_freq(omega)
        A = ref.A
    else:
        A = assemble_A(g, m, omega)[mask][:, mask].tocsr()
    rng = np.random.default_rng(dims[1])
    x = np.zeros(g.n_edges, complex)
    x[mask] = rng.standard_normal(mask.sum()) + 1j * rng.standard_normal(mask.sum())
    x = x.astype(np.complex64).astype(np.complex128)
    y = s.apply_kernel(3, x)
    D = A.diagonal()
    err = np.abs(y[mask] - (A @ x[mask]) / D)
    assert np.all(err <= 64 * 2.0 ** -24 * (abs(A) @ np.abs(x[mask])) / np.abs(D))
    assert np.all(y[~mask] == 0)
