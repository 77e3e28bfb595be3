"""mt3d_mult_aii_device_noalloc against mt3d_mult_aii (other FP64 kernels) at
the edges of its 16 x 4 x 4 node tiles, from the smallest grid up, and with y
on top of x, which takes another route; relative 2-norm 1e-13 as the operator
tests."""
import numpy as np
import pytest
import torch

from helpers import random_model, relerr
from mt3d import capi, models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(2, 2, 2), (2, 3, 5), (15, 3, 4), (16, 4, 3), (17, 5, 7), (31, 8, 9), (33, 13, 16)])
@pytest.mark.parametrize("formulation", [capi.FORM_CCDC, capi.FORM_CCGD])
@pytest.mark.parametrize("adjt", [False, True])
def test_interior_product(cuda, nx, ny, nz, formulation, adjt):
    rng = np.random.default_rng(nx + 100 * ny + 10000 * nz)
    g = models.Grid(rng.uniform(200.0, 900.0, nx), rng.uniform(200.0, 900.0, ny), rng.uniform(40.0, 400.0, nz),
                    max(1, nz // 4))
    m = random_model(g, seed=nz)
    s = capi.Solver(g)
    s.set_formulation(formulation)
    s.update_cond(m.m_earth, m.air_cond)
    s.update_freq(2 * np.pi * 0.3)
    x = rng.standard_normal(s.nEi) + 1j * rng.standard_normal(s.nEi)
    want = s.mult_aii(x, adjt=adjt)
    xd = torch.from_numpy(x).to("cuda")
    yd = torch.full_like(xd, complex(np.nan, np.nan))
    s.mult_aii_device_noalloc(xd.data_ptr(), yd.data_ptr(), adjt=adjt)
    torch.cuda.synchronize()
    assert np.array_equal(xd.cpu().numpy(), x)
    assert relerr(yd.cpu().numpy(), want) <= 1e-13
    s.mult_aii_device_noalloc(xd.data_ptr(), xd.data_ptr(), adjt=adjt)
    torch.cuda.synchronize()
    assert relerr(xd.cpu().numpy(), want) <= 1e-13
