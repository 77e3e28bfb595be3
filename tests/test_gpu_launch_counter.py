"""mt3d_launch_counter is exact while several host threads use the library: a
handle that captures its cycle as a graph counts its own launches, whatever
another thread issues meanwhile."""
import threading

import numpy as np
import pytest

from helpers import random_model, small_grid
from mt3d import bc as mbc
from mt3d import capi

pytestmark = pytest.mark.gpu


def test_counter_with_a_second_thread(cuda):
    import torch
    g = small_grid()
    m = random_model(g, seed=3)
    omega = 2 * np.pi * 0.5
    bcv = mbc.boundary_1d(m, omega, 1)

    def solver():
        s = capi.Solver(g)
        s.set_formulation(capi.FORM_CCGD)
        s.set_poly(0.9)
        s.update_cond(m.m_earth, m.air_cond)
        s.update_freq(omega)
        return s

    L = capi.load()
    other = solver()
    other.set_stream(torch.cuda.Stream().cuda_stream)
    x = torch.zeros(other.nEi, dtype=torch.complex128, device="cuda")
    y = torch.empty_like(x)
    c0 = L.mt3d_launch_counter()
    other.mult_aii_device_noalloc(x.data_ptr(), y.data_ptr())
    per = L.mt3d_launch_counter() - c0
    assert per == 1

    def solve():  # a fresh handle (its set-up launches count too), so a fresh capture
        c = L.mt3d_launch_counter()
        s = solver()
        s.set_control(IterPerDivCor=120, MaxDivCor=20, precision=capi.PREC_MIXED)
        _, rc = s.fwdsolve(bc=bcv)
        assert rc == 0
        return s, L.mt3d_launch_counter() - c

    alone = solve()[1]
    assert solve()[1] == alone
    stop, calls = threading.Event(), [0]

    def work():
        while not stop.is_set():
            other.mult_aii_device_noalloc(x.data_ptr(), y.data_ptr())
            calls[0] += 1
            if calls[0] % 256 == 0:
                torch.cuda.synchronize()

    t = threading.Thread(target=work)
    c0 = L.mt3d_launch_counter()
    t.start()
    for _ in range(5):
        solve()
    stop.set()
    t.join()
    torch.cuda.synchronize()
    assert calls[0] > 100
    assert L.mt3d_launch_counter() - c0 == 5 * alone + calls[0] * per
