"""The boundary solver's reciprocals, which take the place of divisions at every
pivot of its eliminations.

Real: within one unit in the last place of the rounded 1 / x, over all mantissas
and exponents (the truncated series lies within 0.57 of one; see rcp_fast).
Complex: |z|^2 carries two roundings, its reciprocal one unit, each product one
more: 5 * 2^-53 relative in each component.  Where |z|^2 would over- or underflow,
Smith's algorithm, 1e-15 of |1 / z|."""
import numpy as np
import pytest

from helpers import random_model, small_grid
from mt3d import capi, models

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solver(cuda):
    return capi.Solver(models.make_grid(8, 8, 2, 6))


def mantissas(rng, n):
    """[1, 2): uniform, next to the ends, and with the lower 32 bits all ones or
    all zeros (what the instruction drops)"""
    u = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    k = n // 4
    u[:k] |= np.uint64(0xffffffff)
    u[k:2 * k] &= ~np.uint64(0xffffffff)
    u[2 * k:2 * k + 1000] = np.arange(1000, dtype=np.uint64)
    u[2 * k + 1000:2 * k + 2000] = np.uint64((1 << 52) - 1) - np.arange(1000, dtype=np.uint64)
    return (u | np.uint64(0x3ff0000000000000)).view(np.float64)


def test_real_within_one_ulp(solver):
    rng = np.random.default_rng(0)
    n = 1 << 20
    x = np.ldexp(mantissas(rng, n), rng.integers(-1020, 1020, n)) * rng.choice([-1.0, 1.0], n)
    y, _ = solver.check_reciprocal(x + 0j)
    want = 1.0 / x
    assert np.all(np.abs(y - want) <= np.spacing(np.abs(want)))


def test_complex(solver):
    rng = np.random.default_rng(1)
    n = 1 << 20
    e = rng.integers(-400, 400, n)
    re = np.ldexp(mantissas(rng, n), e) * rng.choice([-1.0, 1.0], n)
    im = np.ldexp(mantissas(rng, n)[rng.permutation(n)], e + rng.integers(-60, 60, n)) * rng.choice([-1.0, 1.0], n)
    _, w = solver.check_reciprocal(re + 1j * im)
    a, b = re.astype(np.longdouble), im.astype(np.longdouble)
    d = a * a + b * b
    u = np.longdouble(2.0) ** -53
    assert np.all(np.abs(w.real - a / d) <= 5 * u * np.abs(a / d))
    assert np.all(np.abs(w.imag + b / d) <= 5 * u * np.abs(b / d))


def test_complex_beyond_the_range_of_the_square(solver):
    rng = np.random.default_rng(2)
    n = 1 << 16
    e = rng.choice([-1, 1], n) * rng.integers(485, 1000, n)
    z = np.ldexp(rng.uniform(1, 2, n), e) + 1j * np.ldexp(rng.uniform(1, 2, n), e + rng.integers(-20, 20, n))
    _, w = solver.check_reciprocal(z)
    a, b = z.real.astype(np.longdouble), z.imag.astype(np.longdouble)
    d = a * a + b * b  # 15 bits of exponent
    assert np.all(np.hypot(w.real - a / d, w.imag + b / d) <= 1e-15 / np.sqrt(d))


@pytest.mark.parametrize("omega", [1e-300, 1e155, 1e165, 1e250, 1e300])
def test_boundary_data_at_absurd_frequencies(cuda, omega):
    """Finite at any frequency the call accepts; the field is gone below the top
    from 1e100 on, whatever the frequency."""
    g = small_grid(24, 20, 5, 19)
    m = random_model(g, seed=3)
    s = capi.Solver(g)
    s.update_cond(m.m_earth, m.air_cond)
    for imode in (1, 2):
        s.update_freq(omega)
        e = s.compute_bc(imode)
        assert np.all(np.isfinite(e.view(float)))
        if omega > 1:
            s.update_freq(1e100)
            assert np.max(np.abs(e - s.compute_bc(imode))) < 1e-30
