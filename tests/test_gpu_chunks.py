"""The staged stencils over chunks of node planes of every kind (mt3d_set_chunks):
the whole column in one chunk, two, three, one plane a chunk, and a count that
leaves chunks without planes.  The grid has 71 node planes, so a single chunk goes
round every ring of slots many times and reads the plane tables of the fused
stencil (32 planes each) three times, and its last tiles hold two node columns and
three rows.

Products: FP64 (kernel 1) to 1e-13 in the 2-norm, FP32 (2, 3) per edge within
64 * 2^-24 (|A| |x|)_e, as in test_gpu_kernels.py.

Cycles: five iterations of the fused FP32 BiCGStab, so its two or four products, inner
products, shadow resets and final conversion, against the method restated with
the assembled operator in 64 bits.  The restatement in 32 bits (sums of the inner
products in 64, as the kernels') differs from that by its rounding alone; the
kernels may by sixteen times as much, since they form curls and potentials whose
cross terms, of the size of the diagonal, cancel where the assembled operator has
a zero."""
import numpy as np
import pytest

from helpers import assemble_A, random_model, relerr
from mt3d import bc as mbc
from mt3d import capi, models
from oracle.oracle import interior_edge_mask

pytestmark = pytest.mark.gpu

CHUNKS = [1, 2, 3, 48, 71]  # 48: chunks of 2 planes, the last 12 without any
OMEGAS = 2 * np.pi * np.array([0.3, 3.0])


def grid():
    return models.make_grid(33, 18, 10, 60, core=400.0, n_pad=3, pad_growth=1.5, air_first=60.0, air_growth=1.6,
                            earth_first=60.0, earth_growth=1.05)


def operators(g, m, form):
    """(interior operator, right-hand side of boundary data) per frequency"""
    from oracle.sp2 import SP2
    mask = interior_edge_mask(g)
    out = []
    for k, om in enumerate(OMEGAS):
        A = assemble_A(g, m, om)
        bc = mbc.boundary_1d(m, om, 1 + k)
        b = -(A[mask][:, ~mask] @ bc[~mask])
        if form == capi.FORM_CCGD:
            ref = SP2(g, m)
            ref.set_freq(om)
            out.append((ref.A.tocsr(), b, bc))
        else:
            out.append((A[mask][:, mask].tocsr(), b, bc))
    return out


def bicgstab(A, b, n, c, restart, dtype):
    """n iterations of BiCGStab from zero, preconditioned with D = diag A or
    c D^-1 (2 - c A D^-1); the shadow is reset to the residual every `restart`
    iterations.  Returns the best iterate and its iteration."""
    scale = np.linalg.norm(b)
    A, b = A.astype(dtype), (b / scale).astype(dtype)
    d = 1 / A.diagonal()
    t_ = dtype(1).real.dtype.type

    def M(v):
        w = d * v
        return w if not c else t_(c) * (t_(2) * w - t_(c) * (d * (A @ w)))

    def dot(x, y):
        return np.vdot(x.astype(complex), y.astype(complex))

    x = np.zeros_like(b)
    r, rt, p = b, b, b
    rho = dot(rt, r)
    best, kept, at = 1.0, x, 0
    for it in range(1, n + 1):
        ph = M(p)
        v = A @ ph
        al = rho / dot(rt, v)
        s = r - dtype(al) * v
        sh = M(s)
        t = A @ sh
        om = dot(t, s) / dot(t, t).real
        x = x + dtype(al) * ph + dtype(om) * sh
        r = s - dtype(om) * t
        rn = np.sqrt(dot(r, r).real)
        if rn < best:
            best, kept, at = rn, x, it
        if restart and it % restart == 0:
            rt, p, rho = r, r, dot(r, r)
            continue
        rho, rho1 = dot(rt, r), rho
        p = r + dtype((rho / rho1) * (al / om)) * (p - dtype(om) * v)
    return kept.astype(complex) * scale, at


@pytest.fixture(scope="module", params=[capi.FORM_CCDC, capi.FORM_CCGD], ids=["ccdc", "ccgd"])
def prob(cuda, request):
    g = grid()
    m = random_model(g, seed=6)
    s = capi.Solver(g)
    s.set_formulation(request.param)
    s.update_cond(m.m_earth, m.air_cond)
    return g, interior_edge_mask(g), operators(g, m, request.param), s, request.param


@pytest.mark.parametrize("chunks", CHUNKS)
@pytest.mark.parametrize("kernel", [1, 2, 3])
def test_products(prob, kernel, chunks):
    g, mask, ops, s, _ = prob
    A = ops[1][0]
    s.set_control(precision=capi.PREC_MIXED)
    s.update_freq(OMEGAS[1])
    s.set_chunks(chunks)
    rng = np.random.default_rng(2)
    x = np.zeros(g.n_edges, complex)
    x[mask] = rng.standard_normal(mask.sum()) + 1j * rng.standard_normal(mask.sum())
    x = x.astype(np.complex64).astype(complex)
    y = s.apply_kernel(kernel, x)
    assert np.all(y[~mask] == 0)
    if kernel == 1:
        assert relerr(y[mask], A @ x[mask]) < 1e-13
        return
    D = A.diagonal() if kernel == 3 else np.ones(mask.sum())
    err = np.abs(y[mask] - (A @ x[mask]) / D)
    assert np.all(err <= 64 * 2.0 ** -24 * (abs(A) @ np.abs(x[mask])) / np.abs(D))


@pytest.mark.parametrize("poly,restart", [(0.0, 0), (0.0, 2), (0.9, 0), (0.9, 2)])
def test_cycles(prob, poly, restart):
    g, mask, ops, s, form = prob
    resets = restart if form == capi.FORM_CCGD else 0  # the grad-div formulation's, as the reference's
    want = []
    for A, b, _ in ops:
        x64, at = bicgstab(A, b, 5, poly, resets, np.complex128)
        x32, at32 = bicgstab(A, b, 5, poly, resets, np.complex64)
        assert at == at32 >= 1
        want.append((x64, 16 * relerr(x32, x64)))
    s.set_control(IterPerDivCor=5, MaxDivCor=1, tolEMfwd=1e-30, precision=capi.PREC_MIXED)
    s.set_poly(poly)
    s.set_restart(restart)
    for chunks in CHUNKS:
        s.set_chunks(chunks)
        e, _, rc = s.fwdsolve_batch(OMEGAS, bc=np.stack([o[2] for o in ops]))
        assert rc == 1
        for r, (x64, tol) in enumerate(want):
            assert relerr(e[r][mask], x64) <= tol, (chunks, r)
