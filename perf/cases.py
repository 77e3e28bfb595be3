"""The work this solver is used for, as cases that can be timed and checked.

The cases are what a ModEM host asks of the library, each through the C ABI
(include/mt3d.h) or its Python binding (mt3d/capi.py):

  apply   y = A x on device vectors (mt3d_mult_aii_device_noalloc): the
          operator alone, for callers with an iteration of their own;
  bc      boundary data and first guess of one polarisation
          (mt3d_compute_bc_device): once per frequency and polarisation;
  solve   FWDsolve3D of a batch of forward right-hand sides on one grid,
          fields resident on the device (mt3d_fwdsolve_batch_device), mixed
          precision with the polynomial or the diagonal preconditioner, or
          plain FP64;
  multi   the same over two grids of uneven size in one call
          (mt3d_fwdsolve_multi_device);
  data    impedances at surface sites from the fields of both polarisations
          (mt3d_impedance_device), or the adjoint sources of their data weights
          (mt3d_lmult_t_device).

Grids follow the repository's own configurations (24^3, 40x40x40, 64x64x48,
100x100x60, 200x200x100) and odd sizes between them; the conductivity is a
seeded random field of log10 resistivity (mean 2, standard deviation 0.5,
correlation length 5 cells, clipped to 0..4), air above.  The forward solves go to a relative residual of 1e-12, the tolerance of gradient
checks, so that the fields are those of the system to about ten digits
whatever path an iteration took to them.  Transposed solves run through the
same kernels; their right-hand sides carry a correction 1 / (omega mu0) times
the source, so a residual of 1e-12 of it leaves their fields only seven
digits, and they are not listed for that.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "modem-gpu_b200"))
from mt3d import capi, models  # noqa: E402

MU0 = 3.14159265357898 * 0.0000004
SIGMA_AIR = float(np.float32(1.0e-10))
C128 = torch.complex128


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def _apply(nx, ny, na, ne, gd, adjt, hz):
    return {"kind": "apply", "nx": nx, "ny": ny, "na": na, "ne": ne, "gd": gd, "adjt": adjt, "hz": hz}


def _bc(nx, ny, na, ne, mode, hz):
    return {"kind": "bc", "nx": nx, "ny": ny, "na": na, "ne": ne, "mode": mode, "hz": hz}


def _solve(nx, ny, na, ne, nf, lo, hi, pols, poly, fp64):
    """nf frequencies log-spaced lo .. hi Hz, `pols` polarisations of each."""
    return {"kind": "solve", "nx": nx, "ny": ny, "na": na, "ne": ne, "nf": nf, "lo": lo, "hi": hi, "pols": pols,
            "poly": poly, "fp64": fp64}


def _multi(nx, ny, na, ne, nx2, ny2, na2, ne2, nf, lo, hi):
    return {"kind": "multi", "nx": nx, "ny": ny, "na": na, "ne": ne, "nx2": nx2, "ny2": ny2, "na2": na2, "ne2": ne2,
            "nf": nf, "lo": lo, "hi": hi, "pols": 2, "poly": 0.9, "fp64": False}


def _data(nx, ny, na, ne, nrec, adj, hz):
    """nrec x nrec sites: impedances, or (adj) their adjoint sources."""
    return {"kind": "data", "nx": nx, "ny": ny, "na": na, "ne": ne, "nrec": nrec, "adj": adj, "hz": hz}


def listed():
    out = []

    def add(name, case):
        out.append(dict(case, name=name))

    # the smallest call: the curl-curl product on the 24^3 grid, bound by its launches
    add("apply 24^3", _apply(24, 24, 8, 16, False, False, 0.1))
    # the largest grid that entry takes, odd sizes, grad-div and transposed
    add("apply 51x50x53 gd adj", _apply(51, 50, 9, 44, True, True, 10.0))
    # boundary data: a small grid, an odd one, and the 200x200x100 model's
    add("bc 40^3", _bc(40, 40, 8, 32, 1, 1.0))
    add("bc 101x83x61", _bc(101, 83, 10, 51, 2, 0.03))
    add("bc 200x200x100", _bc(200, 200, 12, 88, 2, 10.0))
    # one frequency's forward pair on the small forward grid: latency bound
    add("solve 24^3", _solve(24, 24, 8, 16, 1, 0.1, 0.1, 2, 0.9, False))
    # plain FP64, one frequency's pair
    add("solve 64x64x48 fp64", _solve(64, 64, 10, 38, 1, 1.0, 1.0, 2, 0.0, True))
    # the diagonal preconditioner alone (the library's default), odd sizes, two frequencies
    add("solve 49x75x43 diag", _solve(49, 75, 9, 34, 2, 0.1, 10.0, 2, 0.0, False))
    # two uneven grids in one call, four frequencies of each
    add("multi 40^3 + 64x64x48", _multi(40, 40, 8, 32, 64, 64, 10, 38, 4, 0.01, 100.0))
    # the precision model: one frequency's pair
    add("solve 100x100x60", _solve(100, 100, 10, 50, 1, 1.0, 1.0, 2, 0.9, False))
    # the largest model: one polarisation
    add("solve 200x200x100", _solve(200, 200, 12, 88, 1, 100.0, 100.0, 1, 0.9, False))
    # adjoint sources of a 20 x 20 array of sites
    add("sources 100x100x60", _data(100, 100, 10, 50, 20, True, 1.0))
    return out


def draw(rng):
    def size(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    def hz(lo, hi):
        return round(lo * (hi / lo) ** rng.random(), 5)

    kind = rng.choice(["apply", "apply", "bc", "bc", "bc", "data", "solve", "solve", "solve", "solve", "multi"])
    if kind == "apply":
        nx, ny, nz = size(16, 51), size(16, 51), size(16, 51)
        na = max(5, nz // 6)
        return _apply(nx, ny, na, nz - na, rng.random() < 0.5, rng.random() < 0.5, hz(1e-3, 1e2))
    if kind == "bc":
        nx, ny, nz = size(24, 200), size(24, 200), size(24, 100)
        na = max(5, nz // 8)
        return _bc(nx, ny, na, nz - na, rng.choice([1, 2]), hz(1e-3, 1e2))
    if kind == "multi":
        z, z2 = size(24, 40), size(28, 48)
        return _multi(size(24, 48), size(24, 48), 7, z - 7, size(36, 64), size(36, 64), 8, z2 - 8,
                      rng.choice([1, 2, 3]), hz(0.03, 0.3), hz(1.0, 50.0))
    nx, ny, nz = size(24, 110), size(24, 110), size(24, 60)
    na = max(7, nz // 7)
    fp64 = rng.random() < 0.25
    poly = 0.0 if fp64 else rng.choice([0.0, 0.9, 0.9])
    f = hz(0.05, 50.0)
    if kind == "data":
        return _data(nx, ny, na, nz - na, rng.randrange(3, 21), rng.random() < 0.5, f)
    return _solve(nx, ny, na, nz - na, 1, f, f, rng.choice([1, 2]), poly, fp64)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _axis(n, core, pad, growth):
    p = core * growth ** np.arange(1, pad + 1)
    return np.concatenate([p[::-1], np.full(n - 2 * pad, core), p])


def _grid(nx, ny, na, ne):
    """Core cells of 500 m with four growing cells of padding on every side;
    layers growing from 50 m downwards (slower the more there are, as the
    repository's configurations do) and upwards into the air."""
    growth = 1.2 if ne <= 50 else 1.2 - 0.13 * (ne - 50) / 38
    air = 1.5 if na <= 10 else 1.6
    earth = 50.0 * growth ** np.arange(ne)
    return models.Grid(_axis(nx, 500.0, 4, 1.5), _axis(ny, 500.0, 4, 1.5),
                       np.concatenate([(50.0 * air ** np.arange(na))[::-1], earth]), na)


def _field(shape, seed):
    """Gaussian random field on the (z, y, x) cells, exponential covariance
    of 5 cells, drawn in the spectrum of a periodic box."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    noise = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    k2 = sum((torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * 2 * math.pi).square().reshape(
        [-1 if a == b else 1 for b in range(3)]) for a, n in enumerate(shape))
    f = torch.fft.ifftn(torch.fft.fftn(noise) / (1.0 + 25.0 * k2)).real
    return (f - f.mean()) / f.std()


def _model(case, seed, sfx=""):
    """The grid and ln(sigma) of its earth cells, shape (ne, ny, nx), on the device."""
    g = _grid(case["nx" + sfx], case["ny" + sfx], case["na" + sfx], case["ne" + sfx])
    lr = torch.clamp(2.0 + 0.5 * _field((g.nzEarth, g.ny, g.nx), seed), 0.0, 4.0)
    return g, -math.log(10.0) * lr


def _normal(n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.view_as_complex(torch.randn((n, 2), generator=gen, device="cuda", dtype=torch.float64))


def _cells(g, nrec):
    """Cells under the sites: nrec x nrec of the core, y slowest."""
    ix = np.linspace(g.nx * 0.3, g.nx * 0.7, nrec).astype(int)
    iy = np.linspace(g.ny * 0.3, g.ny * 0.7, nrec).astype(int)
    return np.tile(ix, nrec), np.repeat(iy, nrec)


def _sites(g, nrec):
    """Sites at the surface centres of those cells, from the grid origin."""
    i, j = _cells(g, nrec)
    x, y = np.concatenate([[0.0], np.cumsum(g.dx)]), np.concatenate([[0.0], np.cumsum(g.dy)])
    return np.stack([(x[i] + x[i + 1]) / 2, (y[j] + y[j + 1]) / 2, np.zeros(i.size)], 1)


def _weights(nsite, seed):
    """Data weights: residuals over squared errors, of no particular scale."""
    rng = np.random.default_rng(seed)
    return rng.standard_normal((nsite, 2, 2)) + 1j * rng.standard_normal((nsite, 2, 2))


def _dual(d):
    return np.concatenate([[d[0]], d[:-1] + d[1:], [d[-1]]]) / 2


def _omegas(case):
    lo, hi, n = case["lo"], case["hi"], case["nf"]
    f = [lo] if n == 1 else [lo * (hi / lo) ** (i / (n - 1)) for i in range(n)]
    return [2 * math.pi * x for x in f]


def _rows(case):
    """(omega, mode) of every right-hand side."""
    return [(w, mode) for w in _omegas(case) for mode in (1, 2)[:case["pols"]]]


def _solver(g, m, gd):
    s = capi.Solver(g)
    s.set_formulation(capi.FORM_CCGD if gd else capi.FORM_CCDC)
    s.update_cond(m.cpu().numpy().reshape(-1), models.AIR_COND_LOGE)
    return s


def _compute_bc(s, mode, omega, e0):
    rc = s.L.mt3d_compute_bc_device(s.h, mode, ctypes.c_double(omega), ctypes.c_void_p(e0.data_ptr()))
    if rc:
        raise RuntimeError("mt3d_compute_bc_device: status %d" % rc)


def _controlled(case, g, m):
    """A solver under the control a solve runs with: cycles of 300 iterations
    between FP64 residuals, restarted only there."""
    s = _solver(g, m, True)
    s.set_control(IterPerDivCor=300, MaxDivCor=60, tolEMfwd=1e-12, tolEMadj=1e-12,
                  precision=capi.PREC_FP64 if case["fp64"] else capi.PREC_MIXED)
    s.set_restart(0)
    s.set_poly(case["poly"])
    return s


def _solve_state(case, seed, sfx=""):
    g, m = _model(case, seed, sfx)
    s = _controlled(case, g, m)
    rows = _rows(case)
    bc = torch.empty((len(rows), s.nE), dtype=C128, device="cuda")
    for r, (w, mode) in enumerate(rows):
        _compute_bc(s, mode, w, bc[r])  # boundary data and first guess in one
    return {"s": s, "om": np.array([r[0] for r in rows]), "bc": bc, "e": torch.empty_like(bc)}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("apply", "bc", "data"):
        g, m = _model(case, seed)
        s = _solver(g, m, kind == "apply" and case["gd"])
        omega = 2 * math.pi * case["hz"]
        s.update_freq(omega)
        st = {"kind": kind, "s": s, "omega": omega}
        if kind == "apply":
            st["adjt"] = case["adjt"]
            st["x"] = _normal(s.nEi, seed + 1)
            st["y"] = torch.empty_like(st["x"])
        elif kind == "bc":
            st["mode"] = case["mode"]
            st["e0"] = torch.empty(s.nE, dtype=C128, device="cuda")
        else:
            n, st["adj"], st["sites"] = case["nrec"] ** 2, case["adj"], _sites(g, case["nrec"])
            st["e"] = torch.empty((2, s.nE), dtype=C128, device="cuda")
            for mode in (1, 2):  # the fields: the 2-D solutions
                _compute_bc(s, mode, omega, st["e"][mode - 1])
            if case["adj"]:
                st["d"], st["src"] = _weights(n, seed + 1), torch.empty_like(st["e"])
        return st
    if kind == "solve":
        return dict(_solve_state(case, seed), kind=kind)
    return {"kind": kind, "grids": [_solve_state(case, seed), _solve_state(case, seed + 7, "2")]}


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(st):
    kind = st["kind"]
    if kind == "apply":
        st["s"].mult_aii_device_noalloc(st["x"].data_ptr(), st["y"].data_ptr(), st["adjt"])
        return st["y"]
    if kind == "bc":
        _compute_bc(st["s"], st["mode"], st["omega"], st["e0"])
        return st["e0"]
    if kind == "data":
        e1, e2 = st["e"][0].data_ptr(), st["e"][1].data_ptr()
        if not st["adj"]:
            return st["s"].impedance(st["omega"], st["sites"], e1, e2)
        st["s"].lmult_t_device(st["omega"], st["sites"], e1, e2, st["d"], st["src"][0].data_ptr(),
                               st["src"][1].data_ptr())
        return list(st["src"].unbind())
    gs = st["grids"] if kind == "multi" else [st]
    for q in gs:
        q["e"].copy_(q["bc"])  # the 2-D solution is the first guess
    if kind == "multi":
        capi.fwdsolve_multi([q["s"] for q in gs], [q["om"] for q in gs], [q["e"].data_ptr() for q in gs],
                            bc=[q["bc"].data_ptr() for q in gs], device=True)
    else:
        st["s"].fwdsolve_batch_device(st["om"], st["e"].data_ptr(), st["bc"].data_ptr())
    return [list(q["e"].unbind()) for q in gs]


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    def edges(sfx=""):
        g = _grid(case["nx" + sfx], case["ny" + sfx], case["na" + sfx], case["ne" + sfx])
        return g.n_edges, g.n_interior_edges

    nE, nEi = edges()
    kind = case["kind"]
    if kind == "apply":  # x, y and sigma once; about 60 operations per edge
        return {"bytes": 40 * nEi + (8 * nE // 3 if case["gd"] else 0), "flops": 60 * nEi}
    nz = case["na"] + case["ne"]
    if kind == "bc":
        # a symmetric band factorisation of every slice (complex multiply-adds
        # of 8 operations, half the band), the cells read, the field written
        nh, ns = (case["ny"], case["nx"]) if case["mode"] == 2 else (case["nx"], case["ny"])
        m = min(nz, nh) - 1
        return {"bytes": 16 * nE + 8 * case["nx"] * case["ny"] * nz, "flops": 4.0 * ns * (nh - 1) * (nz - 1) * m * m}
    # first guess and boundary data in, field out, sigma: how often the method
    # passes over its vectors is its own affair
    if kind == "data":
        # per site some 32 entries of the fields for E and B; impedances out,
        # or the source vectors, zeros and all
        n = case["nrec"] ** 2
        return {"bytes": n * (32 * 2 * 16 + 64) + (2 * 16 * nE if case["adj"] else 0), "flops": n * 1000}
    rows = len(_rows(case))
    if kind == "multi":
        nE += edges("2")[0]
    return {"bytes": rows * nE * 16 * 3 + 8 * nE, "flops": rows * nE * 200}


# --------------------------------------------------------------------------
# the same in 64 bits with plain torch
# --------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "multi":
        return [_exact_solve(case, seed), _exact_solve(case, seed + 7, "2")]
    if kind == "solve":
        r = _exact_solve(case, seed)
        return None if r is None else [r]
    g, m = _model(case, seed)
    ex = _Exact(g, m, kind == "apply" and case["gd"])
    omega = 2 * math.pi * case["hz"]
    if kind == "bc":
        return ex.boundary(case["mode"], omega)
    if kind == "data":
        e0, cells = [ex.boundary(mode, omega) for mode in (1, 2)], _cells(g, case["nrec"])
        if not case["adj"]:
            return ex.impedance(e0, omega, cells)
        return ex.impedance_sources(e0, omega, cells, _weights(case["nrec"] ** 2, seed + 1))
    x = torch.zeros(g.n_edges, dtype=C128, device="cuda")
    x[ex.interior] = _normal(int(ex.interior.sum()), seed + 1)
    return ex.operator(x, omega, case["adjt"])[ex.interior]


def _exact_solve(case, seed, sfx=""):
    g, m = _model(case, seed, sfx)
    if g.n_edges > 2500000:
        return None  # minutes of plain torch
    ex = _Exact(g, m, True)
    out = []
    for w, mode in _rows(case):
        e0 = ex.boundary(mode, w)
        b = torch.where(ex.interior, -ex.curlcurl(torch.where(ex.interior, 0, e0)), 0)
        x = ex.solve(b, w)
        out.append(None if x is None else torch.where(ex.interior, x, e0))
    return out


class _Exact:
    """The staggered-grid operators on flat full edge vectors (x-, y-, then
    z-edges, x fastest), components as (z, y, x) arrays."""

    def __init__(self, g, m, gd):
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        self.g, self.gd = g, gd
        nx, ny, nz, na = g.nx, g.ny, g.nz, g.nzAir
        self.d = dx, dy, dz = t(g.dx), t(g.dy), t(g.dz)
        self.D = dX, dY, dZ = t(_dual(g.dx)), t(_dual(g.dy)), t(_dual(g.dz))
        X, Y, Z = (lambda a: a[None, None, :]), (lambda a: a[None, :, None]), (lambda a: a[:, None, None])
        self.shapes = [(nz + 1, ny + 1, nx), (nz + 1, ny, nx + 1), (nz, ny + 1, nx + 1)]
        full = lambda parts: torch.cat([p.expand(s).reshape(-1) for p, s in zip(parts, self.shapes)])
        self.L = [X(dx), Y(dy), Z(dz)]
        self.A = [Y(dY) * Z(dZ), X(dX) * Z(dZ), X(dX) * Y(dY)]
        self.vE = full([l * a for l, a in zip(self.L, self.A)])
        # dual edge length over face area of the x-, y- and z-faces
        self.W = [X(dX) / (Y(dy) * Z(dz)), Y(dY) / (X(dx) * Z(dz)), Z(dZ) / (X(dx) * Y(dy))]
        inx = lambda n: (torch.arange(n + 1, device="cuda") > 0) & (torch.arange(n + 1, device="cuda") < n)
        ix, iy, iz = inx(nx), inx(ny), inx(nz)
        self.interior = full([Y(iy) & Z(iz), X(ix) & Z(iz), X(ix) & Y(iy)])
        self.sig = torch.cat([torch.full((na, ny, nx), SIGMA_AIR, device="cuda", dtype=torch.float64), m.exp()])
        vc = X(dx) * Y(dy) * Z(dz)

        def mean(axes):
            """Volume-weighted mean of the cells around the edges or nodes."""
            pad = [1 if a in axes else 0 for a in (2, 2, 1, 1, 0, 0)]
            num, den = (torch.nn.functional.pad(q, pad) for q in (self.sig * vc, vc))
            for a in axes:
                n = num.shape[a] - 1
                num = num.narrow(a, 0, n) + num.narrow(a, 1, n)
                den = den.narrow(a, 0, n) + den.narrow(a, 1, n)
            return num / den

        s = [mean((0, 1)), mean((0, 2)), mean((1, 2))]
        if gd:
            s = torch.where(self.interior, torch.cat([q.reshape(-1) for q in s]), 0)
            sx, sy, sz = self.split(s)
            earth = torch.zeros((nz + 1, ny + 1, nx + 1), dtype=torch.bool, device="cuda")
            for q, a in ((sx, 2), (sy, 1), (sz, 0)):
                e = q >= 1.1 * SIGMA_AIR
                earth.narrow(a, 0, q.shape[a]).logical_or_(e)
                earth.narrow(a, 1, q.shape[a]).logical_or_(e)
            inner = X(ix) & Y(iy) & Z(iz)
            self.earth = earth & inner
            vN = X(dX) * Y(dY) * Z(dZ)
            self.wN = torch.where(inner, torch.where(earth, 1 / (mean((0, 1, 2)) * vN), 1 / vN), 0)
            self.sE = s
        else:  # the plain curl-curl operator has no conductivity on the air cells' edges
            s[0][:na, :ny] = 0
            s[1][:na, :, :nx] = 0
            s[2][:na, :ny, :nx] = 0
            self.sE = torch.cat([q.reshape(-1) for q in s])

    def split(self, e):
        out, o = [], 0
        for s in self.shapes:
            n = s[0] * s[1] * s[2]
            out.append(e[o:o + n].reshape(s))
            o += n
        return out

    def curlcurl(self, e):
        """V_E curl curl e, as L T^t W T L on all edges."""
        x, y, z = (c * l for c, l in zip(self.split(e), self.L))
        dif = lambda a, d: a.diff(dim=d)
        fx = (dif(z, 1) - dif(y, 0)) * self.W[0]
        fy = (dif(x, 0) - dif(z, 2)) * self.W[1]
        fz = (dif(y, 2) - dif(x, 1)) * self.W[2]

        def dift(a, d):  # transpose of diff
            pad = [0, 0, 0, 0, 0, 0]
            lo, hi = list(pad), list(pad)
            lo[2 * (2 - d)], hi[2 * (2 - d) + 1] = 1, 1
            return torch.nn.functional.pad(a, lo) - torch.nn.functional.pad(a, hi)

        ox = (dift(fy, 0) - dift(fz, 1)) * self.L[0]
        oy = (dift(fz, 2) - dift(fx, 0)) * self.L[1]
        oz = (dift(fx, 1) - dift(fy, 2)) * self.L[2]
        return torch.cat([ox.reshape(-1), oy.reshape(-1), oz.reshape(-1)])

    def nodes(self, parts):
        """G^t: what ends at a node minus what starts there."""
        out = torch.zeros(self.wN.shape, dtype=C128, device="cuda")
        for q, a in zip(parts, (2, 1, 0)):
            out.narrow(a, 1, q.shape[a]).add_(q)
            out.narrow(a, 0, q.shape[a]).sub_(q)
        return out

    def graddiv(self, e, adjt):
        s, x = self.split(self.sE), self.split(e)
        one = [q * a for q, a in zip(x, self.A)]
        if not adjt:
            phi = self.wN * torch.where(self.earth, self.nodes([q * c for q, c in zip(one, s)]), self.nodes(one))
            out = [phi.diff(dim=a) * d for a, d in zip((2, 1, 0), self.A)]
        else:
            phi = self.wN * self.nodes(one)
            pe, pa = torch.where(self.earth, phi, 0), torch.where(self.earth, 0, phi)
            out = [(pe.diff(dim=a) * c + pa.diff(dim=a)) * d for a, c, d in zip((2, 1, 0), s, self.A)]
        return torch.cat([q.reshape(-1) for q in out])

    def operator(self, e, omega, adjt=False):
        """A e on the interior edges (zero elsewhere), e zero on the boundary."""
        out = self.curlcurl(e) + (1j if adjt else -1j) * omega * MU0 * self.sE * self.vE * e
        if self.gd:
            out = out + self.graddiv(e, adjt)
        return torch.where(self.interior, out, 0)

    def diagonal(self, omega):
        """Diagonal of A from the same factors."""
        nx, ny, nz = self.g.nx, self.g.ny, self.g.nz

        def both(a, d):
            lo, hi = [0] * 6, [0] * 6
            lo[2 * (2 - d)], hi[2 * (2 - d) + 1] = 1, 1
            return torch.nn.functional.pad(a, lo) + torch.nn.functional.pad(a, hi)

        W = [w.expand(s) for w, s in zip(self.W, [(nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)])]
        d = [(both(W[1], 0) + both(W[2], 1)) * self.L[0] ** 2, (both(W[2], 2) + both(W[0], 0)) * self.L[1] ** 2,
             (both(W[0], 1) + both(W[1], 2)) * self.L[2] ** 2]
        s = self.split(self.sE)
        for q, a in enumerate((2, 1, 0)):
            n = self.shapes[q][a]
            lo, hi = self.wN.narrow(a, 0, n), self.wN.narrow(a, 1, n)
            el, eh = self.earth.narrow(a, 0, n), self.earth.narrow(a, 1, n)
            d[q] = d[q] + self.A[q] ** 2 * (lo * torch.where(el, s[q], 1) + hi * torch.where(eh, s[q], 1))
        d = torch.cat([q.reshape(-1) for q in d]) - 1j * omega * MU0 * self.sE * self.vE
        return torch.where(self.interior, d, 1)

    def solve(self, b, omega):
        """BiCGStab with the diagonal on the full vectors (boundary entries
        zero), restarted from the true residual, to 1e-13 of |b| or to where
        it gets no further; None short of 1e-12."""
        dinv = 1 / self.diagonal(omega)
        bn = torch.linalg.vector_norm(b)
        x = torch.zeros_like(b)
        for _ in range(12):
            r = b - self.operator(x, omega)
            if float(torch.linalg.vector_norm(r) / bn) < 1e-13:
                break
            rt, p, d = r.clone(), r.clone(), torch.zeros_like(b)
            rho = torch.vdot(rt, r)
            target = 1e-5 * torch.linalg.vector_norm(r)
            for it in range(4000):
                ph = dinv * p
                v = self.operator(ph, omega)
                alpha = rho / torch.vdot(rt, v)
                s = r - alpha * v
                sh = dinv * s
                t = self.operator(sh, omega)
                om = torch.vdot(t, s) / torch.vdot(t, t)
                d += alpha * ph + om * sh
                r = s - om * t
                if it % 16 == 15 and bool(torch.linalg.vector_norm(r) < torch.maximum(target, 5e-14 * bn)):
                    break
                rho, old = torch.vdot(rt, r), rho
                p = r + (rho / old) * (alpha / om) * (p - om * v)
            x = x + d
        r = b - self.operator(x, omega)
        return x if float(torch.linalg.vector_norm(r) / bn) < 1e-12 else None

    def functionals(self, e, omega, cells):
        """Ex, Ey, Bx, By at the surface centres of the cells (i, j): means of
        the edges or faces around them, B = (-i / omega) curl E."""
        i, j = (torch.from_numpy(q).cuda() for q in cells)
        k = self.g.nzAir
        (dx, dy, dz), (x, y, z) = self.d, self.split(e)
        bx, by = [], []
        for q in (k - 1, k):  # the faces above and below the surface
            fx = lambda a: (z[q, j + 1, a] - z[q, j, a]) / dy[j] - (y[q + 1, j, a] - y[q, j, a]) / dz[q]
            fy = lambda a: (x[q + 1, a, i] - x[q, a, i]) / dz[q] - (z[q, a, i + 1] - z[q, a, i]) / dx[i]
            bx.append((fx(i) + fx(i + 1)) / 2)
            by.append((fy(j) + fy(j + 1)) / 2)
        up = dz[k - 1] / (dz[k - 1] + dz[k])  # weight of the faces below
        mix = lambda b: (-1j / omega) * ((1 - up) * b[0] + up * b[1])
        return torch.stack([(x[k, j, i] + x[k, j + 1, i]) / 2, (y[k, j, i] + y[k, j, i + 1]) / 2, mix(bx), mix(by)])

    def impedance(self, e0, omega, cells):
        """Z = E B^-1 per site."""
        return torch.matmul(*self._eb(e0, omega, cells))

    def _eb(self, e0, omega, cells):
        v = torch.stack([self.functionals(e, omega, cells) for e in e0], -1)  # functional, site, polarisation
        return v[:2].permute(1, 0, 2), torch.linalg.inv(v[2:].permute(1, 0, 2))

    def impedance_sources(self, e0, omega, cells, d):
        """Sum over sites of conj(d_ij) times the derivative of Z_ij with
        respect to the field of each polarisation."""
        ee, binv = self._eb(e0, omega, cells)
        z = ee @ binv
        dc = torch.from_numpy(d).cuda().conj()
        out = []
        for k in range(2):
            s = (dc * binv[:, k][:, None, :]).sum(2)  # site, i
            f = torch.cat([s.T, -torch.einsum("si,sim->ms", s, z)])
            e = torch.zeros_like(e0[0], requires_grad=True)
            # the gradient of a complex-linear map is its conjugate transpose
            g, = torch.autograd.grad(self.functionals(e, omega, cells), e, f.conj())
            out.append(g.conj().resolve_conj())
        return out

    def boundary(self, mode, omega):
        """E0 of one polarisation: a 2-D TE problem per slice between 1-D
        columns (side columns in full, the bottom value of every other)."""
        g = self.g
        nz = g.nz
        # slices: conductivity (slice, h, k); the horizontal axis is y for mode 2, x for mode 1
        sig = self.sig.permute(2, 1, 0) if mode == 2 else self.sig.permute(1, 2, 0)
        sig = sig.contiguous()
        ns, nh = sig.shape[0], sig.shape[1]
        dh, dz = (self.d[1] if mode == 2 else self.d[0]), self.d[2]
        om = omega * MU0
        col = torch.cat([sig[:, :1], (sig[:, :-1] * dh[:-1, None] + sig[:, 1:] * dh[1:, None]) /
                         (dh[:-1] + dh[1:])[:, None], sig[:, -1:]], dim=1)
        c1 = self._columns(col.reshape(-1, nz), om).reshape(ns, nh + 1, nz + 1)
        cz, cy = dz[1:] + dz[:-1], dh[1:] + dh[:-1]  # at the inner nodes
        n, m = nh - 1, nz - 1
        wt = dh[:, None] * dz[None, :]
        sw = sig * wt
        quad = lambda a: a[..., :-1, :-1] + a[..., 1:, :-1] + a[..., :-1, 1:] + a[..., 1:, 1:]
        diag = (-2 * cz[None] * (1 / dh[1:] + 1 / dh[:-1])[:, None] - 2 * cy[:, None] * (1 / dz[1:] + 1 / dz[:-1])[None]
                )[None] + 1j * om * (cy[:, None] * cz[None])[None] * (quad(sw) / quad(wt))
        rhs = torch.zeros((ns, n, m), dtype=C128, device="cuda")
        rhs[:, 0] = -2 * cz / dh[0] * c1[:, 0, 1:nz]
        rhs[:, -1] -= 2 * cz / dh[-1] * c1[:, nh, 1:nz]
        rhs[:, :, 0] -= 2 * cy / dz[0]
        rhs[:, :, -1] -= 2 * cy / dz[-1] * c1[:, 1:nh, nz]
        inv, y = [], []
        for q in range(n):
            S = torch.diag_embed(diag[:, q])
            off = 2 * cy[q] / dz[1:-1]
            S += torch.diag(off, 1) + torch.diag(off, -1)
            f = rhs[:, q]
            if q:
                w = 2 * cz / dh[q]
                S = S - w[None, :, None] * inv[-1] * w[None, None, :]
                f = f - w * (inv[-1] @ y[-1][..., None])[..., 0]
            inv.append(torch.linalg.inv(S))
            y.append(f)
        u = torch.zeros((ns, nh + 1, nz + 1), dtype=C128, device="cuda")
        u[:, 0], u[:, nh], u[:, :, 0] = c1[:, 0], c1[:, nh], 1
        u[:, :, nz] = 0
        for q in range(n - 1, -1, -1):
            f = y[q] if q == n - 1 else y[q] - 2 * cz / dh[q + 1] * u[:, q + 2, 1:nz]
            u[:, q + 1, 1:nz] = (inv[q] @ f[..., None])[..., 0]
        e = torch.zeros(g.n_edges, dtype=C128, device="cuda")
        self.split(e)[0 if mode == 2 else 1].copy_(u.permute(2, 1, 0) if mode == 2 else u.permute(2, 0, 1))
        return e

    def _columns(self, s, om):
        """1-D TE columns (ncol, nz): E = 1 at the top, one skin depth of the
        last layer below the bottom; all nz + 1 nodes."""
        nz = s.shape[1]
        dz = self.d[2].expand_as(s)
        last = s[:, -1:]
        s = torch.cat([s, last], 1)
        d = torch.cat([dz, torch.sqrt(2 / (last * om))], 1)
        au, ad = 2 / d[:, :-1], 2 / d[:, 1:]
        diag = -au - ad + 1j * om * (s[:, 1:] * d[:, 1:] + s[:, :-1] * d[:, :-1])
        cp, dp = [], []
        for j in range(nz):
            if j == 0:
                den, num = diag[:, 0], (-au[:, 0]).to(C128)
            else:
                den, num = diag[:, j] - ad[:, j - 1] * cp[-1], -ad[:, j - 1] * dp[-1]
            cp.append(ad[:, j] / den)
            dp.append(num / den)
        x = [dp[-1]]
        for j in range(nz - 2, -1, -1):
            x.append(dp[j] - cp[j] * x[-1])
        return torch.stack([torch.ones_like(x[0])] + x[::-1], 1)
