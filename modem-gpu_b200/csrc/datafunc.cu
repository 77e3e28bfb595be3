// datafunc.cu -- the Full_Impedance data functional on the GPU.
//
// dataResp for Full_Impedance (f90/3D_MT/DataFunc.f90:143-189): at each site
// the horizontal electric fields (EinterpSetUp, f90/3D_MT/EMfieldInterp.f90:
// 141-324) and magnetic fields (BfromESetUp, :470-647, on BinterpSetUp,
// :329-465) of the two polarisations are sparse linear functionals of the
// edge field; Z = E B^-1 (Kramer's rule), Z(2(i-1)+j) = sum_m E(i,m) B^-1(m,j).
// Everything per site runs on the device: the functionals' interpolation
// indices and weights, the dot products with the fields, the 2 x 2 inversions
// and the adjoint sources.  Only the grid's coordinates, the sites and the data
// weights go up in one copy, and the scratch stays with the handle.  (Built
// on the host with a linear search per coordinate, a sort of the entries by
// edge and ten allocations, the adjoint sources of 400 sites on 100 x 100 x 60
// cells took 1.97 ms; here 0.19 ms.)  Site azimuths are zero (the reference's
// rotate_Model2Data with zero angles).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include <atomic>

#include "solver.h"

namespace mt3d {

extern std::atomic<long long> g_launch_count;
__host__ __device__ inline cd cd_add(cd a, cd b) { return {a.re + b.re, a.im + b.im}; }
__host__ __device__ inline cd cd_sub(cd a, cd b) { return {a.re - b.re, a.im - b.im}; }

namespace {

// grid coordinates as setup_grid builds them (f90/3D_MT/GridDef.f90:301-394),
// 1-based like the Fortran (index 0 unused)
struct Coords {
    std::vector<double> xE, yE, zE, xC, yC, zC, dx, dy, dz, dX, dY, dZ;
};

Coords make_coords(const std::vector<double> &dx, const std::vector<double> &dy, const std::vector<double> &dz,
                   const std::vector<double> &delX, const std::vector<double> &delY, const std::vector<double> &delZ,
                   int nzAir, const double *origin)
{
    const int nx = (int)dx.size(), ny = (int)dy.size(), nz = (int)dz.size();
    Coords c;
    auto one = [](const std::vector<double> &v) {
        std::vector<double> r(v.size() + 1, 0.0);
        for (size_t i = 0; i < v.size(); i++) r[i + 1] = v[i];
        return r;
    };
    c.dx = one(dx); c.dy = one(dy); c.dz = one(dz);
    c.dX = one(delX); c.dY = one(delY); c.dZ = one(delZ);
    c.xE.assign(nx + 2, 0.0); c.yE.assign(ny + 2, 0.0); c.zE.assign(nz + 2, 0.0);
    c.xC.assign(nx + 1, 0.0); c.yC.assign(ny + 1, 0.0); c.zC.assign(nz + 1, 0.0);
    c.xE[1] = origin[0];
    c.yE[1] = origin[1];
    double cum = 0.0;
    for (int i = 1; i <= nx; i++) { cum += c.dx[i]; c.xE[i + 1] = cum + origin[0]; }
    cum = 0.0;
    for (int i = 1; i <= ny; i++) { cum += c.dy[i]; c.yE[i + 1] = cum + origin[1]; }
    cum = 0.0;
    c.zE[1] = 0.0;
    for (int i = 1; i <= nz; i++) { cum += c.dz[i]; c.zE[i + 1] = cum; }
    const double air = c.zE[nzAir + 1];
    cum = 0.0;
    for (int i = 1; i <= nx; i++) { cum += c.dX[i]; c.xC[i] = cum + origin[0]; }
    cum = 0.0;
    for (int i = 1; i <= ny; i++) { cum += c.dY[i]; c.yC[i] = cum + origin[1]; }
    cum = 0.0;
    for (int i = 1; i <= nz; i++) { cum += c.dZ[i]; c.zC[i] = cum; }
    for (int i = 1; i <= nz; i++) {
        c.zC[i] = c.zC[i] - air + origin[2];
        c.zE[i] = c.zE[i] - air + origin[2];
    }
    c.zE[nz + 1] = c.zE[nz + 1] - air + origin[2];
    return c;
}

// clean (f90/UTILS/utilities.f90:100-114)
__host__ __device__ inline double clean(double x) { return round(x * 1.0e13) / 1.0e13; }

// coordinates of one axis on the device: the nodes (n + 1) and centres (n),
// each as cleaned for the search and as they are
struct Axis {
    int n;
    const double *node, *cnode, *centre, *ccentre;
    const double *d, *del;  // cell widths and node-centred widths
};
struct SiteGrid {
    Axis ax[3];
    int nx, ny, nz;
    double ioi;  // i ISIGN / omega = i ioi
};

// interpolation of one functional (0 Ex, 1 Ey, 2 Bx, 3 By) at a site: along
// each axis the 1-based point before the site (0: none) and the weight of the
// point after it
struct SiteFun {
    int p[3];
    double w[3];
};

// minNode (f90/UTILS/utilities.f90:196-225): points whose cleaned coordinate
// does not exceed x; the coordinates grow, so by bisection
__device__ int min_node(double x, const double *c, int n)
{
    int lo = 0, hi = n;
    while (lo < hi) {
        const int q = (lo + hi) / 2;
        if (c[q] > x) hi = q;
        else lo = q + 1;
    }
    return lo;
}

// E lies on edges: centred along its own axis; B on faces: centred along the
// other two (EinterpSetUp and BinterpSetUp without conductivity weighting)
__device__ SiteFun site_fun(const SiteGrid &g, const double *x, int f)
{
    SiteFun r;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const Axis &A = g.ax[a];
        const bool centred = (a == (f & 1)) == (f < 2);
        const double xc = clean(x[a]);
        const int nmax = centred ? A.n : A.n + 1;
        const int p = centred ? min_node(xc, A.ccentre, A.n) : min_node(xc, A.cnode, A.n + 1);
        r.p[a] = p;
        if (p > 0 && p < nmax) r.w[a] = centred ? (x[a] - A.centre[p - 1]) / A.del[p] : (x[a] - A.node[p - 1]) / A.d[p - 1];
        else r.w[a] = p <= 0 ? 1.0 : 0.0;
    }
    return r;
}

// flat 0-based edge index of 1-based (component, i, j, k); -1 outside the grid
__device__ __forceinline__ int edge_flat(const SiteGrid &g, int c, int i, int j, int k)
{
    const int nx = g.nx, ny = g.ny, nz = g.nz, nXe = nx * (ny + 1) * (nz + 1), nYe = (nx + 1) * ny * (nz + 1);
    i--, j--, k--;
    if (i < 0 || j < 0 || k < 0) return -1;
    if (c == 1) return (i < nx && j <= ny && k <= nz) ? i + nx * (j + (ny + 1) * k) : -1;
    if (c == 2) return (i <= nx && j < ny && k <= nz) ? nXe + i + (nx + 1) * (j + ny * k) : -1;
    return (i <= nx && j <= ny && k < nz) ? nXe + nYe + i + (nx + 1) * (j + (ny + 1) * k) : -1;
}

// Term t of functional f: t = 4 corner + q for B (four edges a face, the
// circulation over the area, times i ioi: BfromESetUp), corner for E; corner =
// 4 n + 2 m + p.  False where the corner has no weight; edge -1 outside the
// grid; the coefficient is re + i im.
__device__ bool site_term(const SiteGrid &g, const SiteFun &s, int f, int t, int &edge, double &re, double &im)
{
    const int corner = f < 2 ? t : t >> 2, n = corner >> 2, m = (corner >> 1) & 1, p = corner & 1;
    const double w = (n ? s.w[0] : 1.0 - s.w[0]) * (m ? s.w[1] : 1.0 - s.w[1]) * (p ? s.w[2] : 1.0 - s.w[2]);
    if (!(w > 0)) return false;
    const int I = s.p[0] + n, J = s.p[1] + m, K = s.p[2] + p;
    if (f < 2) {
        edge = edge_flat(g, f + 1, I, J, K);
        re = w;
        im = 0.0;
        return true;
    }
    re = 0.0;
    im = 0.0;
    edge = -1;
    const int h = f == 2 ? J : I;  // the face's horizontal cell
    if (h < 1 || h > (f == 2 ? g.ny : g.nx) || K < 1 || K > g.nz) return true;
    const double dh = g.ax[f == 2 ? 1 : 0].d[h - 1], dz = g.ax[2].d[K - 1], S = dh * dz;
    const int q = t & 3;
    double c;
    if (f == 2) {
        if (q < 2) {
            edge = edge_flat(g, 2, I, J, K + q);
            c = q ? -dh / S : dh / S;
        } else {
            edge = edge_flat(g, 3, I, J + (q - 2), K);
            c = q == 2 ? -dz / S : dz / S;
        }
    } else {
        if (q < 2) {
            edge = edge_flat(g, 3, I + q, J, K);
            c = q ? -dz / S : dz / S;
        } else {
            edge = edge_flat(g, 1, I, J, K + (q - 2));
            c = q == 2 ? -dh / S : dh / S;
        }
    }
    im = c * w * g.ioi;
    return true;
}
__device__ __forceinline__ int site_terms(int f) { return f < 2 ? 8 : 32; }
constexpr int kSiteTerms = 80;  // of the four functionals

__device__ __forceinline__ cd shfl_cd(cd v, int src)
{
    return {__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src)};
}

}  // namespace

// Four lanes per site, one functional each: the functionals on both
// polarisations, Z and B^-1 (dataResp); with d non-null also the weights of
// the four functionals in the adjoint source of each polarisation k (Lrows +
// LmultT for Full_Impedance, f90/3D_MT/DataFunc.f90:465-869,
// f90/SENS/DataSens.f90:130-225):
//   s_k = sum_ij conj(d_ij) B^-1(k, j) (Le_i - Z_i1 Lbx - Z_i2 Lby)
// err: the first site (+ 1) with an edge outside the grid.
__global__ void __launch_bounds__(64) k_site(SiteGrid g, int nsite, const double *xyz, SiteFun *fun, const double2 *e1,
                                             const double2 *e2, double2 *Z, const double2 *d, double2 *W, unsigned *err)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, f = t & 3;
    const bool live = t >> 2 < nsite;
    const int s = live ? t >> 2 : nsite - 1;  // (every lane takes part in the exchange)
    const SiteFun sf = site_fun(g, xyz + 3 * (size_t)s, f);
    if (live) fun[4 * (size_t)s + f] = sf;
    cd a = {0.0, 0.0}, b = {0.0, 0.0};
    for (int q = 0; q < site_terms(f); q++) {
        int e;
        double re, im;
        if (!site_term(g, sf, f, q, e, re, im)) continue;
        if (e < 0) {
            if (live) atomicMin(err, (unsigned)s + 1u);
            continue;
        }
        const cd c = {re, im};
        const double2 x1 = e1[e], x2 = e2[e];
        a = cd_add(a, cd_mul(c, cd{x1.x, x1.y}));
        b = cd_add(b, cd_mul(c, cd{x2.x, x2.y}));
    }
    __syncwarp();
    cd v[4][2];
    const int l0 = threadIdx.x & 28;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        v[q][0] = shfl_cd(a, l0 + q);
        v[q][1] = shfl_cd(b, l0 + q);
    }
    if (!live) return;
    // EE(i, m) = v[i][m], BB(i, m) = v[2 + i][m]; BB^-1 by Kramer's rule
    const cd det = cd_sub(cd_mul(v[2][0], v[3][1]), cd_mul(v[2][1], v[3][0]));
    cd bi[2][2], z[2][2];
    bi[0][0] = cd_div(v[3][1], det);
    bi[1][1] = cd_div(v[2][0], det);
    bi[0][1] = cd_div(cd{-v[2][1].re, -v[2][1].im}, det);
    bi[1][0] = cd_div(cd{-v[3][0].re, -v[3][0].im}, det);
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            z[i][j] = cd_add(cd_mul(v[i][0], bi[0][j]), cd_mul(v[i][1], bi[1][j]));
            if (Z && f == 2 * i + j) Z[4 * (size_t)s + f] = make_double2(z[i][j].re, z[i][j].im);
        }
    if (!d) return;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        cd w[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const double2 dd = d[4 * (size_t)s + 2 * i + j];
                const cd c = cd_mul(cd{dd.x, -dd.y}, bi[k][j]);  // conj(d_ij) B^-1(k, j)
                w[i] = cd_add(w[i], c);                          // Lex (i = 0) or Ley (i = 1)
                w[2] = cd_sub(w[2], cd_mul(c, z[i][0]));         // Lbx
                w[3] = cd_sub(w[3], cd_mul(c, z[i][1]));         // Lby
            }
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (f == q) W[(4 * (size_t)s + q) * 2 + k] = make_double2(w[q].re, w[q].im);
    }
}

// the adjoint sources cleared, unless a site was refused
__global__ void __launch_bounds__(kThreads) k_site_clear(int nE, double2 *s1, double2 *s2, const unsigned *err)
{
    if (*err != ~0u) return;
    for (int e = blockIdx.x * kThreads + threadIdx.x; e < nE; e += gridDim.x * kThreads)
        s1[e] = s2[e] = make_double2(0, 0);
}

// Adjoint sources.  A block takes one site, a thread one of its terms; the
// thread of the first term with an edge, in the order (site, functional, term),
// adds every site's share of it in that order, the others leave: no atomics
// and no sort, so sources are reproducible.  The search over the other sites
// is a test of three integers each, of order nsite^2 in all: 400 sites a few
// microseconds, 10 000 about two milliseconds.
__global__ void __launch_bounds__(96) k_site_scatter(SiteGrid g, int nsite, const SiteFun *fun, const double2 *W,
                                                     double2 *s1, double2 *s2, const unsigned *err)
{
    constexpr int kTile = 512;
    __shared__ int lo[kTile][3], own[kSiteTerms];
    if (*err != ~0u) return;
    const int s = blockIdx.x, t = threadIdx.x;
    int e = -1;
    if (t < kSiteTerms) {
        const int f = t < 8 ? 0 : t < 16 ? 1 : t < 48 ? 2 : 3, q = t - (f == 0 ? 0 : f == 1 ? 8 : f == 2 ? 16 : 48);
        double re, im;
        if (!site_term(g, fun[4 * (size_t)s + f], f, q, e, re, im)) e = -1;
        own[t] = e;
    }
    __syncthreads();
    bool mine = e >= 0;
    for (int q = 0; q < t && mine; q++) mine = own[q] != e;
    // (i, j, k) of the edge, 1-based
    int i = 0, j = 0, k = 0;
    if (mine) {
        const int nXe = g.nx * (g.ny + 1) * (g.nz + 1), nYe = (g.nx + 1) * g.ny * (g.nz + 1);
        const int c = e < nXe ? 1 : e < nXe + nYe ? 2 : 3;
        const int r = e - (c == 1 ? 0 : c == 2 ? nXe : nXe + nYe), ni = c == 1 ? g.nx : g.nx + 1, nj = c == 2 ? g.ny : g.ny + 1;
        i = r % ni + 1;
        j = r / ni % nj + 1;
        k = r / (ni * nj) + 1;
    }
    cd a = {0, 0}, b = {0, 0};
    for (int s0 = 0; s0 < nsite; s0 += kTile) {
        // a site's edges lie within three of its smallest indices: its points
        // differ by at most one between the functionals, a corner and a face's
        // far side add one each
        __syncthreads();
        for (int q = t; q < min(kTile, nsite - s0); q += blockDim.x)
            for (int x = 0; x < 3; x++) {
                const SiteFun *F = fun + 4 * (size_t)(s0 + q);
                lo[q][x] = min(min(F[0].p[x], F[1].p[x]), min(F[2].p[x], F[3].p[x]));
            }
        __syncthreads();
        for (int q = 0; q < min(kTile, nsite - s0) && mine; q++) {
            if ((unsigned)(i - lo[q][0]) > 3u || (unsigned)(j - lo[q][1]) > 3u || (unsigned)(k - lo[q][2]) > 3u) continue;
            const int r = s0 + q;
            for (int f = 0; f < 4 && mine; f++) {
                const SiteFun sf = fun[4 * (size_t)r + f];
                for (int u = 0; u < site_terms(f); u++) {
                    int ee;
                    double re, im;
                    if (!site_term(g, sf, f, u, ee, re, im) || ee != e) continue;
                    if (r < s) {  // an earlier site has the edge
                        mine = false;
                        break;
                    }
                    const double2 w0 = W[(4 * (size_t)r + f) * 2], w1 = W[(4 * (size_t)r + f) * 2 + 1];
                    a = cd_add(a, cd_mul(cd{re, im}, cd{w0.x, w0.y}));
                    b = cd_add(b, cd_mul(cd{re, im}, cd{w1.x, w1.y}));
                }
            }
        }
    }
    if (!mine) return;
    s1[e] = make_double2(a.re, a.im);
    s2[e] = make_double2(b.re, b.im);
}

int Solver::impedance(double om, int nsite, const double *xyz, const double *origin, const double *e1,
                      const double *e2, double *Zout, bool device)
{
    return data_functional(om, nsite, xyz, origin, e1, e2, nullptr, Zout, nullptr, nullptr, device);
}

int Solver::lmult_t(double om, int nsite, const double *xyz, const double *origin, const double *e1, const double *e2,
                    const double *d, double *s1, double *s2, bool device)
{
    if (!d || !s1 || !s2) return fail(5, "mt3d_lmult_t: invalid arguments");
    return data_functional(om, nsite, xyz, origin, e1, e2, d, nullptr, s1, s2, device);
}

int Solver::data_functional(double om, int nsite, const double *xyz, const double *origin, const double *e1,
                            const double *e2, const double *d, double *Zout, double *s1, double *s2, bool device)
{
    const char *who = d ? "mt3d_lmult_t" : "mt3d_impedance";
    if (nsite < 1 || !xyz || !origin || !e1 || !e2 || !(om > 0) || !std::isfinite(om) || (!d && !Zout))
        return fail(5, std::string(who) + ": invalid arguments");
    for (int q = 0; q < 3 * nsite; q++)
        if (!std::isfinite(xyz[q])) return fail(5, std::string(who) + ": site coordinates must be finite");
    const Coords c = make_coords(dx_, dy_, dz_, delX_, delY_, delZ_, nzAir, origin);
    // one copy up: the coordinates of the axes, the sites and the data weights
    const std::vector<double> *nodes[3] = {&c.xE, &c.yE, &c.zE}, *centres[3] = {&c.xC, &c.yC, &c.zC};
    const int n[3] = {nx, ny, nz};
    std::vector<double> up;
    size_t at[3][4];
    for (int a = 0; a < 3; a++) {
        const auto put = [&](const std::vector<double> &v, int m, bool cl) {
            const size_t o = up.size();
            for (int q = 1; q <= m; q++) up.push_back(cl ? clean(v[q]) : v[q]);
            return o;
        };
        at[a][0] = put(*nodes[a], n[a] + 1, false);
        at[a][1] = put(*nodes[a], n[a] + 1, true);
        at[a][2] = put(*centres[a], n[a], false);
        at[a][3] = put(*centres[a], n[a], true);
    }
    if (up.size() & 1) up.push_back(0.0);  // the weights are read as 16-byte pairs
    const size_t od = up.size();
    if (d) up.insert(up.end(), d, d + 8 * (size_t)nsite);
    const size_t ox = up.size();
    up.insert(up.end(), xyz, xyz + 3 * (size_t)nsite);
    // scratch of the handle: those, the functionals, W, Z and the error word
    const size_t eb = (size_t)nE * sizeof(double2), ns = (size_t)nsite;
    const auto align = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t b0 = align(up.size() * sizeof(double)), b1 = align(4 * ns * sizeof(SiteFun)),
                 b2 = align(8 * ns * sizeof(double2)), b3 = align(4 * ns * sizeof(double2));
    DevBuf de1, de2, ds1, ds2;
    if (site_.alloc(b0 + b1 + b2 + b3 + sizeof(unsigned)) || (!device && (de1.alloc(eb) || de2.alloc(eb))) ||
        (!device && d && (ds1.alloc(eb) || ds2.alloc(eb))))
        return fail(8, std::string(who) + ": out of device memory");
    unsigned char *base = site_.as<unsigned char>();
    const double *tab = reinterpret_cast<const double *>(base);
    SiteFun *fun = reinterpret_cast<SiteFun *>(base + b0);
    double2 *W = reinterpret_cast<double2 *>(base + b0 + b1), *dz = reinterpret_cast<double2 *>(base + b0 + b1 + b2);
    unsigned *err = reinterpret_cast<unsigned *>(base + b0 + b1 + b2 + b3);
    cudaMemcpyAsync(base, up.data(), up.size() * sizeof(double), cudaMemcpyHostToDevice, stream_);
    cudaMemsetAsync(err, 0xff, sizeof(unsigned), stream_);
    SiteGrid g;
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    g.ioi = -1.0 / om;  // i * ISIGN / omega, ISIGN = -1
    const double *dw[3] = {g64_.dx, g64_.dy, g64_.dz}, *del[3] = {g64_.delX, g64_.delY, g64_.delZ};
    for (int a = 0; a < 3; a++)
        g.ax[a] = Axis{n[a], tab + at[a][0], tab + at[a][1], tab + at[a][2], tab + at[a][3], dw[a], del[a]};
    const double2 *p1 = reinterpret_cast<const double2 *>(e1), *p2 = reinterpret_cast<const double2 *>(e2);
    if (!device) {
        cudaMemcpyAsync(de1.as<void>(), e1, eb, cudaMemcpyHostToDevice, stream_);
        cudaMemcpyAsync(de2.as<void>(), e2, eb, cudaMemcpyHostToDevice, stream_);
        p1 = de1.as<double2>();
        p2 = de2.as<double2>();
    }
    g_launch_count.fetch_add(d ? 3 : 1, std::memory_order_relaxed);
    k_site<<<(4 * nsite + 63) / 64, 64, 0, stream_>>>(g, nsite, tab + ox, fun, p1, p2, Zout ? dz : nullptr,
                                                      d ? reinterpret_cast<const double2 *>(tab + od) : nullptr,
                                                      d ? W : nullptr, err);
    double2 *q1 = nullptr, *q2 = nullptr;
    if (d) {
        q1 = device ? reinterpret_cast<double2 *>(s1) : ds1.as<double2>();
        q2 = device ? reinterpret_cast<double2 *>(s2) : ds2.as<double2>();
        k_site_clear<<<148 * 8, kThreads, 0, stream_>>>((int)nE, q1, q2, err);
        k_site_scatter<<<nsite, 96, 0, stream_>>>(g, nsite, fun, W, q1, q2, err);
    }
    // impedances and the error word, which follow one another, in one copy down
    const size_t bz = Zout ? b3 : 0;
    std::vector<unsigned char> down(bz + sizeof(unsigned));
    cudaMemcpyAsync(down.data(), reinterpret_cast<unsigned char *>(err) - bz, down.size(), cudaMemcpyDeviceToHost, stream_);
    if (int rc = sync(who)) return rc;
    unsigned bad;
    std::memcpy(&bad, down.data() + bz, sizeof bad);
    if (bad != ~0u) return fail(5, std::string(who) + ": site " + std::to_string(bad - 1) + " needs an edge outside the grid");
    if (Zout) std::memcpy(Zout, down.data(), 4 * ns * sizeof(double2));
    if (!d || device) return 0;
    cudaMemcpyAsync(s1, q1, eb, cudaMemcpyDeviceToHost, stream_);
    cudaMemcpyAsync(s2, q2, eb, cudaMemcpyDeviceToHost, stream_);
    return sync(who);
}

}  // namespace mt3d
