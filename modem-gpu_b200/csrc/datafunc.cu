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
// cells took 1.97 ms; here 0.09 ms.)  Site azimuths are zero (the reference's
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

// Point before the site along axis a and the weight of the point after it.  E
// lies on edges: centred along its own axis; B on faces: centred along the
// other two (EinterpSetUp and BinterpSetUp without conductivity weighting)
__device__ void site_axis(const SiteGrid &g, const double *x, int f, int a, int &p, double &w)
{
    const Axis &A = g.ax[a];
    const bool centred = (a == (f & 1)) == (f < 2);
    const double xc = clean(x[a]);
    const int nmax = centred ? A.n : A.n + 1;
    p = min_node(xc, centred ? A.ccentre : A.cnode, nmax);
    if (p > 0 && p < nmax) w = centred ? (x[a] - A.centre[p - 1]) / A.del[p] : (x[a] - A.node[p - 1]) / A.d[p - 1];
    else w = p <= 0 ? 1.0 : 0.0;
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
// The terms of functional f that edge (c, i, j, k) can be: its one corner of E,
// the two faces it bounds of B, in ascending order.
__device__ int edge_terms(const SiteFun &s, int f, int c, int i, int j, int k, int (&t)[2])
{
    const auto corner = [&](int I, int J, int K) {
        const unsigned n = I - s.p[0], m = J - s.p[1], p = K - s.p[2];
        return (n | m | p) > 1u ? -1 : (int)(4 * n + 2 * m + p);
    };
    int nt = 0;
    if (f < 2) {
        const int q = c == f + 1 ? corner(i, j, k) : -1;
        if (q >= 0) t[nt++] = q;
        return nt;
    }
    if (c == f - 1) return 0;  // Ex is on no x-face, Ey on no y-face
    // the edge as the far side of the face before it, and as the near side
    const bool vert = c == 3;
    const int lo = !vert ? corner(i, j, k - 1) : f == 2 ? corner(i, j - 1, k) : corner(i - 1, j, k), hi = corner(i, j, k);
    const int q = (f == 2) == vert ? 2 : 0;  // its pair of the face's four edges
    if (lo >= 0) t[nt++] = 4 * lo + q + 1;
    if (hi >= 0) t[nt++] = 4 * hi + q;
    return nt;
}
__device__ __forceinline__ int site_terms(int f) { return f < 2 ? 8 : 32; }
__device__ __forceinline__ int site_base(int f) { return f < 2 ? 8 * f : 32 * f - 48; }  // the terms before them
constexpr int kSiteTerms = 80, kSiteBlock = 96;  // of the four functionals; threads for them

}  // namespace

// A warp per site.  Twelve lanes search the axes of the four functionals, then
// the lanes take the terms of one functional after another and add them up in
// a fixed tree: the functionals on both polarisations, Z and B^-1 (dataResp);
// with d non-null also the weights of the four functionals in the adjoint
// source of each polarisation k (Lrows + LmultT for Full_Impedance,
// f90/3D_MT/DataFunc.f90:465-869, f90/SENS/DataSens.f90:130-225):
//   s_k = sum_ij conj(d_ij) B^-1(k, j) (Le_i - Z_i1 Lbx - Z_i2 Lby)
// err: the first site (+ 1) with an edge outside the grid.  Bound by the
// latency of the searches and gathers: 14 us for 400 sites; 34 us with four
// lanes a site and its terms one after another.
__global__ void __launch_bounds__(64) k_site(SiteGrid g, int nsite, const double *xyz, SiteFun *fun, int *lo,
                                             const double2 *e1, const double2 *e2, double2 *Z, const double2 *d, double2 *W,
                                             unsigned *err)
{
    const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (s >= nsite) return;
    int p = 0;
    double w = 0.0;
    if (lane < 12) site_axis(g, xyz + 3 * (size_t)s, lane / 3, lane % 3, p, w);
    // the smallest of the functionals' points along each axis
    int low = p;
    for (int f = 1; f < 4; f++) low = min(low, __shfl_sync(0xffffffffu, p, (lane + 3 * f) % 12));
    if (lane < 3) lo[3 * (size_t)s + lane] = low;
    cd v[4][2];
#pragma unroll
    for (int f = 0; f < 4; f++) {
        SiteFun sf;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            sf.p[a] = __shfl_sync(0xffffffffu, p, 3 * f + a);
            sf.w[a] = __shfl_sync(0xffffffffu, w, 3 * f + a);
        }
        if (lane == f) fun[4 * (size_t)s + f] = sf;
        double t[4] = {0.0, 0.0, 0.0, 0.0};
        int e;
        double re, im;
        if (lane < site_terms(f) && site_term(g, sf, f, lane, e, re, im)) {
            if (e < 0) {
                atomicMin(err, (unsigned)s + 1u);
            } else {
                const double2 x1 = e1[e], x2 = e2[e];
                const cd a = cd_mul(cd{re, im}, cd{x1.x, x1.y}), b = cd_mul(cd{re, im}, cd{x2.x, x2.y});
                t[0] = a.re;
                t[1] = a.im;
                t[2] = b.re;
                t[3] = b.im;
            }
        }
        __syncwarp();
        warp_sum<4>(t);
        v[f][0] = {t[0], t[1]};
        v[f][1] = {t[2], t[3]};
    }
    if (lane >= 4) return;
    const int f = lane;
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
// and no sort, so sources are reproducible.  The block picks the sites nearby,
// a test of three integers for each site by one thread, of order nsite^2 in
// all, and such a site costs the few terms that the edge can be.  (All 80 terms
// of a site tried and the sites tested by every thread: 94 us for 400 sites;
// the few terms alone: 43 us; now 18 us.)
__global__ void __launch_bounds__(kSiteBlock) k_site_scatter(SiteGrid g, int nsite, const SiteFun *fun, const int *lo,
                                                             const double2 *W, double2 *s1, double2 *s2,
                                                             const unsigned *err)
{
    __shared__ int near[kSiteBlock], found[kSiteBlock / 32];
    if (*err != ~0u) return;
    const int s = blockIdx.x, t = threadIdx.x, lane = t & 31, wp = t >> 5;
    int e = -1;
    if (t < kSiteTerms) {
        const int f = t < 8 ? 0 : t < 16 ? 1 : t < 48 ? 2 : 3;
        double re, im;
        if (!site_term(g, fun[4 * (size_t)s + f], f, t - site_base(f), e, re, im)) e = -1;
    }
    bool mine = e >= 0;
    // component and (i, j, k) of the edge, 1-based
    int c = 0, i = 0, j = 0, k = 0;
    if (mine) {
        const int nXe = g.nx * (g.ny + 1) * (g.nz + 1), nYe = (g.nx + 1) * g.ny * (g.nz + 1);
        c = e < nXe ? 1 : e < nXe + nYe ? 2 : 3;
        const int r = e - (c == 1 ? 0 : c == 2 ? nXe : nXe + nYe), ni = c == 1 ? g.nx : g.nx + 1, nj = c == 2 ? g.ny : g.ny + 1;
        i = r % ni + 1;
        j = r / ni % nj + 1;
        k = r / (ni * nj) + 1;
    }
    const int l0 = lo[3 * (size_t)s], l1 = lo[3 * (size_t)s + 1], l2 = lo[3 * (size_t)s + 2];
    cd a = {0, 0}, b = {0, 0};
    for (int r0 = 0; r0 < nsite; r0 += kSiteBlock) {
        // a site's edges lie within three of its smallest indices: its points
        // differ by at most one between the functionals, a corner and a face's
        // far side add one each
        bool hit = false;
        if (r0 + t < nsite) {
            const int *l = lo + 3 * (size_t)(r0 + t);
            hit = abs(l[0] - l0) <= 3 && abs(l[1] - l1) <= 3 && abs(l[2] - l2) <= 3;
        }
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) found[wp] = __popc(hits);
        __syncthreads();
        int at = 0, all = 0;
        for (int q = 0; q < kSiteBlock / 32; q++) {
            at += q < wp ? found[q] : 0;
            all += found[q];
        }
        if (hit) near[at + __popc(hits & ((1u << lane) - 1u))] = r0 + t;
        __syncthreads();
        for (int q = 0; q < all && mine; q++) {
            const int r = near[q];
            for (int f = 0; f < 4 && mine; f++) {
                int can[2];
                const SiteFun sf = fun[4 * (size_t)r + f];
                const int nt = edge_terms(sf, f, c, i, j, k, can);
                for (int u = 0; u < nt; u++) {
                    int ee;
                    double re, im;
                    if (!site_term(g, sf, f, can[u], ee, re, im) || ee != e) continue;
                    if (r < s || (r == s && site_base(f) + can[u] < t)) {  // an earlier site or term has the edge
                        mine = false;
                        break;
                    }
                    const double2 w0 = W[(4 * (size_t)r + f) * 2], w1 = W[(4 * (size_t)r + f) * 2 + 1];
                    a = cd_add(a, cd_mul(cd{re, im}, cd{w0.x, w0.y}));
                    b = cd_add(b, cd_mul(cd{re, im}, cd{w1.x, w1.y}));
                }
            }
        }
        __syncthreads();
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
    // the error word, set to none; the impedances follow it, for one copy down
    if (up.size() & 1) up.push_back(0.0);
    const size_t oe = up.size();
    up.resize(oe + 2);
    std::memset(&up[oe], 0xff, 2 * sizeof(double));
    // scratch of the handle: those, the impedances, the functionals, W and the smallest indices
    const size_t eb = (size_t)nE * sizeof(double2), ns = (size_t)nsite;
    const auto align = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t bz = Zout ? 4 * ns * sizeof(double2) : 0;
    const size_t b0 = align(up.size() * sizeof(double) + bz), b1 = align(4 * ns * sizeof(SiteFun)),
                 b2 = align(d ? 8 * ns * sizeof(double2) : 0), b3 = 3 * ns * sizeof(int);
    DevBuf de1, de2, ds1, ds2;
    if (site_.alloc(b0 + b1 + b2 + b3) || (!device && (de1.alloc(eb) || de2.alloc(eb))) ||
        (!device && d && (ds1.alloc(eb) || ds2.alloc(eb))))
        return fail(8, std::string(who) + ": out of device memory");
    unsigned char *base = site_.as<unsigned char>();
    const double *tab = reinterpret_cast<const double *>(base);
    unsigned *err = reinterpret_cast<unsigned *>(base + oe * sizeof(double));
    double2 *dz = reinterpret_cast<double2 *>(base + up.size() * sizeof(double));
    SiteFun *fun = reinterpret_cast<SiteFun *>(base + b0);
    double2 *W = reinterpret_cast<double2 *>(base + b0 + b1);
    int *lo = reinterpret_cast<int *>(base + b0 + b1 + b2);
    cudaMemcpyAsync(base, up.data(), up.size() * sizeof(double), cudaMemcpyHostToDevice, stream_);
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
    k_site<<<(nsite + 1) / 2, 64, 0, stream_>>>(g, nsite, tab + ox, fun, lo, p1, p2, Zout ? dz : nullptr,
                                                  d ? reinterpret_cast<const double2 *>(tab + od) : nullptr, d ? W : nullptr,
                                                  err);
    double2 *q1 = nullptr, *q2 = nullptr;
    if (d) {
        q1 = device ? reinterpret_cast<double2 *>(s1) : ds1.as<double2>();
        q2 = device ? reinterpret_cast<double2 *>(s2) : ds2.as<double2>();
        k_site_clear<<<148 * 8, kThreads, 0, stream_>>>((int)nE, q1, q2, err);
        k_site_scatter<<<nsite, kSiteBlock, 0, stream_>>>(g, nsite, fun, lo, W, q1, q2, err);
    }
    std::vector<unsigned char> down(2 * sizeof(double) + bz);
    cudaMemcpyAsync(down.data(), err, down.size(), cudaMemcpyDeviceToHost, stream_);
    if (int rc = sync(who)) return rc;
    unsigned bad;
    std::memcpy(&bad, down.data(), sizeof bad);
    if (bad != ~0u) return fail(5, std::string(who) + ": site " + std::to_string(bad - 1) + " needs an edge outside the grid");
    if (Zout) std::memcpy(Zout, down.data() + 2 * sizeof(double), bz);
    if (!d || device) return 0;
    cudaMemcpyAsync(s1, q1, eb, cudaMemcpyDeviceToHost, stream_);
    cudaMemcpyAsync(s2, q2, eb, cudaMemcpyDeviceToHost, stream_);
    return sync(who);
}

}  // namespace mt3d
