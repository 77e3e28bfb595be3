// bc2d.cu -- boundary conditions and first guess of the 3-D forward problem
// from 2-D TE solutions on the slices of the model (BC_x0_WS,
// f90/3D_MT/FWD/boundary_ws.f90:21-168, through ComputeBC,
// f90/3D_MT/FWD/modelOperator3D.f90:268-293).
//
// imode = 2: one 2-D problem per x-slice (horizontal axis y), field on the
// x-edges; imode = 1: one per y-slice (horizontal axis x), field on the
// y-edges.  Per slice (nh horizontal cells, nz vertical cells, air on top):
//   k_bc1d    the 1-D TE columns of SetBound2D_TE (Fwd1D_TE,
//             f90/3D_MT/FWD/Mod2d/WSfwd1Dmod.f90:70-126): both side columns
//             in full and, for every interior column, the bottom value of the
//             column with the area-averaged conductivity; one thread per
//             column, tridiagonal elimination (the 1-D matrix is diagonally
//             dominant, so no pivoting is needed);
//   k_bc_coef the operator coefficients and right-hand side per unknown;
//   the 2-D TE system of SetupA_TE / FormAII / MulAibWithXb / Fwd2DsolveTE
//             (WSfwd2Dmod.f90:32-127, 325-418; FwdTEmod.f90:104-157):
//             (nh-1)(nz-1) interior nodes, complex symmetric and column
//             diagonally dominant (the off-diagonal entries are real and sum
//             to minus the real part of the diagonal), so elimination without
//             row exchanges is stable; the reference's LAPACK band LU agrees
//             with it to rounding.  In one of two ways:
//   k_bc_sweep, k_bc_subst   when the shorter axis of the slices has at most
//             kBcMaxM interior nodes: block elimination of the grid's lines
//             with the running Schur complement held in registers;
//   k_bc2d, k_bc_back   longer slices: band elimination with the active
//             (m+1) x (m+1) window, m = nz-1, in shared memory or, where it
//             does not fit, in global memory as a circular buffer; each step
//             writes the finished row of U out and loads the one new row and
//             column of A, which no earlier step has touched.
// The output is the full edge vector E0 with the tangential field of the
// bottom face zero (boundary_ws.f90:155-156): its boundary entries are the
// BC, its interior entries the first guess.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>

#include "kernels.h"
#include "solver.h"

namespace mt3d {

extern std::atomic<long long> g_launch_count;

namespace {

__device__ __forceinline__ double2 c2(double re, double im) { return make_double2(re, im); }
__device__ __forceinline__ double2 cm(double2 a, double2 b)
{
    return c2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a / b by Smith's algorithm
__device__ __forceinline__ double2 cdv(double2 a, double2 b)
{
    if (fabs(b.x) >= fabs(b.y)) {
        const double r = b.y / b.x, den = b.x + b.y * r;
        return c2((a.x + a.y * r) / den, (a.y - a.x * r) / den);
    }
    const double r = b.x / b.y, den = b.x * r + b.y;
    return c2((a.x * r + a.y) / den, (a.y * r - a.x) / den);
}

// 1 / x for x and 1 / x normal: one step of the hyperpower iteration of order
// three (M. Altman, Pacific J. Math. 10, 1960), y (1 + e + e^2) with e = 1 - x y,
// from the approximate reciprocal y of the PTX instruction.  That reads the upper
// 32 bits of x, 20 of them mantissa, and returns 20 bits of mantissa (PTX ISA,
// rcp.approx.ftz.f64): |e| <= 2^-19.  What is dropped, e^3, is at most 2^-57, an
// eighth of the last bit's half; with the last rounding the result is within one
// unit in the last place of the rounded 1 / x.  Three dependent operations after
// the instruction, where a division has some ten.
__device__ __forceinline__ double rcp_fast(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
// 1 / z for any z: conj(z) / |z|^2 where |z|^2 is far from over- and underflow,
// as with all but absurd frequencies and cell sizes, Smith's algorithm otherwise
// (out of line)
// |z|^2 in 2^-960 .. 2^960 (so not a NaN): by its exponent, off the FP64 pipe
__device__ __forceinline__ bool square_ok(double n)
{
    return (unsigned)__double2hiint(n) - ((1023u - 960u) << 20) < (2u * 960u) << 20;
}
__device__ __noinline__ double2 crcp_far(double2 z) { return cdv(c2(1.0, 0.0), z); }
__device__ __forceinline__ double2 crcp(double2 z)
{
    const double n = fma(z.x, z.x, z.y * z.y);
    if (!square_ok(n)) return crcp_far(z);
    const double iv = rcp_fast(n);
    return c2(z.x * iv, -z.y * iv);
}

struct Slice {
    const BcArgs &a;
    int s;
    __device__ Slice(const BcArgs &a_, int s_) : a(a_), s(s_) {}
    // conductivity of cell (h, k) of the slice, the air at SIGMA_AIR
    __device__ double ccon(int h, int k) const
    {
        if (k < a.nza) return kSigmaAir;
        const long long c = a.imode == 2 ? s + (long long)a.nx * (h + (long long)a.ny * k)
                                         : h + (long long)a.nx * (s + (long long)a.ny * k);
        return a.sigC[c];
    }
    // flat edge index of node (h, k) of the slice
    __device__ long long edge(int h, int k) const
    {
        return a.imode == 2 ? s + (long long)a.nx * (h + (long long)(a.ny + 1) * k)
                            : a.nXe + h + (long long)(a.nx + 1) * (s + (long long)a.ny * k);
    }
};

}  // namespace

// 1-D TE columns.  Thread (slice, col): col 0 and col nh are the side
// columns (cells 0 and nh-1), solved in full into side[slice][0 / 1][0..nz];
// 1 <= col < nh averages cells col-1 and col and keeps the bottom node only.
__global__ void k_bc1d(BcArgs a)
{
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)a.nslice * (a.nh + 1)) return;
    const int s = (int)(t / (a.nh + 1)), col = (int)(t % (a.nh + 1));
    const Slice sl(a, s);
    const int nz = a.nz;
    const int side = col == 0 ? 0 : (col == a.nh ? 1 : -1);
    auto s1d = [&](int k) -> double {
        if (k < a.nza) return kSigmaAir;
        if (col == 0) return sl.ccon(0, k);
        if (col == a.nh) return sl.ccon(a.nh - 1, k);
        return (sl.ccon(col - 1, k) * a.dh[col - 1] + sl.ccon(col, k) * a.dh[col]) / (a.dh[col - 1] + a.dh[col]);
    };
    const double sb = s1d(nz - 1);
    const double skd = sqrt(2.0 / (sb * a.omue));
    auto dz1 = [&](int k) -> double { return k < nz ? a.dz[k] : skd; };
    auto s1 = [&](int k) -> double { return k < nz ? s1d(k) : sb; };
    double2 *cp = side >= 0 ? a.cpr + ((size_t)s * 2 + side) * nz : nullptr;
    double2 *xs = side >= 0 ? a.side + ((size_t)s * 2 + side) * (nz + 1) : nullptr;
    // row j: ad_{j-1} x_{j-1} + ac_j x_j + ad_j x_{j+1} = r_j, r_0 = -au_0
    // the conductivities and widths of kAhead rows are read ahead of the chain,
    // whose step is one complex reciprocal: 40 us for the columns of 40^3
    // cells, 107 us for 200 x 200 x 100, against 56 and 172 us with the loads
    // and six divisions a row on the chain
    constexpr int kAhead = 8;
    double2 cprev = c2(0, 0), dprev = c2(0, 0);
    double adprev = 0.0, sk = s1(0), dk = dz1(0), au = 2.0 / dk;
    for (int j0 = 0; j0 < nz; j0 += kAhead) {
        double sn[kAhead], dn[kAhead], an[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; q++) {
            sn[q] = s1(min(j0 + q + 1, nz));
            dn[q] = dz1(min(j0 + q + 1, nz));
        }
#pragma unroll
        for (int q = 0; q < kAhead; q++) an[q] = 2.0 / dn[q];
#pragma unroll
        for (int q = 0; q < kAhead; q++) {
            const int j = j0 + q;
            if (j >= nz) break;
            const double ad = an[q], ss = sn[q] * dn[q] + sk * dk;
            const double2 den = c2(-au - ad - adprev * cprev.x, a.omue * ss - adprev * cprev.y);
            const double2 id = crcp(den);
            const double2 r = c2((j == 0 ? -au : 0.0) - adprev * dprev.x, -adprev * dprev.y);
            cprev = c2(ad * id.x, ad * id.y);
            dprev = cm(r, id);
            if (side >= 0) {
                cp[j] = cprev;
                xs[j + 1] = dprev;
            }
            adprev = au = ad;
            sk = sn[q];
            dk = dn[q];
        }
    }
    if (side < 0) {
        a.bottom[(size_t)s * (a.nh + 1) + col] = dprev;  // x at the bottom node = last d'
        return;
    }
    xs[0] = c2(1.0, 0.0);
    double2 xn = dprev;
    for (int j0 = nz - 2; j0 >= 0; j0 -= kAhead) {
        double2 d[kAhead], c[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; q++) {
            const int j = max(j0 - q, 0);
            d[q] = xs[j + 1];
            c[q] = cp[j];
        }
#pragma unroll
        for (int q = 0; q < kAhead; q++) {
            if (j0 - q < 0) break;
            xn = c2(d[q].x - (c[q].x * xn.x - c[q].y * xn.y), d[q].y - (c[q].x * xn.y + c[q].y * xn.x));
            xs[j0 - q + 1] = xn;
        }
    }
}

namespace {
// 2-D operator of one slice: unknown r <-> node (iy, iz) = (r / m + 1, r % m + 1)
struct Op2d {
    const BcArgs &a;
    const Slice &sl;
    int m, n;
    __device__ Op2d(const BcArgs &a_, const Slice &sl_) : a(a_), sl(sl_), m(a_.nz - 1), n((a_.nh - 1) * (a_.nz - 1)) {}
    __device__ double cz(int iz) const { return a.dz[iz] + a.dz[iz - 1]; }
    __device__ double cy(int iy) const { return a.dh[iy] + a.dh[iy - 1]; }
    __device__ double2 diag(int r) const
    {
        const int iy = r / m + 1, iz = r % m + 1;
        const double s00 = sl.ccon(iy, iz), s10 = sl.ccon(iy, iz - 1), s01 = sl.ccon(iy - 1, iz),
                     s11 = sl.ccon(iy - 1, iz - 1);
        const double dzi = a.dz[iz], dzm = a.dz[iz - 1], dyi = a.dh[iy], dym = a.dh[iy - 1];
        const double s2d = (s00 * dzi * dyi + s01 * dzi * dym + s10 * dzm * dyi + s11 * dzm * dym) /
                           (dzi * dyi + dzi * dym + dzm * dyi + dzm * dym);
        const double czv = cz(iz), cyv = cy(iy);
        const double ar = 2.0 * czv / dyi, al = 2.0 * czv / dym, ad = 2.0 * cyv / dzi, au = 2.0 * cyv / dzm;
        return c2(-ar - al - ad - au, a.omue * (cyv * czv * s2d));
    }
    // A(r, r+1): vertical neighbour, none below the last interior row
    __device__ double zc(int r) const
    {
        const int iy = r / m + 1, iz = r % m + 1;
        return iz == m ? 0.0 : 2.0 * cy(iy) / a.dz[iz];
    }
    // A(r, r+m): horizontal neighbour, none right of the last interior column
    __device__ double yc(int r) const
    {
        const int iy = r / m + 1, iz = r % m + 1;
        return iy == a.nh - 1 ? 0.0 : 2.0 * cz(iz) / a.dh[iy];
    }
    __device__ double2 at(int r, int c) const
    {
        if (r >= n || c >= n) return c2(0, 0);
        const int d = c - r;
        if (d == 0) return diag(r);
        if (d == 1) return c2(zc(r), 0);
        if (d == -1) return c2(zc(c), 0);
        if (d == m) return c2(yc(r), 0);
        if (d == -m) return c2(yc(c), 0);
        return c2(0, 0);
    }
    // -A_ib x_b (MulAibWithXb)
    __device__ double2 rhs(int r, const double2 *left, const double2 *right, const double2 *bottom) const
    {
        if (r >= n) return c2(0, 0);
        const int iy = r / m + 1, iz = r % m + 1;
        double2 v = c2(0, 0);
        if (iy == 1) {
            const double b = 2.0 * cz(iz) / a.dh[0];
            v = c2(-(b * left[iz].x), -(b * left[iz].y));
        }
        if (iy == a.nh - 1) {
            const double b = 2.0 * cz(iz) / a.dh[a.nh - 1];
            v = c2(-(b * right[iz].x), -(b * right[iz].y));
        }
        if (iz == 1) v.x -= 2.0 * cy(iy) / a.dz[0];
        if (iz == m) {
            const double b = 2.0 * cy(iy) / a.dz[a.nz - 1];
            v = c2(v.x - b * bottom[iy].x, v.y - b * bottom[iy].y);
        }
        return v;
    }
};
}  // namespace

// Coefficients of the 2-D operators and right-hand sides of the slices of a
// launch chunk, one thread per unknown: the diagonal, the couplings to the
// next unknown of its line and to the same unknown of the next line, and
// -A_ib x_b, so that the elimination reads them instead of forming them on its
// critical path.  Lines are the slice's columns (unknown iz of column iy at
// iy m + iz) or, with a.rows, its rows.
__global__ void k_bc_coef(BcArgs a, int nslices)
{
    const int m = a.nz - 1, n = (a.nh - 1) * m;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)nslices * n) return;
    const int q = (int)(t / n), u = (int)(t % n), s = a.slice0 + q;
    const Slice sl(a, s);
    const Op2d op(a, sl);
    const int nl = a.nh - 1;  // unknowns of a row
    const int r = a.rows ? (u % nl) * m + u / nl : u;
    const double2 *left = a.side + (size_t)s * 2 * (a.nz + 1), *right = left + (a.nz + 1);
    const double2 *bottom = a.bottom + (size_t)s * (a.nh + 1);
    a.cd[t] = op.diag(r);
    a.czc[t] = a.rows ? op.yc(r) : op.zc(r);
    a.cyc[t] = a.rows ? op.zc(r) : op.yc(r);
    a.cb[t] = op.rhs(r, left, right, bottom);
}

// ---------------------------------------------------------------------------
// Block elimination of one slice.  The unknowns are n lines of m (m the
// shorter way); line q couples to line q + 1 through the diagonal matrix C_q
// (real), so eliminating the lines from one end leaves the Schur complements
//   S_q = D_q - C_{q-1} S_{q-1}^-1 C_{q-1},  f_q = b_q - C_{q-1} y_{q-1},
//   y_q = S_q^-1 f_q.
// Both ends are eliminated at once, by two thread blocks that meet in the
// middle line, which halves the serial chain and gives twice the blocks; then
// x_q = y_q - S_q^-1 C x_{q+1} outwards from the middle.
//
// S stays complex symmetric, so a block holds its lower triangle only: N (N +
// 1) / 2 threads with a 5 x 5 tile each in registers (m <= 100: 210 threads,
// 100 registers of tile), and inverts it in place by the symmetric sweep.
// Panel by panel of 5 pivots P, with R = A_P. and G the swept panel (A_PP^-1
// R, and A_PP^-1 itself in the columns of P):
//   A_ij -= R_Pi^T G_Pj (i, j off P);  A_Pj = G_Pj;  A_PP = -G_PP,
// after which A = -S^-1.  A panel's own sweep is a chain of 5 reciprocals, so
// it runs one panel ahead in warps of its own: while the tile threads apply
// panel k, the panel warps apply it to the 5 rows of panel k + 1, which the
// tile threads published one panel before, and sweep them.  The right-hand
// side rides along as one more column of the panels.
//
// Bound by FP64 arithmetic for long lines (half of m^3 complex multiply-adds
// a line) and by the panels' chains for short ones.  One polarisation, against
// the band elimination of k_bc2d (a pivot at a time, two block barriers and
// the whole window through shared memory for each): 200 x 200 x 100 cells 18.4
// against 208.4 ms, 101 x 83 x 61 1.67 against 17.8 ms, 40^3 0.38 against
// 4.66 ms.  (8 x 8 blocks in FP64 matrix instructions, which run at the same
// rate, were slower: 20.6 to 27.9 ms for the first.)  The error against dense 64-bit solves is the same (2e-14).
// ---------------------------------------------------------------------------
constexpr int kBcT = 5;                  // tile edge and panel width
// tiles along a line: 210 threads with a tile each and 4 panel warps, at 168
// registers, take 59 of an SM's 64 thousand; a longer line would need two tiles a
// thread or a second SM
constexpr int kBcMaxN = 20;
constexpr int kBcMaxM = kBcT * kBcMaxN;  // longest line
constexpr int kBcOwn = 32 - kBcT;        // columns of a panel per panel warp; the other lanes hold the pivots'
constexpr int kBcMaxThreads = 352;
// up to 60 unknowns a line two blocks fit on an SM, whose chains overlap
constexpr int kBcPairThreads = 192;

__host__ __device__ constexpr int bc_tiles(int N) { return N * (N + 1) / 2; }
__host__ __device__ constexpr int bc_tile_warps(int N) { return (bc_tiles(N) + 31) / 32; }
__host__ __device__ constexpr int bc_panel_warps(int N) { return (kBcT * N + 1 + kBcOwn - 1) / kBcOwn; }
__host__ __device__ constexpr int bc_sweep_threads(int N) { return 32 * (bc_tile_warps(N) + bc_panel_warps(N)); }
static_assert(bc_sweep_threads(kBcMaxN) <= kBcMaxThreads, "threads of the longest lines");
// shared memory in double2: R, G and the published entries of two panels, f
// twice, the diagonal, and (doubles) the coupling within the line and to the
// two sides
__host__ __device__ constexpr size_t bc_sweep_smem(int N)
{
    return (4 * (size_t)kBcT * (kBcT * N + 1) + 2 * (size_t)kBcT * kBcT * N + 3 * (size_t)kBcT * N) * 16 +
           3 * (size_t)kBcT * N * 8;
}

namespace {
// tile t of the lower triangle -> (row, column) of tiles
__device__ __forceinline__ void bc_tile_of(int t, int &ty, int &tx)
{
    ty = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
    while (ty * (ty + 1) / 2 > t) ty--;
    while ((ty + 1) * (ty + 2) / 2 <= t) ty++;
    tx = t - ty * (ty + 1) / 2;
}
__device__ __forceinline__ double2 shfl2(double2 v, int src)
{
    return c2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
__device__ __forceinline__ void cms(double2 &a, double2 b, double2 c)  // a -= b c
{
    a.x = fma(-b.x, c.x, fma(b.y, c.y, a.x));
    a.y = fma(-b.x, c.y, fma(-b.y, c.x, a.y));
}
}  // namespace

// mid: the middle line of every slice, from the lines on its two sides;
// otherwise block 2 s + side eliminates side `side` of slice s
template <bool mid, int threads, int blocks> __global__ void __launch_bounds__(threads, blocks) k_bc_sweep(BcArgs a)
{
    extern __shared__ double2 sm[];
    constexpr int T = kBcT;
    const int N = a.N, MP = T * N, MA = MP + 1, m = a.m, n = a.n, NT = bc_tiles(N);
    double2 *Rb = sm, *Gb = Rb + 2 * T * MA, *Qb = Gb + 2 * T * MA, *f = Qb + 2 * T * MP, *dg = f + 2 * MP;
    double *cs = reinterpret_cast<double *>(dg + MP), *cs2 = cs + MP, *zc = cs2 + MP;
    const int sl = mid ? blockIdx.x : blockIdx.x >> 1, side = mid ? 0 : blockIdx.x & 1;
    const int cm_ = n / 2;  // the middle line
    const int steps = mid ? 1 : side ? n - 1 - cm_ : cm_;
    if (steps == 0) return;
    const size_t base = (size_t)sl * n * m;
    const double2 *cd = a.cd + base, *cb = a.cb + base;
    const double *cin = a.czc + base, *cout = a.cyc + base;
    double2 *inv = a.inv + (size_t)sl * n * T * T * NT, *y = a.y + base;
    const int tw = bc_tile_warps(N) * 32, tid = threadIdx.x;
    const bool panel = tid >= tw, live = tid < NT;
    const int pt = tid - tw, pw = pt >> 5, lane = tid & 31;
    const bool mine = panel && pt < MP;  // the panel thread of unknown pt
    int ty = 0, tx = 0;
    if (live) bc_tile_of(tid, ty, tx);
    auto line = [&](int st) { return mid ? cm_ : side ? n - 1 - st : st; };

    // coefficients of unknown pt of a line; unknowns past m are an identity
    struct Col {
        double2 d, b;
        double z, c, c2;
    };
    auto load = [&](int q, bool prev) {
        Col v{c2(1, 0), c2(0, 0), 0, 0, 0};
        if (pt < m) {
            v.d = cd[(size_t)q * m + pt];
            v.b = cb[(size_t)q * m + pt];
            v.z = cin[(size_t)q * m + pt];
            if (mid || prev) v.c = cout[(size_t)(mid || !side ? q - 1 : q) * m + pt];
            if (mid && q + 1 < n) v.c2 = cout[(size_t)q * m + pt];
        }
        return v;
    };
    Col nx{};
    if (mine) {
        nx = load(line(0), false);
        if (mid && pt < m) {
            const double2 yl = y[(size_t)(cm_ - 1) * m + pt];
            nx.b = c2(nx.b.x - nx.c * yl.x, nx.b.y - nx.c * yl.y);
            if (cm_ + 1 < n) {
                const double2 yr = y[(size_t)(cm_ + 1) * m + pt];
                nx.b = c2(nx.b.x - nx.c2 * yr.x, nx.b.y - nx.c2 * yr.y);
            }
        }
        f[pt] = nx.b;
        dg[pt] = nx.d;
        zc[pt] = nx.z;
        cs[pt] = nx.c;
        cs2[pt] = nx.c2;
    }
    __syncthreads();

    // the block's barrier, reached by the two roles at places of their own
    auto all_sync = [&]() {
        __syncwarp();
        asm volatile("bar.sync 0;" ::: "memory");
    };

    if (panel) {
        // R and G of panel k from the published entries, panel k - 1 applied first
        const int own = pw * kBcOwn + lane;
        const bool dup = lane >= kBcOwn, ok = dup || own <= MP;
        // far: pivots inverted without squares where those over- or underflow.
        // Otherwise false when one did, in all lanes and warps alike; nothing that a
        // second go reads has changed then.  A test and a branch at every pivot
        // made 200 x 200 x 100 cells 2.2 % slower than none, the tests alone and a
        // branch a panel 1.3 %
        auto sweep_as = [&](int k, auto far) {
            const int P = k * T, K = P - T, col = dup ? P + lane - kBcOwn : own;
            const double2 *R = Rb + ((k - 1) & 1) * T * MA, *G = Gb + ((k - 1) & 1) * T * MA;
            double2 *Rn = Rb + (k & 1) * T * MA, *Gn = Gb + (k & 1) * T * MA;
            const double2 *Q = Qb + (k & 1) * T * MP, *fo = f + (k > 0 ? ((k - 1) & 1) * MP : 0);
            double2 v[T];
#pragma unroll
            for (int r = 0; r < T; r++) v[r] = !ok ? c2(0, 0) : col == MP ? fo[P + r] : Q[r * MP + col];
            if (k > 0 && ok) {
                if (col >= K && col < P) {
#pragma unroll
                    for (int r = 0; r < T; r++) v[r] = G[(col - K) * MA + P + r];
                } else {
#pragma unroll
                    for (int p = 0; p < T; p++) {
                        const double2 g = G[p * MA + col];
#pragma unroll
                        for (int r = 0; r < T; r++) cms(v[r], R[p * MA + P + r], g);
                    }
                }
            }
            if (!dup && ok)
#pragma unroll
                for (int r = 0; r < T; r++) Rn[r * MA + col] = v[r];
            bool ok_sq = true;
#pragma unroll
            for (int p = 0; p < T; p++) {
                double2 l[T];
#pragma unroll
                for (int r = 0; r < T; r++) l[r] = shfl2(v[r], kBcOwn + p);
                double2 iv;
                if constexpr (far.value) {
                    iv = crcp(l[p]);
                } else {
                    const double n2 = fma(l[p].x, l[p].x, l[p].y * l[p].y), den = rcp_fast(n2);
                    iv = c2(l[p].x * den, -l[p].y * den);
                    ok_sq = ok_sq && square_ok(n2);
                }
                const bool pc = col == P + p;
                const double2 g = pc ? iv : cm(v[p], iv);
#pragma unroll
                for (int r = 0; r < T; r++) {
                    if (r == p) continue;
                    if (pc) v[r] = c2(0, 0);
                    cms(v[r], l[r], g);
                }
                v[p] = g;
            }
            if (!dup && ok)
#pragma unroll
                for (int r = 0; r < T; r++) Gn[r * MA + col] = v[r];
            return ok_sq;
        };
        auto sweep = [&](int k) {
            if (!sweep_as(k, std::false_type{})) sweep_as(k, std::true_type{});
        };
        for (int st = 0; st < steps; st++) {
            const bool more = st + 1 < steps;
            if (mine && more) nx = load(line(st + 1), true);
            all_sync();  // panels 0 and 1 are published
            sweep(0);
            all_sync();
            for (int k = 0; k < N; k++) {
                const double2 *R = Rb + (k & 1) * T * MA, *G = Gb + (k & 1) * T * MA;
                const int P = k * T;
                if (mine) {  // the right-hand side
                    double2 v = f[(k & 1) * MP + pt];
                    if (pt >= P && pt < P + T) v = G[(pt - P) * MA + MP];
                    else
#pragma unroll
                        for (int p = 0; p < T; p++) cms(v, R[p * MA + pt], G[p * MA + MP]);
                    f[((k + 1) & 1) * MP + pt] = v;
                }
                if (k + 1 < N) sweep(k + 1);
                all_sync();
            }
            if (mine) {  // f = y; the next line's coefficients
                const double2 v = f[(N & 1) * MP + pt];
                if (pt < m) y[(size_t)line(st) * m + pt] = v;
                if (more) {
                    f[pt] = c2(nx.b.x - nx.c * v.x, nx.b.y - nx.c * v.y);
                    dg[pt] = nx.d;
                    zc[pt] = nx.z;
                    cs[pt] = nx.c;
                }
            }
            all_sync();
        }
        return;
    }

    double2 A[T][T];
    auto publish = [&](int k) {  // panel k's entries as they stand
        double2 *Q = Qb + (k & 1) * T * MP;
        if (live && k < N) {
            if (ty == k) {
#pragma unroll
                for (int i = 0; i < T; i++)
#pragma unroll
                    for (int j = 0; j < T; j++) Q[i * MP + tx * T + j] = A[i][j];
            } else if (tx == k) {
#pragma unroll
                for (int i = 0; i < T; i++)
#pragma unroll
                    for (int j = 0; j < T; j++) Q[j * MP + ty * T + i] = A[i][j];
            }
        }
    };
    for (int st = 0; st < steps; st++) {
        const int q = line(st);
        if (live) {
#pragma unroll
            for (int i = 0; i < T; i++)
#pragma unroll
                for (int j = 0; j < T; j++) {
                    const int r = ty * T + i, c = tx * T + j;
                    double2 v = c2(0, 0);
                    if (mid) {
                        const size_t e = (size_t)(i * T + j) * NT + tid, ln = (size_t)T * T * NT;
                        const double2 u = inv[(size_t)(q - 1) * ln + e];
                        const double w = cs[r] * cs[c];
                        v = c2(w * u.x, w * u.y);
                        if (q + 1 < n) {
                            const double2 u2 = inv[(size_t)(q + 1) * ln + e];
                            const double w2 = cs2[r] * cs2[c];
                            v = c2(v.x + w2 * u2.x, v.y + w2 * u2.y);
                        }
                    } else if (st) {
                        const double w = cs[r] * cs[c];
                        v = c2(w * A[i][j].x, w * A[i][j].y);
                    }
                    if (r == c) v = c2(v.x + dg[r].x, v.y + dg[r].y);
                    if (r == c + 1) v.x += zc[c];
                    if (c == r + 1) v.x += zc[r];
                    A[i][j] = v;
                }
        }
        publish(0);
        publish(1);
        all_sync();
        all_sync();  // panel 0 is swept
        for (int k = 0; k < N; k++) {
            const double2 *R = Rb + (k & 1) * T * MA, *G = Gb + (k & 1) * T * MA;
            if (live) {
                if (ty != k && tx != k) {
#pragma unroll
                    for (int p = 0; p < T; p++) {
                        double2 g[T];
#pragma unroll
                        for (int j = 0; j < T; j++) g[j] = G[p * MA + tx * T + j];
#pragma unroll
                        for (int i = 0; i < T; i++) {
                            const double2 r = R[p * MA + ty * T + i];
#pragma unroll
                            for (int j = 0; j < T; j++) cms(A[i][j], r, g[j]);
                        }
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < T; i++)
#pragma unroll
                        for (int j = 0; j < T; j++) {
                            const double2 v = ty == k ? G[i * MA + tx * T + j] : G[j * MA + ty * T + i];
                            A[i][j] = ty == tx ? c2(-v.x, -v.y) : v;
                        }
                }
            }
            publish(k + 2);
            all_sync();
        }
        if (live && !mid) {  // A = -S^-1
            double2 *o = inv + (size_t)q * T * T * NT + tid;
#pragma unroll
            for (int i = 0; i < T; i++)
#pragma unroll
                for (int j = 0; j < T; j++) o[(size_t)(i * T + j) * NT] = A[i][j];
        }
        all_sync();
    }
}

// x_q = y_q + A_q (C x_{q -+ 1}) outwards from the middle line, block 2 s +
// side; A_q = -S_q^-1 in tiles as k_bc_sweep left it, read once.  A tile
// serves its rows and, by symmetry, its columns; the partial sums of a row
// are added in the order of the tiles.  Block 2 s also writes the middle line
// and the boundary nodes of E0: side columns, 1 along the top; the bottom row
// stays zero.
__global__ void __launch_bounds__(256) k_bc_subst(BcArgs a)
{
    extern __shared__ double2 sm[];
    constexpr int T = kBcT;
    const int N = a.N, MP = T * N, MA = MP + 1, m = a.m, n = a.n, NT = bc_tiles(N), tid = threadIdx.x;
    double2 *v = sm, *part = sm + MP;
    const int q0 = blockIdx.x >> 1, side = blockIdx.x & 1, s = a.slice0 + q0, cm_ = n / 2;
    const Slice sl(a, s);
    const size_t base = (size_t)q0 * n * m;
    const double2 *y = a.y + base, *inv = a.inv + (size_t)q0 * n * T * T * NT;
    const double *cout = a.cyc + base;
    auto edge = [&](int q, int b) { return a.rows ? sl.edge(b + 1, q + 1) : sl.edge(q + 1, b + 1); };
    if (side == 0) {
        const double2 *left = a.side + (size_t)s * 2 * (a.nz + 1), *right = left + (a.nz + 1);
        for (int k = tid; k < a.nz; k += blockDim.x) {
            a.e0[sl.edge(0, k)] = left[k];
            a.e0[sl.edge(a.nh, k)] = right[k];
        }
        for (int h = 1 + tid; h < a.nh; h += blockDim.x) a.e0[sl.edge(h, 0)] = c2(1.0, 0.0);
        if (tid < m) a.e0[edge(cm_, tid)] = y[(size_t)cm_ * m + tid];
    }
    const int steps = side ? n - 1 - cm_ : cm_;
    if (steps == 0) return;
    const bool live = tid < NT, mine = tid < MP;
    int ty = 0, tx = 0;
    if (live) bc_tile_of(tid, ty, tx);
    auto line = [&](int st) { return side ? cm_ + 1 + st : cm_ - 1 - st; };
    // coupling of line q to its neighbour towards the middle
    auto coup = [&](int q) { return tid < m ? cout[(size_t)(side ? q - 1 : q) * m + tid] : 0.0; };
    double2 A[T][T], yq = c2(0, 0);
    auto load = [&](int q) {
        if (live) {
            const double2 *p = inv + (size_t)q * T * T * NT + tid;
#pragma unroll
            for (int i = 0; i < T; i++)
#pragma unroll
                for (int j = 0; j < T; j++) A[i][j] = p[(size_t)(i * T + j) * NT];
        }
        if (mine && tid < m) yq = y[(size_t)q * m + tid];
    };
    load(line(0));
    if (mine) {
        const double c = coup(line(0));
        const double2 x = tid < m ? y[(size_t)cm_ * m + tid] : c2(0, 0);
        v[tid] = c2(c * x.x, c * x.y);
    }
    __syncthreads();
    for (int st = 0; st < steps; st++) {
        const int q = line(st);
        const bool more = st + 1 < steps;
        if (live) {
            double2 pr[T], pc[T];
#pragma unroll
            for (int i = 0; i < T; i++) pr[i] = pc[i] = c2(0, 0);
#pragma unroll
            for (int i = 0; i < T; i++) {
                const double2 vi = v[ty * T + i];
#pragma unroll
                for (int j = 0; j < T; j++) {
                    const double2 w = A[i][j], vj = v[tx * T + j];
                    pr[i].x += w.x * vj.x - w.y * vj.y;
                    pr[i].y += w.x * vj.y + w.y * vj.x;
                    pc[j].x += w.x * vi.x - w.y * vi.y;
                    pc[j].y += w.x * vi.y + w.y * vi.x;
                }
            }
#pragma unroll
            for (int i = 0; i < T; i++) part[tx * MA + ty * T + i] = pr[i];
            if (ty != tx)
#pragma unroll
                for (int i = 0; i < T; i++) part[ty * MA + tx * T + i] = pc[i];
        }
        const double2 yc = yq;
        if (more) load(line(st + 1));  // ahead of their use
        const double cn = more && mine ? coup(line(st + 1)) : 0.0;
        __syncthreads();
        if (mine) {
            double2 x = yc;
            for (int t = 0; t < N; t++) {
                const double2 p = part[t * MA + tid];
                x = c2(x.x + p.x, x.y + p.y);
            }
            if (tid < m) a.e0[edge(q, tid)] = x;
            v[tid] = c2(cn * x.x, cn * x.y);
        }
        __syncthreads();
    }
}

// One block (32 x BY threads) per slice of the launch chunk.
__global__ void __launch_bounds__(1024) k_bc2d(BcArgs a, int smem_window)
{
    extern __shared__ double2 sm[];
    const int s = a.slice0 + blockIdx.x;
    const Slice sl(a, s);
    const Op2d op(a, sl);
    const int m = op.m, n = op.n, M = m + 1;
    double2 *W = smem_window ? sm : a.W + (size_t)blockIdx.x * M * M;
    double2 *rw = smem_window ? sm + (size_t)M * M : sm;  // right-hand side window
    double2 *U = a.U + (size_t)blockIdx.x * n * M;
    double2 *y = a.y + (size_t)blockIdx.x * n;
    const double2 *left = a.side + (size_t)s * 2 * (a.nz + 1), *right = left + (a.nz + 1);
    const double2 *bottom = a.bottom + (size_t)s * (a.nh + 1);
    const int tx = threadIdx.x, ty = threadIdx.y, nt = blockDim.x * blockDim.y, tid = ty * blockDim.x + tx;
    const double2 *cd = a.cd + (size_t)blockIdx.x * n, *cb = a.cb + (size_t)blockIdx.x * n;
    const double *czc = a.czc + (size_t)blockIdx.x * n, *cyc = a.cyc + (size_t)blockIdx.x * n;
    // A(r, c) of the slice from the coefficient arrays
    auto at = [&](int r, int c) -> double2 {
        if (r >= n || c >= n) return c2(0, 0);
        const int d = c - r;
        if (d == 0) return cd[r];
        if (d == 1) return c2(czc[r], 0);
        if (d == -1) return c2(czc[c], 0);
        if (d == m) return c2(cyc[r], 0);
        if (d == -m) return c2(cyc[c], 0);
        return c2(0, 0);
    };

    // boundary nodes of E0: side columns, 1 along the top; the bottom row stays zero
    for (int k = tid; k < a.nz; k += nt) {
        a.e0[sl.edge(0, k)] = left[k];
        a.e0[sl.edge(a.nh, k)] = right[k];
    }
    for (int h = 1 + tid; h < a.nh; h += nt) a.e0[sl.edge(h, 0)] = c2(1.0, 0.0);

    // window of step 0: rows and columns 0..m
    for (int q = tid; q < M * M; q += nt) {
        const int r = q / M, c = q % M;
        W[r * M + c] = at(r, c);
    }
    for (int r = tid; r < M; r += nt) rw[r] = r < n ? cb[r] : c2(0, 0);
    __syncthreads();

    for (int j = 0; j < n; j++) {
        const int s0 = j % M;
        // the row and column rn = j + M that enter at the end of this step hold
        // three nonzeros, A(rn, rn) and the symmetric pairs A(rn - 1, rn),
        // A(rn - m, rn); their loads are issued here, ahead of their use
        const int rn = j + M;
        const bool newrow = rn < n;
        const double2 nd = newrow ? cd[rn] : c2(0, 0), nb = newrow ? cb[rn] : c2(0, 0);
        const double nz1 = newrow ? czc[rn - 1] : 0.0, nym = newrow ? cyc[rn - m] : 0.0;
        const double2 piv = W[s0 * M + s0];
        const double2 rp = cdv(c2(1.0, 0.0), piv);
        // rows j+a, columns j+b, a, b = 1..m
        if (m <= 4 * (int)blockDim.y) {
            // up to four rows per thread: their multipliers in registers, each
            // entry of the pivot row read once per column
            int ras[4];
            double2 ls[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int ai = 1 + ty + q * blockDim.y;
                int ra = s0 + ai;
                if (ra >= M) ra -= M;
                ras[q] = ra;
                ls[q] = ai <= m ? cm(W[ra * M + s0], rp) : c2(0, 0);
            }
            for (int bi = 1 + tx; bi <= m; bi += blockDim.x) {
                int cb = s0 + bi;
                if (cb >= M) cb -= M;
                const double2 u = W[s0 * M + cb];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const double2 l = ls[q];
                    if (l.x == 0.0 && l.y == 0.0) continue;
                    double2 w = W[ras[q] * M + cb];
                    w.x -= l.x * u.x - l.y * u.y;
                    w.y -= l.x * u.y + l.y * u.x;
                    W[ras[q] * M + cb] = w;
                }
            }
            if (tx == 0) {
                const double2 r0 = rw[s0];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const double2 l = ls[q];
                    if (l.x == 0.0 && l.y == 0.0) continue;
                    double2 w = rw[ras[q]];
                    w.x -= l.x * r0.x - l.y * r0.y;
                    w.y -= l.x * r0.y + l.y * r0.x;
                    rw[ras[q]] = w;
                }
            }
        } else {
            for (int ai = 1 + ty; ai <= m; ai += blockDim.y) {
                int ra = s0 + ai;
                if (ra >= M) ra -= M;
                const double2 l = cm(W[ra * M + s0], rp);
                if (l.x == 0.0 && l.y == 0.0) continue;
                for (int bi = 1 + tx; bi <= m; bi += blockDim.x) {
                    int cb = s0 + bi;
                    if (cb >= M) cb -= M;
                    const double2 u = W[s0 * M + cb];
                    double2 w = W[ra * M + cb];
                    w.x -= l.x * u.x - l.y * u.y;
                    w.y -= l.x * u.y + l.y * u.x;
                    W[ra * M + cb] = w;
                }
                if (tx == 0) {
                    const double2 r0 = rw[s0];
                    double2 w = rw[ra];
                    w.x -= l.x * r0.x - l.y * r0.y;
                    w.y -= l.x * r0.y + l.y * r0.x;
                    rw[ra] = w;
                }
            }
        }
        // the finished row of U and of the reduced right-hand side
        for (int bi = tid; bi < M; bi += nt) {
            int cb = s0 + bi;
            if (cb >= M) cb -= M;
            U[(size_t)j * M + bi] = W[s0 * M + cb];
        }
        if (tid == 0) y[j] = rw[s0];
        __syncthreads();
        // slot s0 now takes row rn (columns j+1..j+M) and column rn (rows
        // j+1..j+M-1): column j+1 = rn - m, column rn - 1 and the diagonal
        for (int bi = 1 + tid; bi <= M; bi += nt) {
            int cb = s0 + bi;
            if (cb >= M) cb -= M;
            W[s0 * M + cb] = bi == M ? nd : c2(bi == 1 ? nym : bi == M - 1 ? nz1 : 0.0, 0.0);
        }
        for (int ai = 1 + tid; ai < M; ai += nt) {
            int ra = s0 + ai;
            if (ra >= M) ra -= M;
            W[ra * M + s0] = c2(ai == 1 ? nym : ai == M - 1 ? nz1 : 0.0, 0.0);
        }
        if (tid == 0) rw[s0] = nb;
        __syncthreads();
    }
}

// Back substitution, one warp per slice: x_j = (y_j - sum_b U[j][b] x_{j+b}) /
// U[j][0] from j = n-1 down.  Each lane holds up to kBackP entries of a U row
// (columns lane + 32 p), and the row of step j - 1 is loaded while step j is
// reduced, so the chain waits on shuffles and not on memory.  The last M
// values of x live in shared memory as a circular buffer.
constexpr int kBackP = 8;
__global__ void __launch_bounds__(32) k_bc_back(BcArgs a)
{
    extern __shared__ double2 xs[];
    const int q = blockIdx.x, s = a.slice0 + q;
    const int m = a.nz - 1, n = (a.nh - 1) * m, M = a.nz;
    const Slice sl(a, s);
    const double2 *U = a.U + (size_t)q * n * M, *y = a.y + (size_t)q * n;
    const int tx = threadIdx.x;
    double2 u[kBackP], un[kBackP];
    auto load = [&](int j, double2 *dst) {
#pragma unroll
        for (int p = 0; p < kBackP; p++) {
            const int bi = tx + 32 * p;
            dst[p] = bi < M ? U[(size_t)j * M + bi] : c2(0, 0);
        }
    };
    load(n - 1, u);
    double2 yj = y[n - 1];
    for (int j = n - 1; j >= 0; j--) {
        double2 yn = c2(0, 0);
        if (j > 0) {
            load(j - 1, un);
            yn = y[j - 1];
        }
        double2 acc = c2(0, 0);
#pragma unroll
        for (int p = 0; p < kBackP; p++) {
            const int bi = tx + 32 * p;
            if (bi >= 1 && bi < M && j + bi < n) {
                const double2 xv = xs[(j + bi) % M];
                acc.x += u[p].x * xv.x - u[p].y * xv.y;
                acc.y += u[p].x * xv.y + u[p].y * xv.x;
            }
        }
        for (int bi = tx + 32 * kBackP; bi < M && j + bi < n; bi += 32) {  // rows longer than 32 kBackP
            const double2 uv = U[(size_t)j * M + bi], xv = xs[(j + bi) % M];
            acc.x += uv.x * xv.x - uv.y * xv.y;
            acc.y += uv.x * xv.y + uv.y * xv.x;
        }
        for (int o = 16; o > 0; o >>= 1) {
            acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
            acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
        }
        const double2 dg = c2(__shfl_sync(0xffffffffu, u[0].x, 0), __shfl_sync(0xffffffffu, u[0].y, 0));
        const double2 xj = cdv(c2(yj.x - acc.x, yj.y - acc.y), dg);
        __syncwarp();
        if (tx == 0) {
            xs[j % M] = xj;
            a.e0[sl.edge(j / m + 1, j % m + 1)] = xj;
        }
        __syncwarp();
#pragma unroll
        for (int p = 0; p < kBackP; p++) u[p] = un[p];
        yj = yn;
    }
}

size_t bc_smem_bytes(int nz, bool window_in_smem)
{
    const size_t M = (size_t)nz;
    return (window_in_smem ? M * M + M : M) * sizeof(double2);
}

void launch_bc_coef(const BcArgs &a, int nslices, cudaStream_t s)
{
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    const long long nt = (long long)nslices * (a.nh - 1) * (a.nz - 1);
    k_bc_coef<<<(unsigned)((nt + 255) / 256), 256, 0, s>>>(a, nslices);
}

void launch_bc_back(const BcArgs &a, int nslices, cudaStream_t s)
{
    const size_t smem = (size_t)a.nz * sizeof(double2);
    if (smem > 48 * 1024) cudaFuncSetAttribute(k_bc_back, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    k_bc_back<<<nslices, 32, smem, s>>>(a);
}

void launch_bc1d(const BcArgs &a, cudaStream_t s)
{
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    const long long nt = (long long)a.nslice * (a.nh + 1);
    // (one warp a block: a small grid's columns spread over more SMs)
    k_bc1d<<<(unsigned)((nt + 31) / 32), 32, 0, s>>>(a);
}

static size_t bc_subst_smem(int N) { return ((size_t)kBcT * N + (size_t)N * (kBcT * N + 1)) * sizeof(double2); }

template <int threads, int blocks> static void bc_sweep_launch(const BcArgs &a, int nslices, cudaStream_t s)
{
    const int th = bc_sweep_threads(a.N);
    const size_t sm = bc_sweep_smem(a.N);
    if (sm > 48 * 1024) {
        cudaFuncSetAttribute(k_bc_sweep<false, threads, blocks>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        cudaFuncSetAttribute(k_bc_sweep<true, threads, blocks>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    }
    k_bc_sweep<false, threads, blocks><<<2 * nslices, th, sm, s>>>(a);
    k_bc_sweep<true, threads, blocks><<<nslices, th, sm, s>>>(a);
}

// the three launches of the block elimination
void launch_bc_lines(const BcArgs &a, int nslices, cudaStream_t s)
{
    g_launch_count.fetch_add(3, std::memory_order_relaxed);
    if (bc_sweep_threads(a.N) <= kBcPairThreads) bc_sweep_launch<kBcPairThreads, 2>(a, nslices, s);
    else bc_sweep_launch<kBcMaxThreads, 1>(a, nslices, s);
    const int tb = std::max(32 * bc_tile_warps(a.N), (kBcT * a.N + 31) / 32 * 32);
    k_bc_subst<<<2 * nslices, tb, bc_subst_smem(a.N), s>>>(a);
}

int launch_bc2d(const BcArgs &a, int nblocks, bool window_in_smem, cudaStream_t s)
{
    const size_t smem = bc_smem_bytes(a.nz, window_in_smem);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_bc2d, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    const int m = a.nz - 1;
    const dim3 block(32, m >= 64 ? 32 : 16);
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    k_bc2d<<<nblocks, block, smem, s>>>(a, window_in_smem ? 1 : 0);
    return (int)cudaGetLastError();
}

// the elimination's reciprocals as they stand: y = 1 / Re z, w = 1 / z
__global__ void __launch_bounds__(256) k_bc_reciprocal(int n, const double2 *z, double *y, double2 *w)
{
    const int t = blockIdx.x * 256 + threadIdx.x;
    if (t >= n) return;
    y[t] = rcp_fast(z[t].x);
    w[t] = crcp(z[t]);
}

int Solver::check_reciprocal(int n, const double *z, double *y, double *w)
{
    const char *who = "mt3d_check_reciprocal";
    if (n < 1 || !z || !y || !w) return fail(5, std::string(who) + ": invalid arguments");
    const size_t b = (size_t)n * sizeof(double);
    DevBuf dz, dy, dw;
    if (dz.alloc(2 * b) || dy.alloc(b) || dw.alloc(2 * b)) return fail(8, std::string(who) + ": out of device memory");
    cudaMemcpyAsync(dz.as<void>(), z, 2 * b, cudaMemcpyHostToDevice, stream_);
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    k_bc_reciprocal<<<(unsigned)(((long long)n + 255) / 256), 256, 0, stream_>>>(n, dz.as<double2>(), dy.as<double>(),
                                                                                 dw.as<double2>());
    cudaMemcpyAsync(y, dy.as<void>(), b, cudaMemcpyDeviceToHost, stream_);
    cudaMemcpyAsync(w, dw.as<void>(), 2 * b, cudaMemcpyDeviceToHost, stream_);
    return sync(who);
}

// ---------------------------------------------------------------------------
// host side (ComputeBC)
// ---------------------------------------------------------------------------
int Solver::compute_bc(int imode, double om, double *e0, bool device)
{
    if (!cond_set) return fail(5, "mt3d_compute_bc: conductivity not set (call mt3d_update_cond)");
    if ((imode != 1 && imode != 2) || !e0 || !(om > 0) || !std::isfinite(om))
        return fail(5, "mt3d_compute_bc: invalid arguments");
    const int nh = imode == 2 ? ny : nx, nslice = imode == 2 ? nx : ny;
    if (nh < 3 || nz < 3) return fail(5, "mt3d_compute_bc: the slices need at least 3 x 3 cells");
    const int64_t nC = (int64_t)nx * ny * nz, nEarth = (int64_t)nx * ny * (nz - nzAir);
    const int m = nz - 1, M = nz;
    const int64_t n = (int64_t)(nh - 1) * m;
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev_);
    // the block elimination where its lines, along the shorter axis, fit in
    // registers (10 to 11 times the band elimination's speed at 39, 60 and 99
    // unknowns a line); its work grows with the cube of their length
    const bool rows = nh < nz;
    const int lm = rows ? nh - 1 : m, ln = rows ? m : nh - 1;
    const bool lines = lm <= kBcMaxM;
    const int N = (lm + kBcT - 1) / kBcT;
    const bool smem = lines || bc_smem_bytes(nz, true) <= (size_t)optin;
    // per slice: U rows (n x M) or the tiles of the lines' inverses, reduced
    // right-hand side (n), diagonal (n), operator right-hand side (n), the two
    // couplings (2n doubles = n double2), the window when it is neither in
    // registers nor in shared memory (M x M)
    const size_t fact = lines ? (size_t)ln * kBcT * kBcT * bc_tiles(N) : (size_t)n * M;
    const size_t per_slice = (fact + 4 * (size_t)n + (smem ? 0 : (size_t)M * M)) * sizeof(double2);
    const size_t cap = (size_t)8 << 30;
    const int chunk = (int)std::max<size_t>(1, std::min<size_t>(nslice, cap / per_slice));
    const size_t fixed = ((size_t)nslice * 2 * (nz + 1) + (size_t)nslice * 2 * nz + (size_t)nslice * (nh + 1));
    if (bcs_.alloc(fixed * sizeof(double2) + (size_t)chunk * per_slice) || (!device && bce_.alloc(nE * sizeof(double2))))
        return fail(8, "mt3d_compute_bc: out of device memory");
    BcArgs a{};
    a.imode = imode;
    a.nh = nh;
    a.nz = nz;
    a.nza = nzAir;
    a.nslice = nslice;
    a.nx = nx;
    a.ny = ny;
    a.nXe = g64_.nXe;
    // the 2-D code receives the period 2 pi / omega and forms 2 pi / period
    const double per = (2.0 * kPiRef) / om;
    a.omue = ((2.0 * kPiRef) / per) * kMu0;
    a.dh = imode == 2 ? g64_.dy : g64_.dx;
    a.dz = g64_.dz;
    a.sigC = setup_.as<double>() + nEarth + 2 * nC;
    double2 *p = bcs_.as<double2>();
    a.side = p; p += (size_t)nslice * 2 * (nz + 1);
    a.cpr = p; p += (size_t)nslice * 2 * nz;
    a.bottom = p; p += (size_t)nslice * (nh + 1);
    a.rows = lines && rows;
    a.m = lm;
    a.n = ln;
    a.N = N;
    a.U = a.inv = p; p += (size_t)chunk * fact;
    a.y = p; p += (size_t)chunk * n;
    a.cd = p; p += (size_t)chunk * n;
    a.cb = p; p += (size_t)chunk * n;
    a.czc = reinterpret_cast<double *>(p);
    a.cyc = a.czc + (size_t)chunk * n;
    p += (size_t)chunk * n;
    a.W = smem ? nullptr : p;
    a.e0 = device ? reinterpret_cast<double2 *>(e0) : bce_.as<double2>();
    int rc;
    if ((rc = check(cudaMemsetAsync(a.e0, 0, nE * sizeof(double2), stream_), "mt3d_compute_bc"))) return rc;
    launch_bc1d(a, stream_);
    for (int s0 = 0; s0 < nslice; s0 += chunk) {
        a.slice0 = s0;
        launch_bc_coef(a, std::min(chunk, nslice - s0), stream_);
        if (lines) {
            launch_bc_lines(a, std::min(chunk, nslice - s0), stream_);
            continue;
        }
        if ((rc = check((cudaError_t)launch_bc2d(a, std::min(chunk, nslice - s0), smem, stream_), "mt3d_compute_bc")))
            return rc;
        launch_bc_back(a, std::min(chunk, nslice - s0), stream_);
    }
    if ((rc = check(cudaGetLastError(), "mt3d_compute_bc"))) return rc;
    if (!device &&
        (rc = check(cudaMemcpyAsync(e0, a.e0, nE * sizeof(double2), cudaMemcpyDeviceToHost, stream_), "copy E0")))
        return rc;
    return sync("mt3d_compute_bc");
}

}  // namespace mt3d
