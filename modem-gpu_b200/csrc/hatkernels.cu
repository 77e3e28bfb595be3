// hatkernels.cu -- the FP32 BiCGStab iteration of the mixed-precision solve
// with the diagonal preconditioner fused into the operator kernels.
//
// BiCGStab right-preconditioned with D = diag(A) (BICG, f90/3D_MT/FWD/
// solver.f90:346-555, as the unfused kernels run it) is carried in
// preconditioned variables: u = D^-1 p, vh = D^-1 v, rh = D^-1 r,
// sh = D^-1 s, th = D^-1 t.  Then every vector update is a plain axpy, the
// preconditioner is one division at the output edge of the operator kernels
// (vh = D^-1 A u, th = D^-1 A sh), and no vector of D^-1 exists:
//
//   kh_u         u  = rh + beta (u - omega vh)   (u = rh on the first iteration)
//   kh_vt st. 0  vh = D^-1 A u,       (rt, v)                  -> alpha
//   kh_s         sh = rh - alpha vh
//   kh_vt st. 1  th = D^-1 A sh,      (t, s), (t, t), (s, s)   -> omega, ||r||
//   kh_xr        x += alpha u + omega sh,  rh = sh - omega th,  (rt, r) -> beta
//
// 163 bytes per edge and iteration instead of the 211 of the unfused
// kernels (kb_p, kct_vt, kb_s, kct_vt, kb_xr).  With the polynomial
// preconditioner M^-1 = c D^-1 (2 I - c A D^-1) each operator launch becomes
// two (stages 2, 3 and 4, 5 of hat_vt); kh_xr accumulates yhat = sum (alpha
// u + omega sh) as in the diagonal case, and the end of the cycle turns the
// best yhat into x = M^-1 D yhat = c (2 yhat - c D^-1 A yhat) (stage 6 and
// kh_conv).  The inner products of the
// method in the original variables follow from the hat ones:
//   - the shadow residual is the reference's rt = r0 = b; with y =
//     conj(D) b stored once per cycle (written by kh_cast), (rt, r) =
//     sum conj(y) rh and (rt, v) = sum conj(y) vh;
//   - with W = |D|^2 per edge, computed in the operator kernel where D is,
//     (t, s) = sum W conj(th) sh, (t, t) = sum W |th|^2, and the true
//     residual norm of the new iterate follows without another pass:
//     ||s - omega t||^2 = ||s||^2 - 2 Re(conj(omega) (t, s)) + |omega|^2 ||t||^2.
// The iterates, step lengths and residual norms are those of the unfused
// kernels up to rounding.  (A shadow generated from the edge index instead
// of a stored one, rt = D^-H z with z = +-1 +- i, saves 16 bytes an
// iteration, but its entries scale as 1/|D|, which on the benchmark model
// cost 40 % more iterations and on the reference's cylinder model stalled
// the solve.)
//
// The operator kernels stage u or sh with the tensor copies of tma.cuh.  D =
// V_E xXO-diagonal of the curl-curl term + the grad-div diagonal
// DFA^2 (w_s c_s + w_e c_e) + i omega mu0 sigma V_E, from the staged sigma
// and signed node weights (those of a plane are kept in registers from the
// plane before, so the node ring keeps two slots).  kh_cast computes the same D
// from the global tables.
#include <atomic>
#include <cstring>

#include "finalize.cuh"
#include "tma.cuh"

namespace mt3d {

constexpr int kTX = HatTile::TX, kTY = HatTile::TY, kFW = HatTile::FW, kFR = HatTile::FR, kSW = HatTile::SW,
              kNW = HatTile::NW, kPhX = HatTile::PhX;
constexpr unsigned kFBytes = HatTile::FBytes, kSBytes = HatTile::SBytes, kNBytes = HatTile::NBytes;

extern std::atomic<long long> g_launch_count;
// launches go to the process's count, or, while this thread captures them, to
// the graph's (they count as they run, hat_loop_count)
static thread_local long long *t_captured = nullptr;
static inline void counted(int n)
{
    if (t_captured) *t_captured += n;
    else g_launch_count.fetch_add(n, std::memory_order_relaxed);
}

// diagonal dr + i di of A at an interior edge: the curl-curl part p sp + q sq
// (p, q: the weights of the curls beside the edge; sp, sq: the sums of 1 / d of
// the two cells across each), the grad-div part a^2 (w_s c_s + w_e c_e) with a
// the dual face's area and c = sigma at earth nodes (negative weights), one in
// the air, and di = v sigma with v = omega mu0 V_E.  The roundings are written
// out, so that every kernel has the same D.
__device__ __forceinline__ void hat_diag(float p, float sp, float q, float sq, float v, float sig, bool gd, float a,
                                         float ws, float we, float &dr, float &di)
{
    dr = __fmaf_rn(p, sp, __fmul_rn(q, sq));
    if (gd) {
        const float n = __fadd_rn(fmaxf(ws, __fmul_rn(-ws, sig)), fmaxf(we, __fmul_rn(-we, sig)));
        dr = __fmaf_rn(__fmul_rn(a, a), n, dr);
    }
    di = __fmul_rn(v, sig);
}
// what a plane gives a node's edges: the weights of the curls beside Ex, Ey and
// Ez (dxi delZk, dxi delYj; dyj delXi, dyj delZk; dzk delYj, dzk delXi), and the
// areas of their dual faces
struct HatCoef {
    float xz, xy, yx, yz, zy, zx, ax, ay, az;
};
__device__ __forceinline__ HatCoef hat_coef(const ColGeo<float> &c, const PlaneGeo<float> &p)
{
    return {__fmul_rn(c.dxi, p.delZk),   __fmul_rn(c.dxi, c.delYj),   __fmul_rn(c.dyj, c.delXi),
            __fmul_rn(c.dyj, p.delZk),   __fmul_rn(p.dzk, c.delYj),   __fmul_rn(p.dzk, c.delXi),
            __fmul_rn(c.delYj, p.delZk), __fmul_rn(c.delXi, p.delZk), __fmul_rn(c.delXi, c.delYj)};
}
__device__ __forceinline__ void hat_diag_of(int comp, const ColGeo<float> &c, const PlaneGeo<float> &p, const HatCoef &w,
                                            float wmu, float sig, bool gd, float ws, float we, float &dr, float &di)
{
    const float sx = __fadd_rn(c.rdxi, c.rdxim1), sy = __fadd_rn(c.rdyj, c.rdyjm1), sz = __fadd_rn(p.rdzk, p.rdzkm1);
    if (comp == 0) hat_diag(w.xz, sy, w.xy, sz, __fmul_rn(__fmul_rn(wmu, p.delZk), w.xy), sig, gd, w.ax, ws, we, dr, di);
    else if (comp == 1) hat_diag(w.yz, sx, w.yx, sz, __fmul_rn(__fmul_rn(wmu, p.delZk), w.yx), sig, gd, w.ay, ws, we, dr, di);
    else hat_diag(w.zy, sx, w.zx, sy, __fmul_rn(__fmul_rn(wmu, p.dzk), w.az), sig, gd, w.az, ws, we, dr, di);
}

// y / D and |D|^2, both zero unless `in` (the approximate reciprocal: D^-1 only
// has to be the same in every kernel that applies it, which one function
// guarantees)
__device__ __forceinline__ float2 hat_div(float2 y, float dr, float di, bool in, float &W)
{
    W = __fmaf_rn(dr, dr, __fmul_rn(di, di));
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(W));
    inv = in ? inv : 0.f;
    W = in ? W : 0.f;
    return make_float2((y.x * dr + y.y * di) * inv, (y.y * dr - y.x * di) * inv);
}

// ---------------------------------------------------------------------------
// start of an FP32 cycle: rh = D^-1 b with b = r64 scale on the padded
// layout, the shadow y = conj(D) b (rt = b), x = 0; ||b||^2 = rho = (rt, r).
// The first guess is zero, so r = b and no operator pass is needed.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) kh_cast(KArgs<float> a, const double2 *r64, size_t stride64)
{
    const int r = blockIdx.y;
    if (!a.ost[r].active) return;
    const Geo<float> &g = a.g;
    const size_t off = (size_t)r * stride64, offp = (size_t)r * a.stride;
    const double sc = a.ost[r].scale;
    const float wmu = (float)(a.dsgn * a.ost[r].omega * kMu0);
    double u[1] = {0.0};
    for (int e = blockIdx.x * kThreads + threadIdx.x; e < g.nE; e += gridDim.x * kThreads) {
        const EdgeIdx q = edge_decode(g, e);
        const int pe = a.pl.idx(q.c, q.i, q.j, q.k);
        const double2 v = r64[off + e];
        const float2 b = make_float2((float)(v.x * sc), (float)(v.y * sc));
        float2 rh = make_float2(0.f, 0.f), y = rh;
        if (edge_interior(g, q)) {
            const ColGeo<float> cg = col_geo(g, q.i, q.j);
            const PlaneGeo<float> pg = plane_geo(g, q.k);
            float wns = 0.f, wne = 0.f;
            if (a.gd) {
                const int ns = iN(g, q.i, q.j, q.k);
                wns = a.gdn[ns];
                wne = a.gdn[q.c == 0 ? ns + 1 : q.c == 1 ? ns + g.nx + 1 : ns + (g.nx + 1) * (g.ny + 1)];
            }
            float dr, di, W;
            hat_diag_of(q.c, cg, pg, hat_coef(cg, pg), wmu, a.sigma[e], a.gd != 0, wns, wne, dr, di);
            rh = hat_div(b, dr, di, true, W);
            y = make_float2(dr * b.x + di * b.y, dr * b.y - di * b.x);  // conj(D) b
            u[0] += (double)b.x * b.x + (double)b.y * b.y;
        }
        a.r[offp + pe] = rh;
        a.rt[offp + pe] = y;
        a.x0[offp + pe] = make_float2(0.f, 0.f);
    }
    double tot[1];
    if (block_reduce_last<1>(u, a.parts, a.cnt, r, blockIdx.x, gridDim.x, tot) && threadIdx.x == 0) {
        const double t2[2] = {tot[0], tot[0]};
        fin_init(a.st[r], t2, a.rerr + (size_t)r * a.rerr_stride, a.maxit, a.ost[r].tol_inner);
    }
}

// ---------------------------------------------------------------------------
// elementwise kernels (two complex entries per thread and step)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float4 c2mul2(float2 c, float4 v)
{
    return make_float4(c.x * v.x - c.y * v.y, c.x * v.y + c.y * v.x, c.x * v.z - c.y * v.w, c.x * v.w + c.y * v.z);
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 sub4(float4 a, float4 b) { return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w); }

// pairs of entries of block bx of a right-hand side (a.chunk entries per block)
#define HAT_PAIRS(a, bx)                                                             \
    const int hp_n2 = (a).len / 2, hp_c2 = (a).chunk / 2;                            \
    const int q1 = min(((bx) + 1) * hp_c2, hp_n2);                                    \
    for (int q = (bx) * hp_c2 + threadIdx.x; q < q1; q += kThreads)

// u = rh + beta (u - omega vh); u = rh on the first iteration of a cycle or
// after a restart (block bx of right-hand side r)
__device__ __forceinline__ void hat_u(const KArgs<float> &a, int r, int bx)
{
    const BicgState &st = a.st[r];
    if (st.status != KS_RUNNING || !a.ost[r].active) return;
    const size_t off = (size_t)r * a.stride / 2;
    const float4 *RH = reinterpret_cast<const float4 *>(a.r) + off;
    const float4 *VH = reinterpret_cast<const float4 *>(a.v) + off;
    float4 *U = reinterpret_cast<float4 *>(a.ph) + off;
    if (st.first) {
        HAT_PAIRS(a, bx) U[q] = RH[q];
        return;
    }
    const float2 be = make_float2((float)st.beta.re, (float)st.beta.im);
    const float2 om = make_float2((float)st.omega.re, (float)st.omega.im);
    HAT_PAIRS(a, bx) U[q] = add4(RH[q], c2mul2(be, sub4(U[q], c2mul2(om, VH[q]))));
}

// sh = rh - alpha vh
__device__ __forceinline__ void hat_s(const KArgs<float> &a, int r, int bx)
{
    const BicgState &st = a.st[r];
    if (st.status != KS_RUNNING || !a.ost[r].active) return;
    const size_t off = (size_t)r * a.stride / 2;
    const float4 *RH = reinterpret_cast<const float4 *>(a.r) + off;
    const float4 *VH = reinterpret_cast<const float4 *>(a.v) + off;
    float4 *SH = reinterpret_cast<float4 *>(a.sh) + off;
    const float2 al = make_float2((float)st.alpha.re, (float)st.alpha.im);
    HAT_PAIRS(a, bx) SH[q] = sub4(RH[q], c2mul2(al, VH[q]));
}

// x += alpha u + omega sh (into the buffer that does not hold the best
// iterate); rh = sh - omega th; rho = (z, rh).  The true residual norm of the
// new iterate comes from the inner products of kh_vt stage 1 or 5
// (BicgState::rn2).
__device__ __forceinline__ void hat_xr(const KArgs<float> &a, int r, int bx)
{
    BicgState &st = a.st[r];
    if (st.status != KS_RUNNING || !a.ost[r].active) return;
    const size_t off = (size_t)r * a.stride / 2;
    const float2 al = make_float2((float)st.alpha.re, (float)st.alpha.im);
    const float2 om = make_float2((float)st.omega.re, (float)st.omega.im);
    const int cur = st.xcur, dst = (st.xcur == st.xbest) ? 1 - st.xcur : st.xcur;
    const float4 *XS = reinterpret_cast<const float4 *>(cur == 0 ? a.x0 : a.x1) + off;
    float4 *XD = reinterpret_cast<float4 *>(dst == 0 ? a.x0 : a.x1) + off;
    const float4 *U = reinterpret_cast<const float4 *>(a.ph) + off;
    const float4 *SH = reinterpret_cast<const float4 *>(a.sh) + off;
    const float4 *TH = reinterpret_cast<const float4 *>(a.t) + off;
    float4 *RH = reinterpret_cast<float4 *>(a.r) + off;
    const float4 *Y = reinterpret_cast<const float4 *>(a.rt) + off;
    // with the polynomial preconditioner the iterate is x = M^-1 yhat, and
    // yhat = sum (alpha u + omega sh) accumulates here like the diagonal
    // case's x (u = D^-1 p, sh = D^-1 s); launch_hat_conv turns the cycle's
    // best yhat into x = c (2 yhat - c D^-1 A yhat) at its end
    double u[2] = {0.0, 0.0};
    HAT_PAIRS(a, bx)
    {
        const float4 sh = SH[q];
        XD[q] = add4(add4(XS[q], c2mul2(al, U[q])), c2mul2(om, sh));
        const float4 rn = sub4(sh, c2mul2(om, TH[q]));
        RH[q] = rn;
        const float4 y = Y[q];  // conj(y) rh
        u[0] += (double)y.x * rn.x + (double)y.y * rn.y + (double)y.z * rn.z + (double)y.w * rn.w;
        u[1] += (double)y.x * rn.y - (double)y.y * rn.x + (double)y.z * rn.w - (double)y.w * rn.z;
    }
    double tot[2];
    if (block_reduce_last<2>(u, a.parts, a.cnt, r, bx, a.nblk, tot) && threadIdx.x == 0) {
        double *rerr = a.rerr + (size_t)r * a.rerr_stride;
        const double rnorm = sqrt(st.rn2);
        st.iter += 1;
        st.xcur = dst;
        st.first = 0;
        st.rnorm = rnorm;
        rerr[st.iter - 1] = rnorm / st.bnorm;
        if (!isfinite(rnorm) || !isfinite(tot[0]) || !isfinite(tot[1])) { st.status = KS_NAN; return; }
        if (rnorm < st.btol) {
            st.status = KS_CONVERGED;
            st.xbest = dst;
            return;
        }
        if (rnorm < st.rnormin) {
            st.rnormin = rnorm;
            st.xbest = dst;
            st.imin = st.iter;
        }
        if (st.iter >= st.maxit) {
            st.status = KS_MAXIT;
            return;
        }
        const cd rho_new = {tot[0], tot[1]};
        if (a.restart > 0 && st.iter % a.restart == 0) {
            // restart towards steepest descent (cuBiCG, f90/3D_MT/FWD_SP2/
            // solver.f90:1545-1573): rt = r, rho = (rt, r) = ||r||^2, p = r,
            // omega = 1; the next kh_vt stage 0 or 2 writes the new shadow y = W rh
            st.first = 1;
            st.pad = 1;
            st.rho = {st.rn2, 0.0};
            st.omega = {1.0, 0.0};
            if (cd_zero(st.rho)) st.status = KS_BREAKDOWN;
            return;
        }
        st.rho1 = st.rho;
        st.rho = rho_new;
        if (cd_zero(st.rho)) { st.status = KS_BREAKDOWN; return; }
        st.beta = cd_mul(cd_div(st.rho, st.rho1), cd_div(st.alpha, st.omega));
        if (cd_zero(st.beta)) st.status = KS_BREAKDOWN;
    }
}

// ---------------------------------------------------------------------------
// the operator kernels: the staged stencil of tmakernels.cu with the output
// divided by D at the edge
// ---------------------------------------------------------------------------

// an entry read once, left out of the L1 cache (28 KB beside the ring), where the
// plane tables stay
__device__ __forceinline__ float2 load_once(const float2 *p)
{
    float2 v;
    asm volatile("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}

// grad-div potential of a node, |w| sum of C_e DFA_e x_e over its edges (k_gd_phi
// mode 0), from the fields before and after it along each axis; S and Sz are at
// its sigma in the planes of the node and below it.  Nodes on the boundary have
// the weight zero, and so the potential
__device__ __forceinline__ float2 hat_phi(float wn, float2 xm, float2 x, float2 ym, float2 y, float2 zm, float2 z,
                                          const float *S, const float *Sz, float dX, float dY, float dZ)
{
    constexpr int SW = HatTile::SW, cs = HatTile::FR * SW;
    const bool earth = wn < 0.f;  // C = sigma_E, or one at air nodes
    const auto c = [&](float sig) { return earth ? sig : 1.f; };
    const float2 u = csub(cscale(xm, c(S[-1])), cscale(x, c(S[0])));
    const float2 v = csub(cscale(ym, c(S[cs - SW])), cscale(y, c(S[cs])));
    const float2 w = csub(cscale(zm, c(Sz[2 * cs])), cscale(z, c(S[2 * cs])));
    return cscale(cadd(cadd(cscale(u, dY * dZ), cscale(v, dX * dZ)), cscale(w, dX * dY)), fabsf(wn));
}
// a (after - before) - b (after - before) of two pairs: a curl's component
__device__ __forceinline__ float2 hat_curl(float2 p1, float2 p0, float a, float2 q1, float2 q0, float b)
{
    return csub(cscale(csub(p1, p0), a), cscale(csub(q1, q0), b));
}

// March planes [k0, k1) of tile (i0, j0), right-hand side r, calling
// f(e, yhat, x_e, W, aux_e) for the three edge slots (Ex, Ey, Ez) of every
// node of the thread's two columns, padding slots included: yhat =
// D^-1 (A x)_e and W = |D_e|^2 at interior edges (zero otherwise), e the
// padded index, aux_e the entry of the vector aux (read one plane ahead,
// zero without has_aux).  A thread (tx, ty) of the 128 takes the node columns
// (i0 + tx, j0 + 2 ty) and (i0 + tx, j0 + 2 ty + 1), so the per-plane work of a thread
// (waits, barriers, plane geometry, loop control) is shared by six edges, the
// columns share their row's fields, and the register budget of four blocks per
// SM is 128 per thread.  Returns false (all threads of the block alike) when a
// wait gave up.
//
// curl curl is taken in two steps, as it is defined: the curl on the faces
// after a node,
//   Hx = dEz/dy - dEy/dz,  Hy = dEx/dz - dEz/dx,  Hz = dEy/dx - dEx/dy,
// once for the four edges around each face, then the curl of that on the
// edges times V_E.  The faces below a node come from its own previous plane,
// those before it along x from the lane before (or the tile's halo column),
// along y from the thread's own pair or from the row published in shared
// memory.  The kernel is bound by instruction issue.  With every edge forming its
// eight differences anew (60 complex operations a node for the curls, here 24;
// 30 reads of staged fields, here 21 for two nodes), the diagonal's products
// formed edge by edge and the potentials behind tests, a launch took on average
// over the four of an iteration, in us: 40^3, 8 right-hand sides 25.6, now 23.1;
// 64 x 64 x 48, 8: 61, now 52.8; 100 x 100 x 60, 2: 43.6, now 36.4; 200 x 200 x
// 100, 1: 111, now 92; 4: 376, now 311.  Of that the plane tables in registers
// give 2 % (they fell out of the L1 cache, 28 KB beside the ring, and were
// waited for on every plane), and the pairs of rows four apart 2 to 3 %.
template <bool gd, bool has_aux, typename F>
__device__ __forceinline__ bool hat_march(HatTile::Smem &sm, const TmaParams &tp, const Geo<float> &g, PadLayout pl, int r,
                                          const float2 *__restrict__ aux, float wmu, int i0, int j0, int k0, int k1,
                                          int *err, int limit, F &&f)
{
    const int tx = threadIdx.x % kTX, warp = threadIdx.x >> 5;
    const bool side = (threadIdx.x & 16) != 0;
    // the pair of rows: a warp's two are four rows apart, 80 words of sigma or
    // node weights, so that its halves read different banks
    const int ty = (warp & 1) + 4 * (warp >> 1) + (side ? 2 : 0);
    const int i = i0 + tx, jA = j0 + 2 * ty, jB = jA + 1;
    const bool liveA = i <= g.nx && jA <= g.ny, liveB = i <= g.nx && jB <= g.ny;
    const ColGeo<float> cgA = col_geo(g, min(i, g.nx), min(jA, g.ny));
    const ColGeo<float> cgB = col_geo(g, min(i, g.nx), min(jB, g.ny));
    // of the first column; the second is one row on
    const int hf = (2 * ty + 1) * kFW + tx + 2;  // in a field plane of the tile
    const int hs = (2 * ty + 1) * kSW + tx + 1;  // in a sigma plane
    const int hn = 2 * ty * kPhX + tx;           // in a potential plane
    const int hw = 2 * ty * kNW + tx;            // in a node-weight plane
    constexpr int cf = kFR * kFW, cs = kFR * kSW;
    const int pxy = pl.Px * pl.Py, pc = pl.Pz * pxy;
    const int colA = min(i, pl.Px - 1) + pl.Px * min(jA, pl.Py - 1);
    const int colB = min(i, pl.Px - 1) + pl.Px * min(jB, pl.Py - 1);
    const bool issuer = threadIdx.x == 0;
    const unsigned tx_bytes = kFBytes + kSBytes;
    // the halo, half a warp a side.  Warp 0: potentials of the nodes (i0 .. i0 +
    // 15, j0 + 16) and (i0 + 16, j0 .. j0 + 15).  Warp 2: curls of the row j0 - 1
    // and of the column i0 - 1
    const int hni = side ? kTX : tx, hnj = side ? tx : kTY;
    const int hi = i0 + hni, hj = j0 + hnj;
    float hdX = 0.f, hdY = 0.f;       // warp 0: the node's widths
    float hrN = 0.f, hrT = 0.f;       // warp 2: 1 / d across the row or column and along it
    if (gd && warp == 0) {
        hdX = hi <= g.nx ? g.delX[hi] : 0.f;
        hdY = hj <= g.ny ? g.delY[hj] : 0.f;
    }
    if (warp == 2) {
        if (!side) {
            hrN = j0 >= 1 ? g.rdy[j0 - 1] : 0.f;
            hrT = i < g.nx ? g.rdx[i] : 0.f;
        } else {
            hrN = i0 >= 1 ? g.rdx[i0 - 1] : 0.f;
            hrT = j0 + tx < g.ny ? g.rdy[j0 + tx] : 0.f;
        }
    }

    // a chunk past the last node plane (the last chunks when the chunk count
    // does not divide the planes) has no work; it must return before it
    // issues a copy, since it would never wait for its third plane
    if (k0 >= k1) return true;
    if ((smem_addr(sm.fld[0]) | smem_addr(sm.sig[0]) | smem_addr(sm.nod[0])) & 127u) {
        if (issuer) atomicExch(err, 2);
        return false;
    }
    if (issuer) {
        for (int q = 0; q < HatTile::Ring; q++) mbar_init(smem_addr(&sm.mbar[q]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    unsigned phase = 0;
    const auto slot_of = [&](int p) { return (p - k0 + 1) % HatTile::Ring; };  // p >= k0 - 1
    const auto after = [](int s) { return s == HatTile::Ring - 1 ? 0 : s + 1; };
    // node weights are staged for planes k0 .. k1 (the diagonal and the
    // potentials need them), in slot p & 1
    auto issue = [&](int p) {
        if (!issuer) return;
        const int s = slot_of(p);
        const bool node = gd && p >= k0;
        const unsigned mb = smem_addr(&sm.mbar[s]);
        mbar_expect(mb, tx_bytes + (node ? kNBytes : 0u));
        tma_load4(smem_addr(sm.fld[s]), &tp.in, 2 * (i0 - 2), j0 - 1, p, 3 * r, mb);
        tma_load4(smem_addr(sm.sig[p & 3]), &tp.sig, i0, j0 - 1, p, 0, mb);
        if (node) tma_load3(smem_addr(sm.nod[p & 1]), &tp.node, i0, j0, p, mb);
    };
    auto wait = [&](int s) -> bool {
        if (mbar_wait(smem_addr(&sm.mbar[s]), (phase >> s) & 1u, limit)) {
            phase ^= 1u << s;
            return true;
        }
        return false;
    };
    auto give_up = [&](int first, int last) {
        if (!issuer) return;
        atomicExch(err, 1);
        for (int q = first; q <= last; q++) {
            const int s = slot_of(q);
            if (mbar_wait(smem_addr(&sm.mbar[s]), (phase >> s) & 1u, kWaitLimit)) phase ^= 1u << s;
        }
    };
    const float2 zero = make_float2(0.f, 0.f);
    const auto field = [&](int s) { return reinterpret_cast<const float2 *>(sm.fld[s]); };
    const auto sigma = [&](int p) { return reinterpret_cast<const float *>(sm.sig[p & 3]); };
    // potentials of the thread's nodes at plane p (fields in slot s, those
    // below in slot sb), and of a halo node
    struct Phi {
        float2 a, b, halo;
    };
    auto phi_form = [&](int p, int s, int sb, float dZ) {
        Phi v = {zero, zero, zero};
        const float2 *X = field(s), *Y = X + cf, *Z = Y + cf, *Zb = field(sb) + 2 * cf;
        const float *S = sigma(p), *Sb = sigma(p - 1), *N = reinterpret_cast<const float *>(sm.nod[p & 1]);
        const auto at = [&](int h, int q, float wn, float dX, float dY) {
            return hat_phi(wn, X[h - 1], X[h], Y[h - kFW], Y[h], Zb[h], Z[h], S + q, Sb + q, dX, dY, dZ);
        };
        v.a = at(hf, hs, N[hw], cgA.delXi, cgA.delYj);
        v.b = at(hf + kFW, hs + kSW, N[hw + kNW], cgB.delXi, cgB.delYj);
        if (warp == 0)
            v.halo = at((hnj + 1) * kFW + hni + 2, (hnj + 1) * kSW + hni + 1, N[hnj * kNW + hni], hdX, hdY);
        return v;
    };
    auto phi_put = [&](int p, const Phi &v) {
        float2 *P = sm.phi[p & 1];
        P[hn] = v.a;
        P[hn + kPhX] = v.b;
        if (warp == 0) P[hnj * kPhX + hni] = v.halo;
    };
    // signed node weights of the columns' nodes at the plane being computed:
    // (i, j), (i, j + 1), (i, j + 2), (i + 1, j), (i + 1, j + 1)
    float w0[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    auto node_w = [&](int p, float (&w)[5]) {
        const float *N = reinterpret_cast<const float *>(sm.nod[p & 1]);
        w[0] = N[hw];
        w[1] = N[hw + kNW];
        w[2] = N[hw + 2 * kNW];
        w[3] = N[hw + 1];
        w[4] = N[hw + kNW + 1];
    };
    // (padding entries of aux, where Ex, Ey or Ez does not exist, are zero; the
    // columns are clamped into the layout, so every lane loads)
    float2 axA = zero, ayA = zero, azA = zero, axB = zero, ayB = zero, azB = zero;
    auto load_aux = [&](int k) {
        if (!has_aux) return;
        const float2 *p = aux + pxy * k;
        axA = load_once(p + colA);
        ayA = load_once(p + colA + pc);
        azA = load_once(p + colA + 2 * pc);
        axB = load_once(p + colB);
        ayB = load_once(p + colB + pc);
        azB = load_once(p + colB + 2 * pc);
    };

    // the three edges of one node column at plane k from the fields x, y, z on
    // them and the curls around them: H*, before it along x (i), y (j) and z
    // (k).  Every edge slot is formed without branches: an edge that is not
    // interior (or does not exist: Ex at i = nx, Ey at j = ny, Ez at k = nz, all
    // padding entries of the layout) gets yhat = 0 and W = 0, so it adds nothing
    // to the inner products and keeps its zero.  The shared-memory reads stay
    // inside the tile whatever the edge.
    auto node_edges = [&](const ColGeo<float> &cg, const PlaneGeo<float> &pg, int k, int q, int n, float wS, float wX,
                          float wY, float wZ, float2 p1, int eb, float2 x, float2 y, float2 z, float2 Hx, float2 Hxj, float2 Hxk,
                          float2 Hy, float2 Hyi, float2 Hyk, float2 Hz, float2 Hzi, float2 Hzj, float2 ax, float2 ay,
                          float2 az) {
        const float *S0 = sigma(k) + q;
        const float2 *P0 = sm.phi[k & 1] + n;
        const bool kin = k >= 1 && k <= g.nz - 1;
        const float2 p0 = gd ? P0[0] : zero;
        // A x from its real part, then i omega mu0 sigma V_E x and D^-1
        const HatCoef w = hat_coef(cg, pg);
        const auto edge = [&](int comp, bool in, int e, float2 out, float2 v, float sig, float w1, float2 a) {
            float dr, di, W;
            hat_diag_of(comp, cg, pg, w, wmu, sig, gd, wS, w1, dr, di);
            out.x -= di * v.y;
            out.y += di * v.x;
            out = hat_div(out, dr, di, in, W);
            f(e, out, v, W, a);
        };
        {
            float2 out = csub(cscale(csub(Hz, Hzj), w.xz), cscale(csub(Hy, Hyk), w.xy));
            if (gd) out = cadd(out, cscale(csub(P0[1], p0), w.ax));
            edge(0, cg.intX && kin, eb, out, x, S0[0], wX, ax);
        }
        {
            float2 out = csub(cscale(csub(Hx, Hxk), w.yx), cscale(csub(Hz, Hzi), w.yz));
            if (gd) out = cadd(out, cscale(csub(P0[kPhX], p0), w.ay));
            edge(1, cg.intY && kin, pc + eb, out, y, S0[cs], wY, ay);
        }
        {
            float2 out = csub(cscale(csub(Hy, Hyi), w.zy), cscale(csub(Hx, Hxj), w.zx));
            if (gd) out = cadd(out, cscale(csub(p1, p0), w.az));
            edge(2, cg.intZ && k < g.nz, 2 * pc + eb, out, z, S0[2 * cs], wZ, az);
        }
    };
    const auto lane_before = [](float2 v) {
        return make_float2(__shfl_up_sync(0xffffffffu, v.x, 1, kTX), __shfl_up_sync(0xffffffffu, v.y, 1, kTX));
    };

    // the plane tables, 32 planes from kt on, a plane a lane
    int kt = 0;
    float tdz = 0.f, tdelZ = 0.f, trdz = 0.f, rdzk = k0 > 0 ? g.rdz[k0 - 1] : 0.f;
    auto tables = [&](int k) {
        kt = k;
        const int q = k + (threadIdx.x & 31);
        tdz = q < g.nz ? g.dz[q] : 0.f;
        trdz = q < g.nz ? g.rdz[q] : 0.f;
        tdelZ = g.delZ[min(q, g.nz)];
    };
    tables(k0);
    load_aux(k0);
    issue(k0 - 1);
    issue(k0);
    issue(k0 + 1);
    int s0 = 0, s1 = 1;  // slots of the plane marched and the one after it
    float2 HxAk = zero, HyAk = zero, HxBk = zero, HyBk = zero;  // curls of the plane before
    {
        const bool r0 = wait(s0), r1 = r0 && wait(s1);
        if (r1) {
            const float rdz = rdzk;
            const float2 *X0 = field(s0) + hf, *Y0 = X0 + cf, *Z0 = Y0 + cf, *X1 = field(s1) + hf, *Y1 = X1 + cf;
            HyAk = hat_curl(X1[0], X0[0], rdz, Z0[1], Z0[0], cgA.rdxi);
            HyBk = hat_curl(X1[kFW], X0[kFW], rdz, Z0[kFW + 1], Z0[kFW], cgB.rdxi);
            HxAk = hat_curl(Z0[kFW], Z0[0], cgA.rdyj, Y1[0], Y0[0], rdz);
            HxBk = hat_curl(Z0[2 * kFW], Z0[kFW], cgB.rdyj, Y1[kFW], Y0[kFW], rdz);
            if (gd) {
                phi_put(k0, phi_form(k0, s1, s0, g.delZ[k0]));
                node_w(k0, w0);
            }
        }
        slots_read();
        if (!__syncthreads_and(r1)) {
            give_up(r1 ? k0 + 1 : r0 ? k0 : k0 - 1, k0 + 1);
            return false;
        }
        if (k0 + 2 <= k1) issue(k0 + 2);
        s0 = s1;
        s1 = after(s1);
    }
    // One barrier per plane.  Before it the thread forms the curls of plane k
    // and the potentials of plane k + 1, as soon as its own wait for plane k +
    // 1 has completed, and keeps the fields and sigma of its edges; the
    // barrier publishes the curls, frees the field slot of plane k for the copy
    // issued after it, and makes a wait that gave up end the block as a whole.
    // After it come the edges of plane k, and the potentials of plane k + 1 take
    // the place of plane k - 1's, which no thread reads any more; what the
    // edges of plane k read is written again past the next barrier at the
    // earliest.
    for (int k = k0; k < k1; k++) {
        const bool ok = wait(s1);
        if (k + 1 >= kt + 32) tables(k);
        const float dZ1 = __shfl_sync(0xffffffffu, tdelZ, k + 1 - kt);
        const PlaneGeo<float> pg = {__shfl_sync(0xffffffffu, tdz, k - kt), __shfl_sync(0xffffffffu, tdelZ, k - kt),
                                    __shfl_sync(0xffffffffu, trdz, k - kt), rdzk};
        rdzk = pg.rdzk;
        // (what a wait that gave up leaves here is not used)
        const float2 *X0 = field(s0) + hf, *Y0 = X0 + cf, *Z0 = Y0 + cf, *X1 = field(s1) + hf, *Y1 = X1 + cf;
        const float2 xA = X0[0], yA = Y0[0], zA = Z0[0], xB = X0[kFW], yB = Y0[kFW], zB = Z0[kFW];
        const float2 HxA = hat_curl(zB, zA, cgA.rdyj, Y1[0], yA, pg.rdzk);
        const float2 HyA = hat_curl(X1[0], xA, pg.rdzk, Z0[1], zA, cgA.rdxi);
        const float2 HzA = hat_curl(Y0[1], yA, cgA.rdxi, xB, xA, cgA.rdyj);
        const float2 HxB = hat_curl(Z0[2 * kFW], zB, cgB.rdyj, Y1[kFW], yB, pg.rdzk);
        const float2 HyB = hat_curl(X1[kFW], xB, pg.rdzk, Z0[kFW + 1], zB, cgB.rdxi);
        const float2 HzB = hat_curl(Y0[kFW + 1], yB, cgB.rdxi, X0[2 * kFW], xB, cgB.rdyj);
        if (warp == 2) {
            // T along the row or column, N across it
            const int h = side ? (tx + 1) * kFW + 1 : tx + 2, sN = side ? 1 : kFW, sT = side ? kFW : 1;
            const float2 *T0 = field(s0) + h + (side ? 0 : cf), *T1 = field(s1) + h + (side ? 0 : cf);
            const float2 *N0 = field(s0) + h + (side ? cf : 0), *Zh = field(s0) + h + 2 * cf;
            const float2 a = hat_curl(Zh[sN], Zh[0], hrN, T1[0], T0[0], pg.rdzk);
            const float2 b = hat_curl(T0[sT], T0[0], hrT, N0[sN], N0[0], hrN);
            if (side) {
                sm.lefty[k & 1][tx] = make_float2(-a.x, -a.y);
                sm.leftz[k & 1][tx] = make_float2(-b.x, -b.y);
            } else {
                sm.hx[k & 1][0][tx] = a;
                sm.hz[k & 1][0][tx] = b;
            }
        }
        sm.hx[k & 1][ty + 1][tx] = HxB;
        sm.hz[k & 1][ty + 1][tx] = HzB;
        float w1[5] = {0.f, 0.f, 0.f, 0.f, 0.f};  // plane k + 1
        Phi p1 = {zero, zero, zero};
        if (gd) {
            p1 = phi_form(k + 1, s1, s0, dZ1);
            node_w(k + 1, w1);
        }
        slots_read();
        if (!__syncthreads_and(ok)) {
            give_up(ok ? k + 2 : k + 1, min(k + 2, k1));
            return false;
        }
        if (k + 3 <= k1) issue(k + 3);
        if (gd) phi_put(k + 1, p1);
        float2 HyAi = lane_before(HyA), HzAi = lane_before(HzA), HyBi = lane_before(HyB), HzBi = lane_before(HzB);
        if (tx == 0) {
            HyAi = sm.lefty[k & 1][2 * ty];
            HzAi = sm.leftz[k & 1][2 * ty];
            HyBi = sm.lefty[k & 1][2 * ty + 1];
            HzBi = sm.leftz[k & 1][2 * ty + 1];
        }
        if (liveA)
            node_edges(cgA, pg, k, hs, hn, w0[0], w0[3], w0[1], w1[0], p1.a, colA + pxy * k, xA, yA, zA, HxA, sm.hx[k & 1][ty][tx],
                       HxAk, HyA, HyAi, HyAk, HzA, HzAi, sm.hz[k & 1][ty][tx], axA, ayA, azA);
        if (liveB)
            node_edges(cgB, pg, k, hs + kSW, hn + kPhX, w0[1], w0[4], w0[2], w1[1], p1.b, colB + pxy * k, xB, yB, zB, HxB, HxA,
                       HxBk, HyB, HyBi, HyBk, HzB, HzBi, HzA, axB, ayB, azB);
        if (k + 1 < k1) load_aux(k + 1);
        HxAk = HxA, HyAk = HyA, HxBk = HxB, HyBk = HyB;
        for (int q = 0; q < 5; q++) w0[q] = w1[q];
        s0 = s1;
        s1 = after(s1);
    }
    return true;
}

// The operator launches of one iteration, by stage:
//   diagonal preconditioner
//     0  vh = D^-1 A u,            (rt, v) = sum conj(y) vh  -> alpha
//     1  th = D^-1 A sh,           (t, s)_W, (t, t)_W, (s, s)_W -> omega, ||r||
//   polynomial preconditioner M^-1 = c D^-1 (2 I - c A D^-1)
//     2  w1 = D^-1 A u
//     3  vh = c (2 w1 - c D^-1 A w1),  (rt, v)              -> alpha
//     4  w2 = D^-1 A sh
//     5  th = c (2 w2 - c D^-1 A w2),  (t, s)_W ... with s = sh read from memory
//     6  p = D^-1 A yhat at the end of a cycle (yhat in x0; see kh_conv)
// (D^-1 A (M^-1 p) = c (2 D^-1 A u - c D^-1 A w1) since u = D^-1 p.)  Stages
// 0 and 2 stage u and, after a restart, write the new shadow y = W rh
// (u = rh on that iteration).  For column tile bx and plane chunk bz of gz of
// right-hand side r; the stage and the grad-div term are compile-time.
template <int stage, bool gd>
__device__ __forceinline__ void hat_vt(const TmaParams &tp, const KArgs<float> &a, int r, int bx, int bz, int gz)
{
    constexpr bool kv = stage == 0 || stage == 3;  // (rt, v) and alpha
    constexpr bool kt = stage == 1 || stage == 5;  // omega and ||r||
    constexpr bool poly = stage == 3 || stage == 5;
    constexpr bool dots = kv || kt;
    constexpr bool conv = stage == 6;  // after the cycle, whatever the status
    BicgState &st = a.st[r];
    if ((!conv && st.status != KS_RUNNING) || !a.ost[r].active) return;
    if (!conv && a.sweeps && threadIdx.x == 0 && bx == 0 && bz == 0) atomicAdd(a.sweeps, 1ULL);
    int i0, j0, k0, k1;
    tma_tile_at<HatTile>(a.hmap, bx, i0, j0);
    tma_range_at(a.g.nz, bz, gz, k0, k1);
    const size_t off = (size_t)r * a.stride;
    float2 *out = (stage == 0 || stage == 3 ? a.v : stage == 2 || stage == 6 ? a.p : stage == 4 ? a.s : a.t) + off;
    float2 *Yr = a.rt + off;
    // after a restart (first iteration, pad set) the shadow becomes the
    // current residual: y = W rh, rh being the staged u of this launch
    const bool reset = (stage == 0 || stage == 2) && st.first && st.pad;
    const float2 *aux = kv ? Yr : stage == 5 ? a.sh + off : nullptr;
    const float c2 = 2.f * a.pc, cc = a.pc * a.pc;
    // inner products summed per edge in FP64 (per-plane FP32 partial sums
    // changed the Krylov rounding enough to send more right-hand sides to
    // the FP64 fallback)
    double u[4] = {0.0, 0.0, 0.0, 0.0};
    HatTile::Smem &sm = tma_smem<HatTile>();
    const bool ok = hat_march<gd, kv || stage == 5>(
        sm, tp, a.g, a.pl, r, aux, (float)(a.dsgn * a.ost[r].omega * kMu0), i0, j0, k0, k1, a.err, a.wait_limit,
        // y and W are zero at edges that are not interior, and so are x
        // and xa there (u, sh, w1, w2 and the shadow vanish off the
        // interior): those edges add nothing and need no test
        [&](int e, float2 y, float2 x, float W, float2 xa) {
            if (reset) Yr[e] = make_float2(W * x.x, W * x.y);
            if (poly) y = make_float2(c2 * x.x - cc * y.x, c2 * x.y - cc * y.y);  // c (2 x - c D^-1 A x)
            if (kv) {
                const float2 z = reset ? make_float2(W * x.x, W * x.y) : xa;
                u[0] += (double)z.x * y.x + (double)z.y * y.y;  // conj(y) vh
                u[1] += (double)z.x * y.y - (double)z.y * y.x;
            } else if (kt) {
                const float2 sv = stage == 5 ? xa : x;
                const double w = W;
                u[0] += w * ((double)y.x * sv.x + (double)y.y * sv.y);  // conj(t) s
                u[1] += w * ((double)y.x * sv.y - (double)y.y * sv.x);
                u[2] += w * ((double)y.x * y.x + (double)y.y * y.y);
                u[3] += w * ((double)sv.x * sv.x + (double)sv.y * sv.y);
            }
            out[e] = y;
        });
    if (!ok || !dots) return;
    // the march has read its last staged plane: the field ring is free
    double tot[4];
    if (block_reduce_last_in<4, kHatThreads>(u, a.parts, a.cnt, r, bx + a.hmap.tiles * bz, a.hmap.tiles * gz, tot,
                                reinterpret_cast<double *>(sm.fld[0]), reinterpret_cast<int *>(sm.fld[1])) &&
        threadIdx.x == 0) {
        if (kv) {
            fin_v(st, tot);
            st.pad = 0;
        } else {
            fin_t(st, tot);
            if (st.status == KS_RUNNING) {
                const cd ts = {tot[0], tot[1]}, om = st.omega;
                const double rn2 = tot[3] - 2.0 * (om.re * ts.re + om.im * ts.im) + (om.re * om.re + om.im * om.im) * tot[2];
                st.rn2 = rn2 > 0.0 ? rn2 : 0.0;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// kernels of one grid (blockIdx.y = right-hand side) and of a multi-grid
// batch (one flat block index over the right-hand sides of every grid)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) kh_u(KArgs<float> a) { hat_u(a, blockIdx.y, blockIdx.x); }
__global__ void __launch_bounds__(kThreads) kh_s(KArgs<float> a) { hat_s(a, blockIdx.y, blockIdx.x); }
__global__ void __launch_bounds__(kThreads) kh_xr(KArgs<float> a) { hat_xr(a, blockIdx.y, blockIdx.x); }
template <int stage, bool gd>
__global__ void __launch_bounds__(kHatThreads, 4) kh_vt(const __grid_constant__ TmaParams tp, KArgs<float> a)
{
    hat_vt<stage, gd>(tp, a, blockIdx.y, blockIdx.x, blockIdx.z, gridDim.z);
}

// the grids of a multi-grid batch, passed by value: each grid's arguments,
// its tensor maps (u and sh inputs) and where its blocks start in the flat
// launches
struct alignas(64) HatMulti {
    TmaParams tp[kMaxMultiGrids][4];  // inputs u, sh, w1, w2
    KArgs<float> a[kMaxMultiGrids];
    int ng;
    int nr[kMaxMultiGrids];            // right-hand sides of each grid
    int zch[kMaxMultiGrids];           // node-plane chunks of its stencil launches
    int eb0[kMaxMultiGrids + 1];       // first flat block of each grid: elementwise launches
    int sb0[kMaxMultiGrids + 1];       // first flat block of each grid: stencil launches
};
__device__ __forceinline__ int multi_grid_of(const int *b0, int ng, int b)
{
    int g = 0;
    while (g + 1 < ng && b >= b0[g + 1]) g++;
    return g;
}
template <int K> __global__ void __launch_bounds__(kThreads) kh_elem_multi(const __grid_constant__ HatMulti p)
{
    const int g = multi_grid_of(p.eb0, p.ng, blockIdx.x);
    const KArgs<float> &a = p.a[g];
    const int local = blockIdx.x - p.eb0[g];
    const int r = local / a.nblk, bx = local - r * a.nblk;
    if (K == 0) hat_u(a, r, bx);
    else if (K == 1) hat_s(a, r, bx);
    else hat_xr(a, r, bx);
}
// input map of each stage: u, sh, u, w1, sh, w2, x0
__host__ __device__ constexpr int stage_input(int stage)
{
    return stage == 0 || stage == 2 ? 0 : stage == 1 || stage == 4 ? 1 : stage == 3 ? 2 : stage == 6 ? 4 : 3;
}
template <int stage> __global__ void __launch_bounds__(kHatThreads, 4) kh_vt_multi(const __grid_constant__ HatMulti p)
{
    const int g = multi_grid_of(p.sb0, p.ng, blockIdx.x);
    const KArgs<float> &a = p.a[g];
    const int per = a.hmap.tiles * p.zch[g];
    const int local = blockIdx.x - p.sb0[g];
    const int r = local / per, rem = local - r * per;
    const int bz = rem / a.hmap.tiles, bx = rem - bz * a.hmap.tiles;
    const TmaParams &tp = p.tp[g][stage_input(stage)];
    if (a.gd) hat_vt<stage, true>(tp, a, r, bx, bz, p.zch[g]);
    else hat_vt<stage, false>(tp, a, r, bx, bz, p.zch[g]);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
ColMapHost hat_map(int nx, int ny)
{
    ColMapHost m;
    m.tiles_x = (nx + 1 + kTX - 1) / kTX;
    m.tiles = m.tiles_x * ((ny + 1 + kTY - 1) / kTY);
    return m;
}

static int hat_grid(long n) { return (int)std::min<long>((n + kThreads - 1) / kThreads, 148L * 16); }

void launch_hat_cast(const KArgs<float> &a, const double2 *r64, size_t stride64, int nrhs, cudaStream_t s)
{
    counted(1);
    kh_cast<<<dim3(hat_grid(a.g.nE), nrhs), kThreads, 0, s>>>(a, r64, stride64);
}

template <int stage, bool gd> static void launch_hat_vt_t(const KArgs<float> &a, const TmaParams &tp, int nrhs,
                                                           cudaStream_t s)
{
    const size_t sm = sizeof(HatTile::Smem);
    const int res = tma_resident(kh_vt<stage, gd>, sm, 2 + 2 * stage + (gd ? 1 : 0), kHatThreads);
    const int zc = a.zchunks ? a.zchunks : stage_chunks(a.g.nz, a.hmap.tiles, res, nrhs);
    kh_vt<stage, gd><<<dim3(a.hmap.tiles, nrhs, zc), kHatThreads, sm, s>>>(tp, a);
}
template <int stage> static void launch_hat_stage(const KArgs<float> &a, int nrhs, cudaStream_t s)
{
    counted(1);
    const TmaMaps *m = a.tma;
    TmaParams tp;
    constexpr int in = stage_input(stage);
    tp.in = in == 0 ? m->hph : in == 1 ? m->hsh : in == 2 ? m->hpw : in == 3 ? m->hsw : m->hx0;
    tp.sig = m->hsig;
    tp.node = m->hnode;
    if (a.gd) launch_hat_vt_t<stage, true>(a, tp, nrhs, s);
    else launch_hat_vt_t<stage, false>(a, tp, nrhs, s);
}

// one iteration; the events bracket the operator launches (the two of the
// polynomial preconditioner's first and second half together)
void launch_hat_iter(const KArgs<float> &a, int nrhs, cudaStream_t s, cudaEvent_t *ev)
{
    counted(3);
    const dim3 grid(a.nblk, nrhs);
    const bool poly = a.pc > 0.f;
    kh_u<<<grid, kThreads, 0, s>>>(a);
    if (ev) cudaEventRecord(ev[0], s);
    if (poly) {
        launch_hat_stage<2>(a, nrhs, s);
        launch_hat_stage<3>(a, nrhs, s);
    } else {
        launch_hat_stage<0>(a, nrhs, s);
    }
    if (ev) cudaEventRecord(ev[1], s);
    kh_s<<<grid, kThreads, 0, s>>>(a);
    if (ev) cudaEventRecord(ev[2], s);
    if (poly) {
        launch_hat_stage<4>(a, nrhs, s);
        launch_hat_stage<5>(a, nrhs, s);
    } else {
        launch_hat_stage<1>(a, nrhs, s);
    }
    if (ev) cudaEventRecord(ev[3], s);
    kh_xr<<<grid, kThreads, 0, s>>>(a);
}

void launch_hat_apply(const KArgs<float> &a, int nrhs, cudaStream_t s) { launch_hat_stage<0>(a, nrhs, s); }

// x = c (2 yhat - c p) with p = D^-1 A yhat (stage 6): the cycle's iterate
// from its accumulation in the D^-1-scaled space, for every active right-hand
// side (x0 holds the best yhat after launch_bicg_finish)
__global__ void __launch_bounds__(kThreads) kh_conv(KArgs<float> a)
{
    const int r = blockIdx.y, bx = blockIdx.x;
    if (!a.ost[r].active) return;
    const size_t off = (size_t)r * a.stride / 2;
    float4 *X = reinterpret_cast<float4 *>(a.x0) + off;
    const float4 *P = reinterpret_cast<const float4 *>(a.p) + off;
    const float c2 = 2.f * a.pc, cc = a.pc * a.pc;
    HAT_PAIRS(a, bx)
    {
        const float4 x = X[q], w = P[q];
        X[q] = make_float4(c2 * x.x - cc * w.x, c2 * x.y - cc * w.y, c2 * x.z - cc * w.z, c2 * x.w - cc * w.w);
    }
}
void launch_hat_conv(const KArgs<float> &a, int nrhs, cudaStream_t s)
{
    if (!(a.pc > 0.f)) return;
    launch_hat_stage<6>(a, nrhs, s);
    counted(1);
    kh_conv<<<dim3(a.nblk, nrhs), kThreads, 0, s>>>(a);
}

// the shared-memory attribute and occupancy of every operator kernel, set
// before a capture (tma_resident calls the runtime only the first time)
template <int stage> static void hat_prime_stage()
{
    const size_t sm = sizeof(HatTile::Smem);
    tma_resident(kh_vt<stage, false>, sm, 2 + 2 * stage, kHatThreads);
    tma_resident(kh_vt<stage, true>, sm, 3 + 2 * stage, kHatThreads);
    if (stage < 6) tma_resident(kh_vt_multi<(stage < 6 ? stage : 0)>, sm, 16 + stage, kHatThreads);
}
static void hat_prime()
{
    hat_prime_stage<0>();
    hat_prime_stage<1>();
    hat_prime_stage<2>();
    hat_prime_stage<3>();
    hat_prime_stage<4>();
    hat_prime_stage<5>();
    hat_prime_stage<6>();
}

void HatGraph::reset()
{
    if (exec) cudaGraphExecDestroy(exec);
    exec = nullptr;
    key.clear();
}
HatGraph::~HatGraph()
{
    reset();
    if (cap) cudaStreamDestroy(cap);
}

// ---------------------------------------------------------------------------
// One FP32 cycle as a graph: a loop on the device around kHatBody iterations
// that ends when no right-hand side is running any more.  A cycle captured as
// all its iterations went on through seven empty launches for each that was
// left (1.1 us each): of the 900 iterations in three cycles of a 24^3 solve
// 286 had work.  The loop ends by its count at the latest, so also when a
// bounded wait gave up and left the states as they were.
// ---------------------------------------------------------------------------
constexpr int kHatBody = 10;
struct HatLoop {
    const BicgState *st[kMaxMultiGrids];
    const OuterState *ost[kMaxMultiGrids];
    int n[kMaxMultiGrids], ng, bodies;
    int *count;  // bodies run
};
__global__ void __launch_bounds__(32) kh_more(const __grid_constant__ HatLoop p, cudaGraphConditionalHandle h)
{
    int more = 0;
    for (int g = 0; g < p.ng; g++)
        for (int r = threadIdx.x; r < p.n[g]; r += 32) more |= p.st[g][r].status == KS_RUNNING && p.ost[g][r].active;
    more = __any_sync(0xffffffffu, more);
    if (threadIdx.x) return;
    const int done = ++*p.count;
    cudaGraphSetConditional(h, more && done < p.bodies ? 1u : 0u);
}

static cudaError_t hat_graph_build(HatGraph &hg, cudaGraph_t graph, const KArgs<float> *args, const int *nrhs,
                                   const int *zch, int ng, int maxit)
{
    const int n = ng > 0 ? ng : 1;
    HatLoop p;
    std::memset(&p, 0, sizeof p);
    p.ng = n;
    p.bodies = (maxit + kHatBody - 1) / kHatBody;
    p.count = hat_loop_count(args[0]);
    for (int g = 0; g < n; g++) {
        p.st[g] = args[g].st;
        p.ost[g] = args[g].ost;
        p.n[g] = nrhs[g];
    }
    cudaGraphConditionalHandle h;
    cudaError_t e = cudaGraphConditionalHandleCreate(&h, graph, 1, cudaGraphCondAssignDefault);
    if (e != cudaSuccess) return e;
    cudaMemsetParams ms{};
    ms.dst = p.count;
    ms.elementSize = sizeof(int);
    ms.width = 1;
    ms.height = 1;
    cudaGraphNode_t zero, loop;
    if ((e = cudaGraphAddMemsetNode(&zero, graph, nullptr, 0, &ms)) != cudaSuccess) return e;
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = h;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    if ((e = cudaGraphAddNode(&loop, graph, &zero, 1, &np)) != cudaSuccess) return e;
    const cudaGraph_t body = np.conditional.phGraph_out[0];
    e = cudaStreamBeginCaptureToGraph(hg.cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    hg.launches = 0;
    t_captured = &hg.launches;
    for (int it = 0; it < kHatBody; it++) {
        if (ng > 0) launch_hat_iter_multi(args, nrhs, zch, ng, hg.cap);
        else launch_hat_iter(args[0], nrhs[0], hg.cap);
    }
    counted(1);
    kh_more<<<1, 32, 0, hg.cap>>>(p, h);
    t_captured = nullptr;
    cudaGraph_t out = nullptr;
    return cudaStreamEndCapture(hg.cap, &out);
}

cudaError_t hat_graph_run(HatGraph &hg, const KArgs<float> *args, const int *nrhs, const int *zch, int ng, int maxit,
                          cudaStream_t s)
{
    const int n = ng > 0 ? ng : 1;
    if (ng > kMaxMultiGrids) return cudaErrorInvalidValue;
    // the key: the launch arguments, the tensor maps they point to, the
    // right-hand-side and chunk counts and the cycle length
    std::vector<unsigned char> k;
    auto put = [&](const void *p, size_t b) {
        const unsigned char *c = static_cast<const unsigned char *>(p);
        k.insert(k.end(), c, c + b);
    };
    for (int g = 0; g < n; g++) {
        put(&args[g], sizeof(KArgs<float>));
        if (args[g].tma) put(args[g].tma, sizeof(TmaMaps));
        put(&nrhs[g], sizeof(int));
        const int z = zch ? zch[g] : 0;
        put(&z, sizeof z);
    }
    put(&ng, sizeof ng);
    put(&maxit, sizeof maxit);
    if (!hg.exec || k != hg.key) {
        hg.reset();
        if (!hg.cap) {
            cudaError_t e = cudaStreamCreateWithFlags(&hg.cap, cudaStreamNonBlocking);
            if (e != cudaSuccess) return e;
        }
        hat_prime();
        cudaGraph_t graph = nullptr;
        cudaError_t e = cudaGraphCreate(&graph, 0);
        if (e != cudaSuccess) return e;
        e = hat_graph_build(hg, graph, args, nrhs, zch, ng, maxit);
        if (e == cudaSuccess) e = cudaGraphInstantiate(&hg.exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) {
            hg.exec = nullptr;
            return e;
        }
        hg.key.swap(k);
    }
    return cudaGraphLaunch(hg.exec, s);
}

// one iteration of the fused FP32 BiCGStab over the grids of a multi-grid
// batch: five launches in all, each over the right-hand sides of every grid
// (zch[g]: node-plane chunks of grid g's stencil blocks, 0 for the
// occupancy-based choice)
// as launch_hat_iter, for the grids of a multi-grid batch; ev (4 events, may
// be null) brackets the operator launches
int launch_hat_iter_multi(const KArgs<float> *args, const int *nrhs, const int *zch, int ng, cudaStream_t s,
                          cudaEvent_t *ev)
{
    if (ng < 1 || ng > kMaxMultiGrids) return 1;
    static_assert(sizeof(HatMulti) <= 32000, "multi-grid parameters exceed the kernel parameter space");
    HatMulti p;
    std::memset(&p, 0, sizeof p);
    p.ng = ng;
    const size_t smb = sizeof(HatTile::Smem);
    const int res = tma_resident(kh_vt_multi<0>, smb, 16, kHatThreads);
    tma_resident(kh_vt_multi<1>, smb, 17, kHatThreads);
    tma_resident(kh_vt_multi<2>, smb, 18, kHatThreads);
    tma_resident(kh_vt_multi<3>, smb, 19, kHatThreads);
    tma_resident(kh_vt_multi<4>, smb, 20, kHatThreads);
    tma_resident(kh_vt_multi<5>, smb, 21, kHatThreads);
    p.eb0[0] = p.sb0[0] = 0;
    for (int g = 0; g < ng; g++) {
        p.a[g] = args[g];
        p.nr[g] = nrhs[g];
        p.tp[g][0].in = args[g].tma->hph;
        p.tp[g][1].in = args[g].tma->hsh;
        p.tp[g][2].in = args[g].tma->hpw;
        p.tp[g][3].in = args[g].tma->hsw;
        for (int w = 0; w < 4; w++) {
            p.tp[g][w].sig = args[g].tma->hsig;
            p.tp[g][w].node = args[g].tma->hnode;
        }
        // the count of the grid by itself (the blocks of the grids mix, and the
        // time is flat about it: 262 to 273 ms for 40^3 + 64 x 64 x 48 cells with
        // counts from 3, 5 to 11, 13); more chunks than planes would only add
        // empty ones, and the reductions' partial sums have room for one a plane
        const int own = args[g].zchunks;
        p.zch[g] = std::min(zch && zch[g] > 0 ? zch[g] : own ? own : stage_chunks(args[g].g.nz, args[g].hmap.tiles, res, nrhs[g]),
                            args[g].g.nz + 1);
        p.eb0[g + 1] = p.eb0[g] + nrhs[g] * args[g].nblk;
        p.sb0[g + 1] = p.sb0[g] + nrhs[g] * args[g].hmap.tiles * p.zch[g];
    }
    // the polynomial preconditioner is used when the first grid's handle
    // has it (every handle of a batch shares the control)
    const bool poly = args[0].pc > 0.f;
    counted(poly ? 7 : 5);
    const size_t sm = sizeof(HatTile::Smem);
    kh_elem_multi<0><<<p.eb0[ng], kThreads, 0, s>>>(p);
    if (ev) cudaEventRecord(ev[0], s);
    if (poly) {
        kh_vt_multi<2><<<p.sb0[ng], kHatThreads, sm, s>>>(p);
        kh_vt_multi<3><<<p.sb0[ng], kHatThreads, sm, s>>>(p);
    } else {
        kh_vt_multi<0><<<p.sb0[ng], kHatThreads, sm, s>>>(p);
    }
    if (ev) cudaEventRecord(ev[1], s);
    kh_elem_multi<1><<<p.eb0[ng], kThreads, 0, s>>>(p);
    if (ev) cudaEventRecord(ev[2], s);
    if (poly) {
        kh_vt_multi<4><<<p.sb0[ng], kHatThreads, sm, s>>>(p);
        kh_vt_multi<5><<<p.sb0[ng], kHatThreads, sm, s>>>(p);
    } else {
        kh_vt_multi<1><<<p.sb0[ng], kHatThreads, sm, s>>>(p);
    }
    if (ev) cudaEventRecord(ev[3], s);
    kh_elem_multi<2><<<p.eb0[ng], kThreads, 0, s>>>(p);
    return 0;
}

}  // namespace mt3d
