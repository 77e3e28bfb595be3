// noalloc.cu -- y = A x on caller-owned device vectors with no device
// allocation: the operator product of mt3d_mult_aii straight from one
// interior vector to the other (k_apply_interior), or, where the two overlap,
// through full edge vectors in a fixed scratch.
//
// The scratch (the two full-edge vectors, the grad-div node potentials and
// the per-call state) is one file-scope array per device, shared by every
// handle on that device.  Its address is looked up once per device
// (cudaGetSymbolAddress, with that device current) when mt3d_create makes the
// first handle there: under CUDA's lazy module loading that look-up is what
// commits the array's 16 MiB, and the kernels this entry launches are loaded
// at the same time, so the entry itself takes no device memory, on its first
// call or later.  Two calls on overlapping vectors whose GPU work overlaps in
// time on one device (different streams, handles or host threads) use the
// same scratch and race; calls enqueued on one stream run one after the other
// and are safe.
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <mutex>

#include "common.cuh"
#include "kernels.h"
#include "solver.h"

namespace mt3d {

// 16 MiB: the state record plus (2 nE + nN) complex doubles, enough for
// grids up to about 52^3 cells (nE ~ 3 n^3, nN ~ n^3)
constexpr size_t kNoAllocScratchBytes = size_t(16) << 20;
constexpr size_t kNoAllocStateBytes = 256;
static_assert(sizeof(OuterState) <= kNoAllocStateBytes, "state record does not fit its slot");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
static std::mutex g_noalloc_mutex;
static void *g_noalloc_ptr[kNoAllocMaxDevices] = {};

// device address of the scratch on the current device (set-up on first use)
static int noalloc_scratch(int dev, void **ptr, std::string &err)
{
    if (dev < 0 || dev >= kNoAllocMaxDevices) {
        err = "device ordinal out of range for the fixed scratch table";
        return 5;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            err = std::string("cudaGetSymbolAddress of the fixed scratch failed: ") + cudaGetErrorString(e);
            return 4;
        }
        g_noalloc_ptr[dev] = p;
    }
    *ptr = g_noalloc_ptr[dev];
    return 0;
}

// the per-call state record: all fields zero except omega and active
__global__ void k_noalloc_state(OuterState *st, double omega)
{
    OuterState s{};
    s.omega = omega;
    s.active = 1;
    *st = s;
}

// ---------------------------------------------------------------------------
// The product on interior vectors in one launch.  A block takes the 16 x 4 x
// 4 nodes of its tile, a thread the three edges that leave its node; x is read
// where it lies, the boundary as zeros.  With the grad-div term the block
// first forms the node potentials of its tile and of one plane of nodes past
// it in shared memory (1.66 potentials a node instead of the 6 that edges
// would form on their own).  The grids this entry takes fit in the L2 cache,
// so the call is bound by launches and latency: a clear, a scatter to the full
// vector, the potentials, the product and a gather took 13.1 us a call on
// 24^3 cells and 17.8 us on 51 x 50 x 53 with the grad-div term, this 3.8
// (most of it the host's side of the launch) and 7.5 us.
// gd: 0 none, 1 GD (c at the edge inside the potential), 2 GD^T (outside).
// ---------------------------------------------------------------------------
constexpr int kAiX = 16, kAiY = 4, kAiZ = 4, kAiN = (kAiX + 1) * (kAiY + 1) * (kAiZ + 1);
template <int gd>
__global__ void __launch_bounds__(kAiX *kAiY *kAiZ) k_apply_interior(Geo<double> g, const double *__restrict__ sigma,
                                                                     const double *__restrict__ gdw,
                                                                     const unsigned char *__restrict__ gde, double wmu,
                                                                     const double2 *__restrict__ x,
                                                                     double2 *__restrict__ y)
{
    __shared__ double2 phi[gd ? kAiN : 1];
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int nXi = nx * (ny - 1) * (nz - 1), nYi = (nx - 1) * ny * (nz - 1);
    // place of an interior edge in the interior vectors
    auto pX = [&](int i, int j, int k) { return i + nx * (j - 1 + (ny - 1) * (k - 1)); };
    auto pY = [&](int i, int j, int k) { return nXi + i - 1 + (nx - 1) * (j + ny * (k - 1)); };
    auto pZ = [&](int i, int j, int k) { return nXi + nYi + i - 1 + (nx - 1) * (j - 1 + (ny - 1) * k); };
    auto inx = [&](int i) { return i >= 1 && i < nx; };
    auto iny = [&](int j) { return j >= 1 && j < ny; };
    auto inz = [&](int k) { return k >= 1 && k < nz; };
    const double2 zero = make_double2(0, 0);
    auto X = [&](int i, int j, int k) { return i >= 0 && i < nx && iny(j) && inz(k) ? x[pX(i, j, k)] : zero; };
    auto Y = [&](int i, int j, int k) { return inx(i) && j >= 0 && j < ny && inz(k) ? x[pY(i, j, k)] : zero; };
    auto Z = [&](int i, int j, int k) { return inx(i) && iny(j) && k >= 0 && k < nz ? x[pZ(i, j, k)] : zero; };
    const int i0 = blockIdx.x * kAiX, j0 = blockIdx.y * kAiY, k0 = blockIdx.z * kAiZ;
    if (gd) {
        for (int t = threadIdx.x; t < kAiN; t += kAiX * kAiY * kAiZ) {
            const int i = i0 + t % (kAiX + 1), j = j0 + t / (kAiX + 1) % (kAiY + 1), k = k0 + t / ((kAiX + 1) * (kAiY + 1));
            double2 out = zero;
            if (inx(i) && iny(j) && inz(k)) {
                const int n = iN(g, i, j, k);
                const bool cs = gd == 1 && gde[n];
                const double d0 = g.delY[j] * g.delZ[k], d1 = g.delX[i] * g.delZ[k], d2 = g.delX[i] * g.delY[j];
                auto c = [&](double d, int e) { return cs ? d * sigma[e] : d; };
                // what ends at the node minus what starts there
                out = cscale(x[pX(i - 1, j, k)], c(d0, iX(g, i - 1, j, k)));
                out = csub(out, cscale(x[pX(i, j, k)], c(d0, iX(g, i, j, k))));
                out = cadd(out, cscale(x[pY(i, j - 1, k)], c(d1, iY(g, i, j - 1, k))));
                out = csub(out, cscale(x[pY(i, j, k)], c(d1, iY(g, i, j, k))));
                out = cadd(out, cscale(x[pZ(i, j, k - 1)], c(d2, iZ(g, i, j, k - 1))));
                out = csub(out, cscale(x[pZ(i, j, k)], c(d2, iZ(g, i, j, k))));
                out = cscale(out, gdw[n]);
            }
            phi[t] = out;
        }
        __syncthreads();
    }
    const int ti = threadIdx.x % kAiX, tj = threadIdx.x / kAiX % kAiY, tk = threadIdx.x / (kAiX * kAiY);
    const int i = i0 + ti, j = j0 + tj, k = k0 + tk;
    if (i > nx || j > ny || k > nz) return;
    const int hn = ti + (kAiX + 1) * (tj + (kAiY + 1) * tk);
    // i omega mu0 sigma V_E x and the grad-div term between the nodes hn and hn + step
    auto rest = [&](double2 acc, double2 x0, const EdgeIdx &q, double sg, double dfa, int step, int nstep) {
        const double dt = wmu * sg * edge_volume(g, q);
        acc.x -= dt * x0.y;
        acc.y += dt * x0.x;
        if (gd) {
            double2 a = phi[hn], b = phi[hn + step];
            if (gd == 2) {
                const int n = iN(g, i, j, k);
                if (gde[n]) a = cscale(a, sg);
                if (gde[n + nstep]) b = cscale(b, sg);
            }
            acc = cadd(acc, cscale(csub(b, a), dfa));
        }
        return acc;
    };
    // the stencil of common.cuh
    if (i < nx && iny(j) && inz(k)) {
        const double2 x0 = x[pX(i, j, k)];
        const double2 yy = csub(cadd(csub(Y(i + 1, j, k), Y(i, j, k)), Y(i, j - 1, k)), Y(i + 1, j - 1, k));
        const double2 zz = csub(cadd(csub(Z(i + 1, j, k), Z(i, j, k)), Z(i, j, k - 1)), Z(i + 1, j, k - 1));
        const double2 fyp = cscale(csub(X(i, j + 1, k), x0), g.rdy[j]), fym = cscale(csub(x0, X(i, j - 1, k)), g.rdy[j - 1]);
        const double2 fzp = cscale(csub(X(i, j, k + 1), x0), g.rdz[k]), fzm = cscale(csub(x0, X(i, j, k - 1)), g.rdz[k - 1]);
        double2 acc = cadd(cscale(yy, g.delZ[k]), cscale(zz, g.delY[j]));
        acc = csub(acc, cscale(csub(fyp, fym), g.dx[i] * g.delZ[k]));
        acc = csub(acc, cscale(csub(fzp, fzm), g.dx[i] * g.delY[j]));
        y[pX(i, j, k)] = rest(acc, x0, EdgeIdx{0, i, j, k}, sigma[iX(g, i, j, k)], g.delY[j] * g.delZ[k], 1, 1);
    }
    if (inx(i) && j < ny && inz(k)) {
        const double2 x0 = x[pY(i, j, k)];
        const double2 zz = csub(cadd(csub(Z(i, j + 1, k), Z(i, j, k)), Z(i, j, k - 1)), Z(i, j + 1, k - 1));
        const double2 xx = csub(cadd(csub(X(i, j + 1, k), X(i, j, k)), X(i - 1, j, k)), X(i - 1, j + 1, k));
        const double2 fzp = cscale(csub(Y(i, j, k + 1), x0), g.rdz[k]), fzm = cscale(csub(x0, Y(i, j, k - 1)), g.rdz[k - 1]);
        const double2 fxp = cscale(csub(Y(i + 1, j, k), x0), g.rdx[i]), fxm = cscale(csub(x0, Y(i - 1, j, k)), g.rdx[i - 1]);
        double2 acc = cadd(cscale(zz, g.delX[i]), cscale(xx, g.delZ[k]));
        acc = csub(acc, cscale(csub(fzp, fzm), g.dy[j] * g.delX[i]));
        acc = csub(acc, cscale(csub(fxp, fxm), g.dy[j] * g.delZ[k]));
        y[pY(i, j, k)] = rest(acc, x0, EdgeIdx{1, i, j, k}, sigma[iY(g, i, j, k)], g.delX[i] * g.delZ[k], kAiX + 1, nx + 1);
    }
    if (inx(i) && iny(j) && k < nz) {
        const double2 x0 = x[pZ(i, j, k)];
        const double2 xx = csub(cadd(csub(X(i, j, k + 1), X(i, j, k)), X(i - 1, j, k)), X(i - 1, j, k + 1));
        const double2 yy = csub(cadd(csub(Y(i, j, k + 1), Y(i, j, k)), Y(i, j - 1, k)), Y(i, j - 1, k + 1));
        const double2 fxp = cscale(csub(Z(i + 1, j, k), x0), g.rdx[i]), fxm = cscale(csub(x0, Z(i - 1, j, k)), g.rdx[i - 1]);
        const double2 fyp = cscale(csub(Z(i, j + 1, k), x0), g.rdy[j]), fym = cscale(csub(x0, Z(i, j - 1, k)), g.rdy[j - 1]);
        double2 acc = cadd(cscale(xx, g.delY[j]), cscale(yy, g.delX[i]));
        acc = csub(acc, cscale(csub(fxp, fxm), g.dz[k] * g.delY[j]));
        acc = csub(acc, cscale(csub(fyp, fym), g.dz[k] * g.delX[i]));
        y[pZ(i, j, k)] = rest(acc, x0, EdgeIdx{2, i, j, k}, sigma[iZ(g, i, j, k)], g.delX[i] * g.delY[j],
                              (kAiX + 1) * (kAiY + 1), (nx + 1) * (ny + 1));
    }
}

// set-up at handle creation, with device `dev` current: the scratch address
// (committing the array) and the kernels of the entry (loading their modules)
int noalloc_prepare(int dev, std::string &err)
{
    void *p = nullptr;
    int rc = noalloc_scratch(dev, &p, err);
    if (rc) return rc;
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, k_noalloc_state);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_apply_interior<0>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_apply_interior<1>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_apply_interior<2>);
    if (e == cudaSuccess) e = preload_apply_kernels();
    if (e != cudaSuccess) {
        cudaGetLastError();
        err = std::string("loading the operator kernels failed: ") + cudaGetErrorString(e);
        return 4;
    }
    return 0;
}

extern std::atomic<long long> g_launch_count;

static bool device_vector(const void *p, int dev)
{
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (at.type != cudaMemoryTypeDevice && at.type != cudaMemoryTypeManaged) return false;
    return at.type == cudaMemoryTypeManaged || at.device == dev;
}

int Solver::mult_aii_noalloc(int adjt, const double *x, double *y)
{
    const char *who = "mt3d_mult_aii_device_noalloc";
    if (!cond_set) return fail(5, std::string(who) + ": conductivity not set (call mt3d_update_cond)");
    if (!(omega > 0)) return fail(5, std::string(who) + ": frequency not set (call mt3d_update_freq)");
    if (!x || !y) return fail(5, std::string(who) + ": null vector");
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15)
        return fail(5, std::string(who) + ": x and y must be 16-byte aligned");
    if (!device_vector(x, dev_) || !device_vector(y, dev_))
        return fail(5, std::string(who) + ": x and y must be device memory of the handle's device");
    const bool gd = ctl.formulation == 1;
    const size_t need = kNoAllocStateBytes + sizeof(double2) * (size_t)(2 * nE + (gd ? nN : 0));
    if (need > kNoAllocScratchBytes) {
        char buf[256];
        snprintf(buf, sizeof buf,
                 "%s: this grid needs %zu bytes of scratch, more than the fixed %zu-byte scratch (at most about "
                 "52^3 cells); use mt3d_mult_aii",
                 who, need, kNoAllocScratchBytes);
        return fail(5, buf);
    }
    const uintptr_t bx = reinterpret_cast<uintptr_t>(x), by = reinterpret_cast<uintptr_t>(y), nb = nEi * sizeof(double2);
    if (bx >= by + nb || by >= bx + nb) {
        const double wmu = (adjt ? 1.0 : -1.0) * omega * kMu0;
        const dim3 grid(nx / kAiX + 1, ny / kAiY + 1, nz / kAiZ + 1);
        const double *sg = (gd ? sigs64_ : sig64_).as<double>(), *w = gdw64_.as<double>();
        const unsigned char *earth = gde_.as<unsigned char>();
        const double2 *xi = reinterpret_cast<const double2 *>(x);
        double2 *yi = reinterpret_cast<double2 *>(y);
        auto *kern = !gd ? k_apply_interior<0> : adjt ? k_apply_interior<2> : k_apply_interior<1>;
        kern<<<grid, kAiX * kAiY * kAiZ, 0, stream_>>>(g64_, sg, w, earth, wmu, xi, yi);
        g_launch_count.fetch_add(1, std::memory_order_relaxed);
        return check(cudaGetLastError(), who);
    }
    // y on top of x: the full-vector route, which has read all of x before it
    // writes y
    void *base = nullptr;
    std::string err;
    int rc = noalloc_scratch(dev_, &base, err);
    if (rc) return fail(rc, std::string(who) + ": " + err);
    unsigned char *p = static_cast<unsigned char *>(base);
    OuterState *st = reinterpret_cast<OuterState *>(p);
    double2 *xf = reinterpret_cast<double2 *>(p + kNoAllocStateBytes);
    double2 *yf = xf + nE;
    double2 *phi = gd ? yf + nE : nullptr;
    // the boundary edges of xf must read as zero (the scatter writes only the
    // interior); yf and phi are written in full by their kernels
    if ((rc = check(cudaMemsetAsync(xf, 0, nE * sizeof(double2), stream_), who))) return rc;
    k_noalloc_state<<<1, 1, 0, stream_>>>(st, omega);
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    launch_scatter_interior((int)nEi, edgei_d_.as<int>(), reinterpret_cast<const double2 *>(x), xf, stream_);
    KArgs<double> a = kargs<double>(1, 0);
    a.ost = st;
    a.phi = phi;
    a.dsgn = adjt ? 1.0 : -1.0;
    launch_apply(a, xf, yf, 0, 1, stream_, gd ? (adjt ? 2 : 1) : 0);
    launch_gather_interior((int)nEi, edgei_d_.as<int>(), yf, reinterpret_cast<double2 *>(y), stream_);
    return check(cudaGetLastError(), who);
}

}  // namespace mt3d
