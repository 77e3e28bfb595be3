// tma.cuh -- shared pieces of the TMA-staged FP32 stencil kernels
// (tmakernels.cu, hatkernels.cu): tensor maps, tile and ring geometry, the
// shared-memory ring, mbarrier and tensor-copy wrappers, and the grad-div
// node potential formed from the staged planes.
//
// A block owns TX x TY node columns of one right-hand side and marches a
// chunk of node planes.  Per plane one thread issues the tensor copies of the
// fields (Ex, Ey, Ez over i0-2 .. i0+TX+1, j0-1 .. j0+TY), sigma (i0-1 ..
// i0+TX+2, j0-1 .. j0+TY; its tensor is stored one column to the right, see
// sig_layout) and the signed node weights (i0 .. i0+TX+3, j0 .. j0+TY) into
// rings in shared memory, completed on an mbarrier per field slot.  The x
// coordinates lie on 16-byte boundaries, as tensor copies require; coordinates
// outside a tensor read zeros.  No copy uses cluster multicast.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "colstencil.cuh"
#include "kernels.h"

namespace mt3d {

struct TmaMaps {
    CUtensorMap x0, ph, sh;  // input vectors [nrhs][3][Pz][Py][2 Px] (float)
    CUtensorMap sig;         // sigma [3][Pz][Py][sig_layout(pl).Px] (float)
    CUtensorMap node;        // signed node weights [Pz][Py][Px] (float)
    // the same and the polynomial preconditioner's intermediates (vectors p,
    // s) in the boxes of the fused stencil's tile
    CUtensorMap hx0, hph, hsh, hpw, hsw, hsig, hnode;
    int ok;
};
struct alignas(64) TmaParams {
    CUtensorMap in, sig, node;
};

constexpr int kWaitLimit = 1 << 22;
constexpr int kMaxMultiGrids = 8;  // grids of one multi-grid batch

// A tile of TX x TY node columns: the staged planes and the ring in shared
// memory, its slots 128-byte aligned: the fields of four planes (k-1, k, k+1 in
// use, k+2 in flight), sigma of three (k, k+1, k+2) and the node weights of
// two (k+1, k+2), so that four blocks fit on an SM
template <int TX_, int TY_> struct TmaTile {
    static constexpr int TX = TX_, TY = TY_;
    static constexpr int FW = TX + 4, FR = TY + 2;  // field plane: columns (float2) i0-2 .., rows j0-1 ..
    static constexpr int SW = TX + 4;               // sigma plane: columns i0-1 ..
    static constexpr int NW = TX + 4, NR = TY + 1;  // node plane: columns i0 .., rows j0 ..
    static constexpr int PhX = TX + 1, PhN = (TX + 1) * (TY + 1);
    static constexpr unsigned FBytes = 3 * FR * FW * 8, SBytes = 3 * FR * SW * 4, NBytes = NR * NW * 4;
    static constexpr unsigned slot(unsigned b) { return (b + 127) / 128 * 128; }
    struct Smem {
        alignas(128) unsigned char fld[4][slot(FBytes)];
        alignas(128) unsigned char sig[3][slot(SBytes)];
        alignas(128) unsigned char nod[2][slot(NBytes)];
        float2 phi[2][PhN];
        unsigned long long mbar[4];
    };
};
// the unfused kernels (tmakernels.cu): a thread per node column
using KctTile = TmaTile<32, 8>;
static_assert(KctTile::TX * KctTile::TY == kThreads, "one thread per node column");
// the fused stencil (hatkernels.cu): 128 threads, each on two node rows next to
// one another.  A row of 16 wastes at most 15 lanes on a grid's rim where one of 32
// wastes up to 31 (65 nodes take 80 columns instead of 96, 41 take 48 instead
// of 64, 201 take 208 instead of 224), at the same halo a tile.  us a launch
// against a 32 x 8 tile, both with every edge forming its own differences: 40^3,
// 8 right-hand sides 25.6 (30.5); 100 x 100 x 60, 2: 44.3 (47.5); 200 x 200 x 100,
// 4: 380 (392).
// Its ring holds the fields of three planes (k and k + 1 in use until the curls
// of plane k are formed, then k + 1, k + 2 and k + 3), sigma of four and the
// node weights of two; the curls that cross threads or tiles (hx, hz: the row
// before each thread's pair; left: the column before the tile) and the
// potentials are kept for two planes, so that one barrier a plane is enough.
constexpr int kHatThreads = 128, kHatPairs = 8;
struct HatTile : TmaTile<16, 16> {
    static constexpr int Ring = 3;
    struct Smem {
        alignas(128) unsigned char fld[Ring][slot(FBytes)];
        alignas(128) unsigned char sig[4][slot(SBytes)];
        alignas(128) unsigned char nod[2][slot(NBytes)];
        float2 phi[2][PhN];
        float2 hx[2][kHatPairs + 1][TX], hz[2][kHatPairs + 1][TX];
        float2 lefty[2][TY], leftz[2][TY];
        unsigned long long mbar[Ring];
    };
};
static_assert(kHatThreads == HatTile::TX * kHatPairs && 2 * kHatPairs == HatTile::TY, "fused stencil thread layout");
static_assert(4 * (sizeof(HatTile::Smem) + 1024) <= 228 * 1024, "four blocks of the fused stencil on an SM");
__device__ __forceinline__ int mod3(int p) { return ((p % 3) + 3) % 3; }

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned a, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned a, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned a, unsigned parity)
{
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_wait(unsigned a, unsigned parity, int limit)
{
    for (int it = 0; it < limit; it++)
        if (mbar_try(a, parity)) return true;
    return false;
}
__device__ __forceinline__ void tma_load4(unsigned dst, const CUtensorMap *m, int c0, int c1, int c2, int c3,
                                          unsigned mb)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];\n" ::"r"(dst),
        "l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(mb)
        : "memory");
}
__device__ __forceinline__ void tma_load3(unsigned dst, const CUtensorMap *m, int c0, int c1, int c2, unsigned mb)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(dst),
        "l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(mb)
        : "memory");
}

// Before a barrier after which a copy may go into a slot: the thread's reads of
// the slot are done.  Tensor copies write through the async proxy, which a
// barrier alone does not order after the reads of other threads through the
// generic one, so a value read before the barrier and used after it may be
// fetched late, from the plane that took its place.
__device__ __forceinline__ void slots_read() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// grad-div potential of node (ni, nj) of the tile (global i, j) at plane p:
// the sums of k_gd_phi (mode 0) in the same order, from the staged planes
template <typename Tile>
__device__ __forceinline__ float2 tma_phi_node(const typename Tile::Smem &sm, const Geo<float> &g, int i, int j, int p,
                                               int ni, int nj, float dX, float dY, float dZ)
{
    if (!(i >= 1 && i <= g.nx - 1 && j >= 1 && j <= g.ny - 1 && p >= 1 && p <= g.nz - 1)) return make_float2(0, 0);
    constexpr int FW = Tile::FW, SW = Tile::SW, cf = Tile::FR * FW, cs = Tile::FR * SW;
    const int sp = p & 3, sz = (p - 1) & 3;
    const float2 *F = reinterpret_cast<const float2 *>(sm.fld[sp]);
    const float2 *Fz = reinterpret_cast<const float2 *>(sm.fld[sz]) + 2 * cf;
    const float *S = reinterpret_cast<const float *>(sm.sig[p % 3]);
    const float *Sz = reinterpret_cast<const float *>(sm.sig[(p - 1) % 3]) + 2 * cs;
    const float wn = reinterpret_cast<const float *>(sm.nod[p & 1])[nj * Tile::NW + ni];
    const int h = (nj + 1) * FW + ni + 2, hs = (nj + 1) * SW + ni + 1;
    const float dfa0 = dY * dZ, dfa1 = dX * dZ, dfa2 = dX * dY;
    float2 acc;
    if (wn < 0.f) {  // earth node: C = sigma_E
        acc = cscale(F[h - 1], dfa0 * S[hs - 1]);                    // Ex(i-1, j, p)
        acc = csub(acc, cscale(F[h], dfa0 * S[hs]));                  // Ex(i, j, p)
        acc = cadd(acc, cscale(F[cf + h - FW], dfa1 * S[cs + hs - SW]));  // Ey(i, j-1, p)
        acc = csub(acc, cscale(F[cf + h], dfa1 * S[cs + hs]));        // Ey(i, j, p)
        acc = cadd(acc, cscale(Fz[h], dfa2 * Sz[hs]));                // Ez(i, j, p-1)
        acc = csub(acc, cscale(F[2 * cf + h], dfa2 * S[2 * cs + hs]));  // Ez(i, j, p)
        return cscale(acc, -wn);
    }
    acc = cscale(F[h - 1], dfa0);
    acc = csub(acc, cscale(F[h], dfa0));
    acc = cadd(acc, cscale(F[cf + h - FW], dfa1));
    acc = csub(acc, cscale(F[cf + h], dfa1));
    acc = cadd(acc, cscale(Fz[h], dfa2));
    acc = csub(acc, cscale(F[2 * cf + h], dfa2));
    return cscale(acc, wn);
}

// tile (i0, j0) of column-tile bx, and node planes [k0, k1) of chunk bz of gz
template <typename Tile> __device__ __forceinline__ void tma_tile_at(const ColMap &m, int bx, int &i0, int &j0)
{
    i0 = (bx % m.tiles_x) * Tile::TX;
    j0 = (bx / m.tiles_x) * Tile::TY;
}
__device__ __forceinline__ void tma_range_at(int nz, int bz, int gz, int &k0, int &k1)
{
    const int kc = (nz + 1 + gz - 1) / gz;
    k0 = bz * kc;
    k1 = min(k0 + kc, nz + 1);
}
template <typename Tile> __device__ __forceinline__ typename Tile::Smem &tma_smem()
{
    extern __shared__ __align__(128) unsigned char tma_raw[];
    return *reinterpret_cast<typename Tile::Smem *>(tma_raw);
}

// the chunk count of stagekernels.cu, for the resident blocks of these
// kernels; `slot` identifies the kernel (its shared-memory attribute is set
// the first time its slot is seen), so every kernel needs its own slot
constexpr int kTmaSlots = 24;
template <typename K> inline int tma_resident(K kern, size_t smem, int slot, int threads = kThreads)
{
    static std::mutex mu;
    static int occ[64][kTmaSlots] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    std::lock_guard<std::mutex> lock(mu);
    if (!occ[dev][slot]) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        int n = 0, sms = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        occ[dev][slot] = std::max(1, n) * std::max(1, sms);
    }
    return occ[dev][slot];
}

}  // namespace mt3d
