// kernels_dmma.cu -- native FP64 and complex128 GEMM on the FP64 tensor pipe.
//
// Replaces the per-tile cublasDgemm / cublasZgemm call of the reference
// (blas/blasx_dgemm.c:87-95, blas/blasx_zgemm.c:88) with a hand-written
// sm_100a kernel built on DMMA (mma.sync m16n8k{4,8,16}, f64 in, f64
// accumulate).
//
// The tile itself (DMMA fragments, the cp.async ring, the alpha / beta
// epilogue) is dmma_tile.cuh, shared with the serving executor; this file
// holds the launches, with the CTA geometry and the k split chosen by an
// estimate of the time.
#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "dmma_tile.cuh"
#include "kernels.h"

namespace bx {

namespace {

using namespace dev;

template <bool CPLX, bool AKC, bool BKC, int KI, int G>
__global__ void __launch_bounds__(Tile<CPLX, G>::THREADS, Tile<CPLX, G>::PER_SM)
    dmma_gemm_kernel(const DmmaParams p) {
    if (p.guard && *p.guard != 0) return;  // the emulated path produced C
    extern __shared__ __align__(16) double smem[];
    dmma_tile<CPLX, AKC, BKC, KI, G>(p, blockIdx.x, smem);
}

// The emulated path's fallback: one resident set of CTAs that take tiles from
// a counter. It usually has nothing to do, and the exits of a CTA per tile took
// 6 us at 2048^3. A product that does fall back pays for the counter: 653 us
// there, 559 with a CTA per tile. (From four sets of tiles on it is a CTA per
// tile again: the counter cost 4096 x 3000 x 2500 2.6%, tiles dealt out in
// advance 6%, and the exits cost a large product less. A kernel of its own: the
// loop in the plain one made that 3% slower.)
template <bool CPLX, bool AKC, bool BKC, int KI, int G>
__global__ void __launch_bounds__(Tile<CPLX, G>::THREADS, Tile<CPLX, G>::PER_SM)
    dmma_queue_kernel(const DmmaParams p) {
    if (*p.guard != 0) return;
    extern __shared__ __align__(16) double smem[];
    __shared__ int s_tile;
    const int tiles = p.tiles_m * p.tiles_n;
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(p.queue, 1);
        __syncthreads();
        const int tile = s_tile;
        if (tile >= tiles) break;
        dmma_tile<CPLX, AKC, BKC, KI, G>(p, tile, smem);
        __syncthreads();  // the next tile's copies reuse the stages, its claim s_tile
    }
    // every CTA draws one number past the tiles; the last of them resets the counter
    if (threadIdx.x == 0 && s_tile == tiles + int(gridDim.x) - 1) atomicExch(p.queue, 0);
}

// One C tile per cluster, its k extent cut over the cluster's CTAs.
template <bool CPLX, bool AKC, bool BKC, int KI, int G>
__global__ void __launch_bounds__(Tile<CPLX, G>::THREADS, Tile<CPLX, G>::PER_SM)
    dmma_split_kernel(const DmmaParams p, int splits) {
    if (p.guard && *p.guard != 0) return;  // uniform
    extern __shared__ __align__(16) double smem[];
    dmma_tile<CPLX, AKC, BKC, KI, G, true>(p, blockIdx.x / splits, smem, blockIdx.x % splits, splits);
}

int num_sms() {
    static const int sms = [] {
        int dev = 0, n = 148;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            n = 148;
        return n;
    }();
    return sms;
}

// Shared memory of a CTA that leaves an SM two of them.
constexpr size_t kTwoPerSm = 100 * 1024;

template <bool CPLX, bool AKC, bool BKC, int KI, int G>
int launch_cfg(const DmmaParams &p, int splits, cudaStream_t s, size_t least_smem) {
    using TL = Tile<CPLX, G>;
    constexpr size_t need = dmma_smem_bytes<CPLX, AKC, BKC, G>();
    static_assert(need <= 227 * 1024, "shared memory budget");
    const size_t smem = std::max(need, least_smem);
    const int64_t tiles = int64_t(p.tiles_m) * p.tiles_n;
    if constexpr (G == 2) {
        if (splits > 1) {
            auto kern = dmma_split_kernel<CPLX, AKC, BKC, KI, G>;
            BX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
            BX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            cudaLaunchAttribute at;
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = unsigned(splits);
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(unsigned(tiles * splits));
            cfg.blockDim = dim3(TL::THREADS);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = s;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            BX_CUDA(cudaLaunchKernelEx(&cfg, kern, p, splits));
            count_launch();
            return BLASX_OK;
        }
    }
    auto kern = dmma_gemm_kernel<CPLX, AKC, BKC, KI, G>;
    int64_t grid = tiles;
    if constexpr (G != 0 && (CPLX || KI == 16)) {
        const int64_t set = int64_t(least_smem ? 2 : TL::PER_SM) * num_sms();
        if (p.guard && p.queue && tiles <= 4 * set) {
            kern = dmma_queue_kernel<CPLX, AKC, BKC, KI, G>;
            grid = std::min(tiles, set);
        }
    }
    BX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    kern<<<unsigned(grid), TL::THREADS, smem, s>>>(p);
    BX_CUDA(cudaGetLastError());
    count_launch();
    return BLASX_OK;
}

// Instruction K of the FP64 MMA with the 64x64 and 128x128 tiles: 16 by
// default (BLASX_DMMA_K = 4, 8 or 16).
int dmma_k() {
    static const int k = [] {
        const char *e = getenv("BLASX_DMMA_K");
        const int v = e ? atoi(e) : 16;
        return (v == 4 || v == 8) ? v : 16;
    }();
    return k;
}

// The tile geometry and the k split of one problem.
struct Geometry {
    int g, splits, per_sm;
};

// Chosen by the estimated time in SM cycles. An SM does 64 FP64 multiply-adds
// per cycle; with n CTAs of a tile resident it reaches the fraction eff[n] of
// that, measured per tile (few warps cannot cover the shared-memory and
// barrier latencies: one 64x64 CTA alone reaches 55%, three 87%). A grid runs
// as full rounds of PER_SM CTAs on every SM and one more with what is left.
// Cutting k over a cluster costs about 8000 cycles (the exchange of the partial
// tiles and the cluster launch: 512^3 took 18.6 us with a cut of 2 against
// 16.6 without), so it is for fewer tiles than SMs with a long k: 96 x 64 x
// 11904 fell from 590 us (two 64x64 tiles) to 33 with a cut of 8.
// BLASX_DMMA_TILE = 32, 48 (64x48), 64 or 128 forces an FP64 tile.
struct TileModel {
    int g, bm, bn, per_sm;
    double eff[4];
};
constexpr double kSplitCycles = 8000.0;
// (64x64 FP64 tiles also two to an SM, by more shared memory than they need:
// 585 of them are two such rounds, but one of three per SM and a third of one
// that reaches 55%.)
constexpr TileModel kReal[] = {{1, 64, 64, 3, {0.55, 0.79, 0.87, 0}},
                               {1, 64, 64, 2, {0.55, 0.77, 0, 0}},
                               {3, 64, 48, 4, {0.53, 0.73, 0.77, 0.85}},
                               {2, 32, 32, 4, {0.43, 0.61, 0.70, 0.72}},
                               {0, 128, 128, 1, {0.78, 0, 0, 0}}};  // a single, nearly full wave
constexpr TileModel kCplx[] = {{1, 64, 64, 2, {0.72, 0.86, 0, 0}}, {2, 32, 32, 4, {0.56, 0.76, 0.80, 0.83}}};

// Whether an operand with this base and leading dimension is copied 16 bytes
// at a time (as DmmaParams::vec_a).
bool wide_copies(const void *p, int64_t ld) { return ld % 2 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// What a tile loses against its fraction on some layouts of the operands, in
// full rounds (n = 0) or in the last one with n CTAs of it per SM.
// Two k-contiguous operands: 32x32 FP64 tiles 15%, 64x64 complex128 tiles 20%
// (3000 x 3000 x 200: 634 us, 520 with 32x32 tiles; 2496 x 3072 x 83: 296 and
// 230; the 64x128 tile, which served them before, 583 and 270).
// FP64 operands that are m- or n-contiguous and copied 8 bytes at a time (odd
// leading dimension): a smaller tile copies more of them per multiply-add, 6%
// each against 64x64 (1000^3 NT: 32x32 tiles 111 us, 64x64 95; with even ones
// 89 and 85), which lose 5% with three per SM in the last round (9832 x 116 x
// 721 NN, odd: 105 us, 32x32 93).
// 64x48 tiles of two such operands (NT) cover their latencies badly with one
// or two CTAs per SM, whatever the copies (1003 x 777 x 641, odd: 70.5 us,
// 64x64 64.2).
double layout_cost(const TileModel &m, double macs, const Gemm &g, int64_t n) {
    const bool a_k = g.ta != NoTrans, b_k = g.tb == NoTrans;
    if (macs != 1.0) return m.g == 1 && a_k && b_k ? 1.2 : 1.0;
    const int narrow = (!a_k && !wide_copies(g.A, g.lda)) + (!b_k && !wide_copies(g.B, g.ldb));
    if (m.g == 1) return narrow && n == 3 ? 1.05 : 1.0;
    if (m.g == 0) return 1.0;
    double cost = 1.0 + (m.g == 2 ? 0.06 : 0.065) * narrow;
    if (m.g == 2 && a_k && b_k) cost *= 1.15;
    if (m.g == 3 && !a_k && !b_k && (n == 1 || n == 2)) cost *= 1.12;
    return cost;
}

template <int COUNT> Geometry pick_geometry(const TileModel (&models)[COUNT], double macs, const Gemm &g) {
    const int64_t sms = num_sms();
    Geometry best{models[0].g, 1, models[0].per_sm};
    double best_t = 1e300;
    for (const TileModel &m : models) {
        int64_t tiles = ((g.M + m.bm - 1) / m.bm) * ((g.N + m.bn - 1) / m.bn);
        if (g.uplo) tiles = (tiles + 1) / 2;  // about half of a triangle's tiles compute
        const int max_splits = m.g == 2 ? 16 : 1;
        for (int s = 1; s == 1 || (s <= max_splits && g.K >= int64_t(32) * s && tiles < sms); s *= 2) {
            const int64_t ctas = tiles * s, round = sms * m.per_sm, rest = ctas % round;
            const int64_t n = (rest + sms - 1) / sms;
            const double share = macs * m.bm * m.bn * double((g.K + s - 1) / s) / 64.0;
            const double t = share * (layout_cost(m, macs, g, 0) * double(ctas / round) * m.per_sm /
                                          m.eff[m.per_sm - 1] +
                                      (n ? layout_cost(m, macs, g, n) * double(n) / m.eff[n - 1] : 0.0)) +
                             (s > 1 ? kSplitCycles : 0.0);
            if (t < best_t) {
                best_t = t;
                best = Geometry{m.g, s, m.per_sm};
            }
        }
    }
    return best;
}

int forced_tile() {
    static const int forced = [] {
        const char *e = getenv("BLASX_DMMA_TILE");
        switch (e ? atoi(e) : 0) {
            case 32: return 2;
            case 48: return 3;
            case 64: return 1;
            case 128: return 0;
            default: return -1;
        }
    }();
    return forced;
}

template <bool CPLX, int KI, int G> int launch_g(const Gemm &g, int splits, cudaStream_t s, size_t least_smem = 0) {
    const DmmaParams p = make_params<CPLX, G>(g);
    if (int64_t(p.tiles_m) * p.tiles_n * splits > INT32_MAX)
        return set_error(BLASX_ERR_UNSUPPORTED, "DMMA grid too large");
    const bool akc = g.ta != NoTrans;  // op(A) = A^T: stored K x M, k contiguous
    const bool bkc = g.tb == NoTrans;  // op(B) = B: stored K x N, k contiguous
    if (akc)
        return bkc ? launch_cfg<CPLX, true, true, KI, G>(p, splits, s, least_smem)
                   : launch_cfg<CPLX, true, false, KI, G>(p, splits, s, least_smem);
    return bkc ? launch_cfg<CPLX, false, true, KI, G>(p, splits, s, least_smem)
               : launch_cfg<CPLX, false, false, KI, G>(p, splits, s, least_smem);
}

template <int G> int launch_k(const Gemm &g, cudaStream_t s) {
    switch (dmma_k()) {
        case 4: return launch_g<false, 4, G>(g, 1, s);
        case 8: return launch_g<false, 8, G>(g, 1, s);
        default: return launch_g<false, 16, G>(g, 1, s);
    }
}

int launch_real(const Gemm &g, cudaStream_t s) {
    Geometry x = pick_geometry(kReal, 1.0, g);
    if (forced_tile() >= 0) x = Geometry{forced_tile(), 1, 0};
    switch (x.g) {
        case 0: return launch_k<0>(g, s);
        case 1: return x.per_sm == 2 ? launch_g<false, 16, 1>(g, 1, s, kTwoPerSm) : launch_k<1>(g, s);
        case 3: return launch_g<false, 16, 3>(g, 1, s);
        default: return launch_g<false, 16, 2>(g, x.splits, s);
    }
}

int launch_cplx(const Gemm &g, cudaStream_t s) {
    const Geometry x = pick_geometry(kCplx, 4.0, g);
    return x.g == 1 ? launch_g<true, 8, 1>(g, 1, s) : launch_g<true, 4, 2>(g, x.splits, s);
}

}  // namespace

bool dmma_supported(const Gemm &g) {
    return (g.dt == DType::F64 || g.dt == DType::C128) && g.M <= INT32_MAX && g.N <= INT32_MAX &&
           g.K <= INT32_MAX;
}

int launch_gemm_dmma(const Gemm &g, cudaStream_t s) {
    if (g.dt == DType::F64) return launch_real(g, s);
    if (g.dt == DType::C128) return launch_cplx(g, s);
    return set_error(BLASX_ERR_UNSUPPORTED, "DMMA kernel handles FP64 and complex128 only");
}

}  // namespace bx
