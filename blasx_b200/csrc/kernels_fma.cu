// kernels_fma.cu -- native FP32 and complex64 GEMM on the CUDA cores: the
// launches of the tiles of fma_tile.cuh.
#include <algorithm>
#include <cstdint>

#include "fma_tile.cuh"
#include "kernels.h"

namespace bx {
namespace {

using namespace dev;

// The tiles (outputs, groups a k-step is cut over, k-step, stages) and the
// CTAs per SM they are compiled for. Measured, FP32 / complex64:
//                         320x257x190   512^3   2048x2048x200   4096x4096x1024
//   kWide  32x32, 8 groups    6.4 us    14.5      86 / --          1089
//   kSmall 32x32, 4 groups    8.4       14.5      70               1036
//   kLarge 64x64, 1 group    14.2       25.3      51                852
//   before: 64x64 (128x128)  33.0       82.0      92 (60)         1516 (850)
//   complex64, 211x300x257: 16.5 / 18.6, cut over 4 CTAs 14.5; before 61.6;
//   512^3 35-38, before 113; 2048x2048x512 449 (kSmall), 64x64 SIMT tile 433.
template <typename T> struct Cfg;
template <> struct Cfg<float> {
    using Wide = FmaTile<float, 1, 1, 8, 64, 2>;
    using Small = FmaTile<float, 1, 1, 4, 32, 4>;
    using Large = FmaTile<float, 2, 2, 1, 16, 4>;
    static constexpr int small_per_sm = 4;
    static constexpr int64_t min_k = 256;  // least k per CTA of a cluster
};
template <> struct Cfg<c2> {
    using Wide = FmaTile<c2, 1, 1, 8, 64, 2>;
    using Small = FmaTile<c2, 1, 1, 4, 32, 4>;
    static constexpr int small_per_sm = 2;
    static constexpr int64_t min_k = 64;
};

template <typename TL, typename T, bool AKC, bool BKC, int PER_SM>
__global__ void __launch_bounds__(TL::THREADS, PER_SM) fma_gemm_kernel(const FmaParams<T> p, const int *guard) {
    if (guard && *guard != 0) return;  // the emulated path produced C
    extern __shared__ __align__(16) unsigned char smem[];
    fma_tile<TL, T, AKC, BKC, false>(p, blockIdx.x, reinterpret_cast<T *>(smem), 0, 1);
}

// The emulated path's fallback: a resident set of CTAs that take tiles from
// the counter, as dmma_queue_kernel.
template <typename TL, typename T, bool AKC, bool BKC, int PER_SM>
__global__ void __launch_bounds__(TL::THREADS, PER_SM)
    fma_queue_kernel(const FmaParams<T> p, const int *guard, int *queue) {
    if (*guard != 0) return;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_tile;
    const int tiles = p.tiles_m * p.tiles_n;
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(queue, 1);
        __syncthreads();
        const int tile = s_tile;
        if (tile >= tiles) break;
        fma_tile<TL, T, AKC, BKC, false>(p, tile, reinterpret_cast<T *>(smem), 0, 1);
        __syncthreads();  // the next tile's copies reuse the stages, its claim s_tile
    }
    if (threadIdx.x == 0 && s_tile == tiles + int(gridDim.x) - 1) atomicExch(queue, 0);
}

// One tile per cluster, its k extent cut over the cluster's CTAs.
template <typename TL, typename T, bool AKC, bool BKC>
__global__ void __launch_bounds__(TL::THREADS)
    fma_split_kernel(const FmaParams<T> p, const int *guard, int splits) {
    if (guard && *guard != 0) return;  // uniform
    extern __shared__ __align__(16) unsigned char smem[];
    fma_tile<TL, T, AKC, BKC, true>(p, blockIdx.x / splits, reinterpret_cast<T *>(smem), blockIdx.x % splits, splits);
}

constexpr int kSms = 148;

// Bytes per copy of an operand with this base and leading dimension.
template <typename T> int copy_width(const void *p, int64_t ld) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p) | uintptr_t(ld * int64_t(sizeof(T)));
    return a % 16 == 0 ? 16 : a % 8 == 0 ? 8 : 4;
}

template <typename TL, typename T> FmaParams<T> params(const Gemm &g) {
    FmaParams<T> p;
    p.s = SimtParams<T>{g.ta, g.tb, int(g.M), int(g.N), int(g.K), from_cplx<T>(g.alpha), from_cplx<T>(g.beta),
                        static_cast<const T *>(g.A), g.lda, static_cast<const T *>(g.B), g.ldb,
                        static_cast<T *>(g.C), g.ldc, g.beta_zero() ? 1 : 0, g.uplo, g.diag};
    p.tiles_m = int((g.M + TL::BM - 1) / TL::BM);
    p.tiles_n = int((g.N + TL::BN - 1) / TL::BN);
    p.wa = copy_width<T>(g.A, g.lda);
    p.wb = copy_width<T>(g.B, g.ldb);
    return p;
}

template <typename TL, typename T, bool AKC, bool BKC, int PER_SM>
int launch_tile(const Gemm &g, int splits, cudaStream_t s) {
    const FmaParams<T> p = params<TL, T>(g);
    const int64_t tiles = int64_t(p.tiles_m) * p.tiles_n;
    if (tiles * splits > INT32_MAX) return set_error(BLASX_ERR_UNSUPPORTED, "FMA grid too large");
    constexpr size_t smem = fma_smem_bytes<TL, T, AKC, BKC>();
    if constexpr (TL::KS == 4) {
        if (splits > 1) {
            auto kern = fma_split_kernel<TL, T, AKC, BKC>;
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
            BX_CUDA(cudaLaunchKernelEx(&cfg, kern, p, g.guard, splits));
            count_launch();
            return BLASX_OK;
        }
    }
    const int64_t set = int64_t(PER_SM) * kSms;
    if (g.guard && g.queue && tiles <= 4 * set) {
        auto kern = fma_queue_kernel<TL, T, AKC, BKC, PER_SM>;
        BX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        kern<<<unsigned(std::min(tiles, set)), TL::THREADS, smem, s>>>(p, g.guard, g.queue);
    } else {
        auto kern = fma_gemm_kernel<TL, T, AKC, BKC, PER_SM>;
        BX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        kern<<<unsigned(tiles), TL::THREADS, smem, s>>>(p, g.guard);
    }
    BX_CUDA(cudaGetLastError());
    count_launch();
    return BLASX_OK;
}

template <typename TL, typename T, int PER_SM> int launch_layout(const Gemm &g, int splits, cudaStream_t s) {
    const bool akc = g.ta != NoTrans, bkc = g.tb == NoTrans;
    if (akc) return bkc ? launch_tile<TL, T, true, true, PER_SM>(g, splits, s) : launch_tile<TL, T, true, false, PER_SM>(g, splits, s);
    return bkc ? launch_tile<TL, T, false, true, PER_SM>(g, splits, s) : launch_tile<TL, T, false, false, PER_SM>(g, splits, s);
}

template <typename T> int launch_t(const Gemm &g, cudaStream_t s) {
    using C = Cfg<T>;
    auto tiles = [&](int64_t edge) {
        const int64_t t = ((g.M + edge - 1) / edge) * ((g.N + edge - 1) / edge);
        return g.uplo ? (t + 1) / 2 : t;  // about half of a triangle's tiles compute
    };
    const int64_t t32 = tiles(32);
    // fewer tiles than SMs: cut k while the CTAs stay within two per SM and
    // keep min_k each (FP32 96 x 64 x 9000: 117 us whole, 23 cut over 8)
    int splits = 1;
    while (t32 < kSms && splits < 16 && t32 * 2 * splits <= 2 * kSms && g.K >= C::min_k * 2 * splits) splits *= 2;
    if (splits > 1) return launch_layout<typename C::Small, T, C::small_per_sm>(g, splits, s);
    // up to two 32x32 tiles per SM leave registers and issue slots for 8 groups
    if (t32 <= 2 * kSms) return launch_layout<typename C::Wide, T, sizeof(T) == 4 ? 2 : 1>(g, 1, s);
    if constexpr (sizeof(T) == 4) {
        // 64x64 tiles once they give every SM three (900 x 700 x 400, 165 of
        // them: 33 us with 32x32 tiles, 39 with 64x64)
        if (tiles(64) >= 3 * kSms) return launch_layout<typename C::Large, T, 4>(g, 1, s);
    }
    return launch_layout<typename C::Small, T, C::small_per_sm>(g, 1, s);
}

}  // namespace

bool fma_preferred(const Gemm &g) {
    if (g.dt == DType::F32) return (g.N + 127) / 128 <= 65535;
    // complex64: the 64x64 SIMT tile from three of them per two SMs on
    // (1394 x 699 x 66, 242 tiles: 35 us, 45 with 32x32 tiles; 512^3, 64
    // tiles: 113 against 35)
    return g.dt == DType::C64 && 2 * ((g.M + 63) / 64) * ((g.N + 63) / 64) < 3 * kSms && (g.N + 63) / 64 <= 65535;
}

int launch_gemm_fma(const Gemm &g, cudaStream_t s) {
    return g.dt == DType::F32 ? launch_t<float>(g, s) : launch_t<c2>(g, s);
}

}  // namespace bx
