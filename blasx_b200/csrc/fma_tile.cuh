// fma_tile.cuh -- the native FP32 / complex64 GEMM tile on the CUDA cores of
// the standalone kernels (kernels_fma.cu).
//
// What bounds a small product is not arithmetic: it is how many SMs get a
// tile and how long a tile's chain of loads is. So the tiles are small (32x32
// or 64x64), operands stream through a cp.async ring several k-steps ahead,
// and the k extent is shared: each k-step is cut over KS groups of warps of a
// CTA, and for few tiles the whole extent over the CTAs of a cluster; the
// partial tiles are added in a fixed order through shared memory.
//
// A warp computes 32x32 outputs, a thread 8x4 of them: lane = 8 mg + ng holds
// 8 rows and 4 columns. Each operand keeps its contiguity: a k-contiguous
// source lands as [row][k], else as [k][row], rows padded by 16 bytes, and is
// read back in 16-byte words (VE elements) along its contiguous direction, so
// 32 multiply-adds per k take three of them (float).
//
// Copies are 16 bytes wide where leading dimension and base allow it, else 8
// or 4; the source-size operand of cp.async fills with zeros what lies beyond
// M, N or K, and nothing outside the matrices is read.
#pragma once

#include <cstdint>

#include "dmma_tile.cuh"
#include "simt_tile.cuh"

namespace bx {
namespace dev {

template <typename T> struct FmaParams {
    SimtParams<T> s;
    int tiles_m, tiles_n;
    int wa, wb;  // bytes per copy: 16, 8 or 4
};

// A tile of 32 WM x 32 WN outputs, each k-step of BK cut over KS groups of
// WM x WN warps, in a ring of STAGES k-steps.
template <typename T, int WM_, int WN_, int KS_, int BK_, int STAGES_> struct FmaTile {
    static constexpr int WM = WM_, WN = WN_, KS = KS_, BK = BK_, STAGES = STAGES_;
    static constexpr int BM = 32 * WM, BN = 32 * WN, THREADS = 32 * WM * WN * KS, KG = BK / KS;
    static constexpr int VE = 16 / int(sizeof(T));  // elements per 16 bytes
    static_assert(KG % VE == 0, "a group's share of a k-step is whole 16-byte words");
};

// Shared-memory geometry of an operand tile of R rows (elements of T).
template <typename TL, typename T, int R, bool KC> struct FmaOp {
    static constexpr int stride = (KC ? TL::BK : R) + TL::VE;
    static constexpr int size = KC ? R * stride : TL::BK * stride;
    __device__ static int idx(int r, int k) { return KC ? r * stride + k : k * stride + r; }
};

template <typename TL, typename T, bool AKC, bool BKC> constexpr size_t fma_smem_bytes() {
    const size_t ring = size_t(TL::STAGES) * (FmaOp<TL, T, TL::BM, AKC>::size + FmaOp<TL, T, TL::BN, BKC>::size);
    const size_t part = size_t(TL::KS) * TL::BN * (TL::BM + TL::VE);
    return (ring > part ? ring : part) * sizeof(T);
}

template <int BYTES> __device__ __forceinline__ void fma_copy(uint32_t dst, const void *src, int valid) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(valid) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;\n" ::"r"(dst), "l"(src), "r"(valid), "n"(BYTES)
                     : "memory");
}

// Copies the R x BK tile at (r0, k0) of an operand (as load_tile of
// dmma_tile.cuh), W bytes per copy.
template <typename TL, typename T, int R, bool KC, int W>
__device__ __forceinline__ void fma_load(uint32_t sbase, const T *src, int64_t ld, int r0, int k0, int rows, int kdim,
                                         int tid) {
    using S = FmaOp<TL, T, R, KC>;
    constexpr int V = W >= int(sizeof(T)) ? W / int(sizeof(T)) : 1;  // elements per chunk
    constexpr int PARTS = W >= int(sizeof(T)) ? 1 : int(sizeof(T)) / W;
    constexpr int CHUNKS = R * TL::BK / V, PER_ROW = KC ? TL::BK / V : R / V;
#pragma unroll
    for (int i = 0; i < (CHUNKS + TL::THREADS - 1) / TL::THREADS; ++i) {
        const int e = tid + i * TL::THREADS;
        if (CHUNKS % TL::THREADS != 0 && e >= CHUNKS) break;
        const int c = (e % PER_ROW) * V, o = e / PER_ROW;
        const int r = KC ? o : c, k = KC ? c : o;
        const int gr = r0 + r, gk = k0 + k;
        int valid = KC ? (gr < rows ? min(V, kdim - gk) : 0) : (gk < kdim ? min(V, rows - gr) : 0);
        valid = max(valid, 0);
        const T *p = src + (valid ? (KC ? gk + int64_t(gr) * ld : gr + int64_t(gk) * ld) : 0);
        const uint32_t dst = sbase + uint32_t(S::idx(r, k)) * uint32_t(sizeof(T));
#pragma unroll
        for (int q = 0; q < PARTS; ++q)
            fma_copy<W>(dst + q * W, reinterpret_cast<const char *>(p) + q * W,
                        PARTS == 1 ? valid * int(sizeof(T)) : (valid ? W : 0));
    }
}

template <typename TL, typename T, int R, bool KC>
__device__ __forceinline__ void fma_load_any(int w, uint32_t sbase, const T *src, int64_t ld, int r0, int k0, int rows,
                                             int kdim, int tid) {
    if (w == 16) fma_load<TL, T, R, KC, 16>(sbase, src, ld, r0, k0, rows, kdim, tid);
    else if (sizeof(T) == 8 && w == 8) fma_load<TL, T, R, KC, 8>(sbase, src, ld, r0, k0, rows, kdim, tid);
    else fma_load<TL, T, R, KC, 4>(sbase, src, ld, r0, k0, rows, kdim, tid);
}

// A T of the shared memory of CTA `rank` of the cluster.
template <typename T> __device__ __forceinline__ T fma_cluster_read(const T *local, uint32_t rank) {
    uint32_t addr;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(local)), "r"(rank));
    T v;
    if constexpr (sizeof(T) == 4) {
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    } else {
        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.re), "=f"(v.im) : "r"(addr) : "memory");
    }
    return v;
}

// One C tile; with SPLIT, the share of CTA `rank` of a cluster of `splits`.
template <typename TL, typename T, bool AKC, bool BKC, bool SPLIT>
__device__ __forceinline__ void fma_tile(const FmaParams<T> &fp, int tile, T *smem, int rank, int splits) {
    using Ar = Arith<T>;
    constexpr int BM = TL::BM, BN = TL::BN, BK = TL::BK, ST = TL::STAGES, KG = TL::KG, VE = TL::VE;
    using SA = FmaOp<TL, T, BM, AKC>;
    using SB = FmaOp<TL, T, BN, BKC>;
    const SimtParams<T> &p = fp.s;
    T *sA = smem, *sB = smem + ST * SA::size;
    const int tm = tile % fp.tiles_m, tn = tile / fp.tiles_m;
    const int m0 = tm * BM, n0 = tn * BN;
    // triangular output: a tile with no entry inside computes nothing (uniform per CTA and cluster)
    if (p.uplo == 1 && int64_t(m0) - (n0 + BN - 1) > p.diag) return;
    if (p.uplo == 2 && int64_t(m0 + BM - 1) - n0 < p.diag) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = warp / (TL::WM * TL::WN), wm = warp % TL::WM, wn = warp / TL::WM % TL::WN;
    const int mg = lane >> 3, ng = lane & 7;
    // the rows and columns of this thread, matching the 16-byte reads
    auto row = [&](int i) { return wm * 32 + (AKC ? mg + 4 * i : i / VE * (4 * VE) + mg * VE + i % VE); };
    auto col = [&](int j) { return wn * 32 + (BKC ? ng + 8 * j : j / VE * (8 * VE) + ng * VE + j % VE); };

    const int kt_all = (p.K + BK - 1) / BK;
    const int kt0 = SPLIT ? int(int64_t(kt_all) * rank / splits) : 0;
    const int kts = SPLIT ? int(int64_t(kt_all) * (rank + 1) / splits) - kt0 : kt_all;
    auto load_stage = [&](int stage, int kt) {
        fma_load_any<TL, T, BM, AKC>(fp.wa, smem_u32(sA + stage * SA::size), p.A, p.lda, m0, kt * BK, p.M, p.K, tid);
        fma_load_any<TL, T, BN, BKC>(fp.wb, smem_u32(sB + stage * SB::size), p.B, p.ldb, n0, kt * BK, p.N, p.K, tid);
    };
    const bool conj_a = p.ta == ConjT, conj_b = p.tb == ConjT;

    T acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = Ar::zero();
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < kts) load_stage(s, kt0 + s);
        cp_async_commit();
    }
    for (int kt = 0; kt < kts; ++kt) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        if (kt + ST - 1 < kts) load_stage((kt + ST - 1) % ST, kt0 + kt + ST - 1);
        cp_async_commit();
        const T *a_s = sA + (kt % ST) * SA::size;
        const T *b_s = sB + (kt % ST) * SB::size;
#pragma unroll
        for (int kk = 0; kk < KG; kk += VE) {
            const int k = group * KG + kk;
            __align__(16) T a[8][VE], b[4][VE];
            __align__(16) T w[VE];
            if (AKC) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    *reinterpret_cast<float4 *>(a[i]) = *reinterpret_cast<const float4 *>(&a_s[SA::idx(row(i), k)]);
            } else {
#pragma unroll
                for (int v = 0; v < VE; ++v)
#pragma unroll
                    for (int i = 0; i < 8; i += VE) {
                        *reinterpret_cast<float4 *>(w) =
                            *reinterpret_cast<const float4 *>(&a_s[SA::idx(row(i), k + v)]);
#pragma unroll
                        for (int u = 0; u < VE; ++u) a[i + u][v] = w[u];
                    }
            }
            if (BKC) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    *reinterpret_cast<float4 *>(b[j]) = *reinterpret_cast<const float4 *>(&b_s[SB::idx(col(j), k)]);
            } else {
#pragma unroll
                for (int v = 0; v < VE; ++v)
#pragma unroll
                    for (int j = 0; j < 4; j += VE) {
                        *reinterpret_cast<float4 *>(w) =
                            *reinterpret_cast<const float4 *>(&b_s[SB::idx(col(j), k + v)]);
#pragma unroll
                        for (int u = 0; u < VE; ++u) b[j + u][v] = w[u];
                    }
            }
            if constexpr (sizeof(T) == 8) {
                if (conj_a) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int v = 0; v < VE; ++v) a[i][v] = Ar::conj(a[i][v]);
                }
                if (conj_b) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int v = 0; v < VE; ++v) b[j][v] = Ar::conj(b[j][v]);
                }
            }
#pragma unroll
            for (int v = 0; v < VE; ++v)
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = Ar::fma(a[i][v], b[j][v], acc[i][j]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();

    // partial tiles by columns, one per group, in place of the operand stages
    constexpr int LD = BM + VE, PART = BN * LD;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) smem[group * PART + col(j) * LD + row(i)] = acc[i][j];
    int c_lo = 0, c_hi = BN;
    if constexpr (SPLIT) {
        const int per = (BN + splits - 1) / splits;  // columns this CTA finishes
        c_lo = min(BN, rank * per);
        c_hi = min(BN, c_lo + per);
        dmma_cluster_sync();
    } else {
        __syncthreads();
    }
    // four entries at a time, their C values loaded before any is stored
    constexpr int BATCH = 4;
    const int entries = (c_hi - c_lo) * BM;
    for (int e0 = tid; e0 < entries; e0 += BATCH * TL::THREADS) {
        T cin[BATCH];
        bool in[BATCH];
#pragma unroll
        for (int b = 0; b < BATCH; ++b) {
            const int e = e0 + b * TL::THREADS;
            const int gm = m0 + e % BM, gn = n0 + c_lo + e / BM;
            in[b] = e < entries && gm < p.M && gn < p.N &&
                    !(p.uplo && (p.uplo == 1 ? gm - int64_t(gn) > p.diag : gm - int64_t(gn) < p.diag));
            cin[b] = in[b] && !p.beta_zero ? p.C[gm + gn * p.ldc] : Ar::zero();
        }
#pragma unroll
        for (int b = 0; b < BATCH; ++b) {
            if (!in[b]) continue;
            const int e = e0 + b * TL::THREADS, r = e % BM, c = c_lo + e / BM;
            T v = Ar::zero();
            if constexpr (SPLIT) {
                for (int q = 0; q < splits; ++q)
#pragma unroll
                    for (int g = 0; g < TL::KS; ++g)
                        v = Ar::add(v, fma_cluster_read(&smem[g * PART + c * LD + r], uint32_t(q)));
            } else {
#pragma unroll
                for (int g = 0; g < TL::KS; ++g) v = Ar::add(v, smem[g * PART + c * LD + r]);
            }
            v = Ar::mul(p.alpha, v);
            if (!p.beta_zero) v = Ar::add(v, Ar::mul(p.beta, cin[b]));
            p.C[m0 + r + (n0 + c) * p.ldc] = v;
        }
    }
    if constexpr (SPLIT) dmma_cluster_sync();  // no CTA leaves while another reads its partial tiles
}

}  // namespace dev
}  // namespace bx
