// trsm.cu -- triangular solve (cblas_?trsm) and triangular multiply
// (cblas_?trmm) with many right-hand sides on device operands.
//
// op(A) X = alpha B (left) or X op(A) = alpha B (right) is solved by
// recursive halving of the order-K triangle: solve the first half, update
// the second half's right-hand sides with one GEMM (device_gemm: native, or
// emulated on the INT8 tensor cores where the precision mode selects it),
// solve the second half. The top-level updates carry most of the K^2 * (M or
// N) work with K up to K/2, the shape the emulated GEMM needs; blocks of at
// most 256 rows are solved by substitution in one kernel.
//
// Every GEMM reads op(A) only in an off-diagonal rectangle inside the stored
// triangle, and the substitution kernel reads only the stored triangle of its
// diagonal block (not the diagonal when it is unit): the other triangle of A
// is never read.
#include <algorithm>

#include "arith.cuh"
#include "kernels.h"

namespace bx {
namespace {

// Geometry of the substitution kernel. A warp holds a few right-hand-side
// vectors of a block of kBlock rows in registers: lane l owns rows l, l + 32,
// ... of each.
constexpr int kBlock = 256, kRows = kBlock / 32;
constexpr int kBlockThreads = 256;
constexpr int kSms = 148;
constexpr int kPanelLd = kBlock + 1;
// Columns of S staged at a time (PANEL): 16, and 8 for complex128 with more
// CTAs than SMs, where two panels of 16 (135 KB) leave an SM one CTA (256 x
// 4096 199 us, 163 with 8; 2048 x 8192 4.62 ms, 4.07). With an SM to itself a
// CTA is better off with fewer barriers (2048 x 64: 498 us, 538 with 8).
constexpr int kPanel = 16, kSmallPanel = 8;
// Vectors per warp: 16 bytes of each row per lane (32 registers in all).
template <typename T> struct Vecs {
    static constexpr int n = 16 / int(sizeof(T));
};

template <typename T> __device__ inline T negate(T a) { return -a; }
template <> __device__ inline z2 negate<z2>(z2 a) { return {-a.re, -a.im}; }
template <> __device__ inline c2 negate<c2>(c2 a) { return {-a.re, -a.im}; }

template <typename T> __device__ inline T shfl(T v, int src) { return __shfl_sync(0xffffffffu, v, src); }
template <> __device__ inline z2 shfl<z2>(z2 v, int src) {
    return {__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src)};
}
template <> __device__ inline c2 shfl<c2>(c2 v, int src) {
    return {__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src)};
}

// One scalar of shared memory from global memory, or zero.
template <typename T> __device__ __forceinline__ void copy_or_zero(T *dst, const T *src, bool in) {
    using R = typename Arith<T>::R;
    constexpr int RW = int(sizeof(R)), PARTS = int(sizeof(T)) / RW;
#pragma unroll
    for (int q = 0; q < PARTS; ++q)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;\n" ::"r"(
                         uint32_t(__cvta_generic_to_shared(dst)) + q * RW),
                     "l"(reinterpret_cast<const char *>(src) + q * RW), "r"(in ? RW : 0), "n"(RW)
                     : "memory");
}

// Solves S x = c for nvec vectors at once, S the bs x bs (bs <= kBlock) system
// matrix of one diagonal block: S = op(A_block) for a left solve, the
// transpose of op(A_block) for a right solve (x op(A) = c is op(A)^T x^T =
// c^T). S[i][k] is A[i + k lda] (s_trans = 0) or A[k + i lda] (s_trans = 1),
// conjugated when s_conj. S is lower (FORWARD substitution) or upper; only
// that triangle of S, and its diagonal unless UNIT, is read. Vector v,
// element i: left: C[i + v ldc] (columns of B); right: C[v + i ldc] (rows of
// B). Each vector is scaled by `scale` (alpha) on load.
//
// What bounds it: the chain of bs dependent steps of each vector (a
// reciprocal multiply, a shuffle and a multiply-add; about 210 cycles a step
// with the barrier and the copies of its panel), and beside it the FP64 pipe. So a block is as tall as its vectors fit in registers, one
// launch instead of four substitutions of 64 rows with three updates between
// them; every warp runs its own vectors, the rows after step k updated by all
// lanes at once, and a step needs no barrier. S passes through shared memory
// a few columns at a time (cp.async, the next panel in flight), zero outside its
// triangle and beyond bs; the CTA's warps share it. Rows beyond bs are zero
// vectors with a unit diagonal. FP64, 256 rows: 28.5 us for 2048 vectors (87
// as four 64-row substitutions and their updates), 132 for 16384 (136); a
// DTRSM of 4096 rows and 2048 vectors fell from 2083 to 1417 us. Four vectors
// per lane and four warps per CTA took 79 us for 2048: with one warp per
// scheduler every instruction's latency shows.
template <typename T, bool FORWARD, bool UNIT, int PANEL>
__global__ void __launch_bounds__(kBlockThreads)
    trsm_block_kernel(const T *__restrict__ A, int64_t lda, T *__restrict__ C, int64_t ldc, int bs, int64_t nvec,
                      int left, int s_trans, int s_conj, T scale) {
    using Ar = Arith<T>;
    constexpr int NV = Vecs<T>::n, TH = kBlockThreads, WARPS = TH / 32;
    static_assert(TH == kBlock, "a thread loads one row of a panel");
    extern __shared__ __align__(16) unsigned char smem[];
    T *P = reinterpret_cast<T *>(smem);            // P[buf][k][i]: S[i][k0 + k]
    T *rdiag = P + 2 * PANEL * kPanelLd;          // 1 / S[k][k]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t v0 = (int64_t(blockIdx.x) * WARPS + warp) * NV;

    // panel at column k0 of S into buffer b. Untransposed: thread i copies
    // row i, column after column (coalesced); transposed: adjacent threads a
    // row's columns. Rows of 32-row groups that the panel's steps do not read
    // are skipped.
    auto load_panel = [&](int k0, int b) {
        T *dst = P + b * PANEL * kPanelLd;
        const int g = k0 / 32 * 32;
        if (!s_trans) {
            const int i = tid;
            if (FORWARD ? i >= g : i < g + 32) {
                const T *src = A + i + int64_t(k0) * lda;
#pragma unroll
                for (int k = 0; k < PANEL; ++k, src += lda) {
                    const bool in = i < bs && k0 + k < bs && (FORWARD ? i > k0 + k : i < k0 + k);
                    copy_or_zero(dst + k * kPanelLd + i, in ? src : A, in);
                }
            }
        } else {
            const int k = tid % PANEL, col = k0 + k;
            const int i0 = (FORWARD ? g : 0) + tid / PANEL, i1 = FORWARD ? kBlock : g + 32;
            const T *src = A + col + int64_t(i0) * lda;
#pragma unroll 2
            for (int i = i0; i < i1; i += TH / PANEL, src += int64_t(TH / PANEL) * lda) {
                const bool in = i < bs && col < bs && (FORWARD ? i > col : i < col);
                copy_or_zero(dst + k * kPanelLd + i, in ? src : A, in);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const int first = FORWARD ? 0 : (bs - 1) / PANEL * PANEL;
    load_panel(first, first / PANEL & 1);
    for (int i = tid; i < kBlock; i += TH) {
        T r = Ar::one();
        if (!UNIT && i < bs) {
            T d = A[i + int64_t(i) * lda];
            if (s_conj) d = Ar::conj(d);
            r = quot(Ar::one(), d);
        }
        rdiag[i] = r;
    }
    // c[m]: minus the sum of S[i][k] x_k so far, until group m's turn; then
    // its right-hand sides are added in one rounding (a running subtraction
    // from them would round at their size at every step) and it is solved
    T c[kRows][NV], rhs[NV];
#pragma unroll
    for (int m = 0; m < kRows; ++m)
#pragma unroll
        for (int v = 0; v < NV; ++v) c[m][v] = Ar::zero();
    auto load_rhs = [&](int m) {
        const int i = lane + 32 * m;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            rhs[v] = Ar::zero();
            if (i < bs && v0 + v < nvec) rhs[v] = left ? C[i + (v0 + v) * ldc] : C[v0 + v + int64_t(i) * ldc];
        }
    };
    load_rhs(FORWARD ? 0 : (bs - 1) / 32);

#pragma unroll
    for (int mm = 0; mm < kRows; ++mm) {
        const int m = FORWARD ? mm : kRows - 1 - mm;  // compile-time after unrolling
        if (32 * m >= bs) continue;
#pragma unroll
        for (int v = 0; v < NV; ++v)  // (a row beyond bs stays zero whatever the scale: inf * 0 is not)
            if (lane + 32 * m < bs) c[m][v] = Ar::add(Ar::mul(scale, rhs[v]), c[m][v]);
        if (FORWARD ? 32 * (m + 1) < bs : m > 0) load_rhs(FORWARD ? m + 1 : m - 1);
#pragma unroll 1
        for (int h = 0; h < 32 / PANEL; ++h) {
            const int part = FORWARD ? h : 32 / PANEL - 1 - h, k0 = 32 * m + PANEL * part;
            if (k0 >= bs) continue;
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();  // the panel has landed, and every warp has left the other buffer
            const int next = FORWARD ? k0 + PANEL : k0 - PANEL;
            if (FORWARD ? next < bs : next >= 0) load_panel(next, next / PANEL & 1);
            const T *panel = P + (k0 / PANEL & 1) * PANEL * kPanelLd + lane;
#pragma unroll 4
            for (int q = 0; q < PANEL; ++q) {
                const int kq = FORWARD ? q : PANEL - 1 - q;
                const int kk = PANEL * part + kq;  // the lane owning row k
                const T *col = panel + kq * kPanelLd;
                T x[NV];
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    const T s = UNIT ? c[m][v] : Ar::mul(c[m][v], rdiag[k0 + kq]);
                    x[v] = shfl(s, kk);
                }
                const bool after = FORWARD ? lane > kk : lane < kk;
                {
                    T s = col[32 * m];
                    if (s_conj) s = Ar::conj(s);
                    s = negate(s);
#pragma unroll
                    for (int v = 0; v < NV; ++v)
                        if (after) c[m][v] = Ar::fma(s, x[v], c[m][v]);
                }
#pragma unroll
                for (int r = 0; r < kRows; ++r) {
                    if (FORWARD ? r <= m : r >= m) continue;
                    T s = col[32 * r];
                    if (s_conj) s = Ar::conj(s);
                    s = negate(s);
#pragma unroll
                    for (int v = 0; v < NV; ++v) c[r][v] = Ar::fma(s, x[v], c[r][v]);
                }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < kRows; ++m)
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int i = lane + 32 * m;
            if (i < bs && v0 + v < nvec) {
                // x_i: the same product that went to the other lanes at step i
                if (!UNIT) c[m][v] = Ar::mul(c[m][v], rdiag[i]);
                if (left) C[i + (v0 + v) * ldc] = c[m][v];
                else C[v0 + v + int64_t(i) * ldc] = c[m][v];
            }
        }
}

template <typename T, bool FORWARD, bool UNIT, int PANEL = kPanel>
int launch_block_k(const Trsm &t, int64_t lo, int64_t hi, cplx scale, int s_trans, cudaStream_t s) {
    constexpr size_t smem = sizeof(T) * (2 * PANEL * kPanelLd + kBlock);
    static const cudaError_t attr = cudaFuncSetAttribute(
        trsm_block_kernel<T, FORWARD, UNIT, PANEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    BX_CUDA(attr);
    const int64_t nvec = t.left ? t.N : t.M;
    const T *A = static_cast<const T *>(t.A) + lo + lo * t.lda;
    T *C = static_cast<T *>(t.B) + (t.left ? lo : lo * t.ldb);
    constexpr int per = kBlockThreads / 32 * Vecs<T>::n;
    const int64_t blocks = (nvec + per - 1) / per;
    if (blocks > 0x7fffffff) return set_error(BLASX_ERR_UNSUPPORTED, "trsm: too many right-hand sides");
    if constexpr (sizeof(T) == 16 && PANEL == kPanel) {
        if (blocks > kSms) return launch_block_k<T, FORWARD, UNIT, kSmallPanel>(t, lo, hi, scale, s_trans, s);
    }
    const bool conj = is_complex(t.dt) && t.trans == ConjT;
    trsm_block_kernel<T, FORWARD, UNIT, PANEL><<<unsigned(blocks), kBlockThreads, smem, s>>>(
        A, t.lda, C, t.ldb, int(hi - lo), nvec, t.left, s_trans, conj, from_cplx<T>(scale));
    BX_CUDA(cudaGetLastError());
    count_launch();
    return BLASX_OK;
}

template <typename T>
int launch_block_t(const Trsm &t, int64_t lo, int64_t hi, cplx scale, int s_trans, int forward, cudaStream_t s) {
    if (forward)
        return t.unit ? launch_block_k<T, true, true>(t, lo, hi, scale, s_trans, s)
                      : launch_block_k<T, true, false>(t, lo, hi, scale, s_trans, s);
    return t.unit ? launch_block_k<T, false, true>(t, lo, hi, scale, s_trans, s)
                  : launch_block_k<T, false, false>(t, lo, hi, scale, s_trans, s);
}

int launch_block(const Trsm &t, int64_t lo, int64_t hi, cplx scale, int s_trans, int forward, cudaStream_t s) {
    switch (t.dt) {
        case DType::F32: return launch_block_t<float>(t, lo, hi, scale, s_trans, forward, s);
        case DType::F64: return launch_block_t<double>(t, lo, hi, scale, s_trans, forward, s);
        case DType::C64: return launch_block_t<c2>(t, lo, hi, scale, s_trans, forward, s);
        default: return launch_block_t<z2>(t, lo, hi, scale, s_trans, forward, s);
    }
}

struct Range {
    int64_t lo, hi;
    int64_t size() const { return hi - lo; }
};

// The system matrix S of the blocks (see trsm_block_kernel) is A or A^T:
// s_trans = 1 when S = A^T. Substitution runs forward when S is lower.
int s_trans_of(const Trsm &t) { return t.left ? t.trans != NoTrans : t.trans == NoTrans; }
bool forward_of(const Trsm &t) { return t.lower != bool(s_trans_of(t)); }

// The two halves of [lo, hi) in solve order: the first has a multiple of
// kBlock rows.
void split(const Trsm &t, Range r, Range *first, Range *second) {
    const int64_t n = r.size();
    const int64_t half = std::min(n - 1, (n / 2 + kBlock - 1) / kBlock * kBlock);
    if (forward_of(t)) {
        *first = {r.lo, r.lo + half};
        *second = {r.lo + half, r.hi};
    } else {
        *first = {r.hi - half, r.hi};
        *second = {r.lo, r.hi - half};
    }
}

// B[tgt] = beta B[tgt] + alpha op(A)[tgt, src] B[src] (left) or
// B[:, tgt] = beta B[:, tgt] + alpha B[:, src] op(A)[src, tgt] (right).
Gemm update_gemm(const Trsm &t, Range tgt, Range src, cplx alpha, cplx beta) {
    const size_t es = elem_size(t.dt);
    const char *A = static_cast<const char *>(t.A);
    char *B = static_cast<char *>(t.B);
    const int tr = (t.trans == ConjT && !is_complex(t.dt)) ? TransT : t.trans;
    Gemm g;
    g.dt = t.dt;
    g.alpha = alpha;
    g.beta = beta;
    g.K = src.size();
    g.resident = t.resident;
    if (t.left) {
        g.M = tgt.size();
        g.N = t.N;
        g.ta = tr;
        g.A = tr == NoTrans ? A + (tgt.lo + src.lo * t.lda) * es : A + (src.lo + tgt.lo * t.lda) * es;
        g.lda = t.lda;
        g.tb = NoTrans;
        g.B = B + src.lo * es;
        g.ldb = t.ldb;
        g.C = B + tgt.lo * es;
    } else {
        g.M = t.M;
        g.N = tgt.size();
        g.ta = NoTrans;
        g.A = B + src.lo * t.ldb * es;
        g.lda = t.ldb;
        g.tb = tr;
        g.B = tr == NoTrans ? A + (src.lo + tgt.lo * t.lda) * es : A + (tgt.lo + src.lo * t.lda) * es;
        g.ldb = t.lda;
        g.C = B + tgt.lo * t.ldb * es;
    }
    g.ldc = t.ldb;
    return g;
}

constexpr cplx kMinusOne{-1.0, 0.0}, kOne{1.0, 0.0};

int solve(const Trsm &t, Range r, cplx scale, cudaStream_t s, bool *emulated) {
    if (r.size() <= kBlock) return launch_block(t, r.lo, r.hi, scale, s_trans_of(t), forward_of(t), s);
    Range first, second;
    split(t, r, &first, &second);
    BX_TRY(solve(t, first, scale, s, emulated));
    BX_TRY(device_gemm(update_gemm(t, second, first, kMinusOne, scale), s));
    if (call_stats().path == 2) *emulated = true;
    return solve(t, second, cplx{1.0, 0.0}, s, emulated);
}

// ---- TRMM: B = alpha op(A) B or alpha B op(A), in place -------------------
// With the vectors of B (columns for a left multiply, rows for a right one)
// the product is v <- alpha S v, S = op(A) or op(A)^T as for the solve. It
// recurses over halves P (earlier rows of S) and Q: for S lower,
// v_Q <- alpha S_QQ v_Q + alpha S_QP v_P needs the original v_P, so Q goes
// first (its multiply, then one GEMM update from P), then P; for S upper,
// P goes first. Every GEMM reads op(A) in an off-diagonal rectangle inside
// the stored triangle. A leaf of at most kTrmmLeaf rows multiplies by its
// diagonal block, completed (zeros, unit diagonal) in a scratch copy, on
// the native kernels: the emulated path never sees a triangle's tip, whose
// single nonzero per row would lose accuracy under per-row scaling.
constexpr int kTrmmLeaf = 256;

void trmm_split(const Trsm &t, Range r, Range *first, Range *second) {
    const int64_t n = r.size();
    const int64_t half = std::min(n - 1, (n / 2 + kTrmmLeaf - 1) / kTrmmLeaf * kTrmmLeaf);
    const Range lo{r.lo, r.lo + half}, hi{r.lo + half, r.hi};
    *first = forward_of(t) ? hi : lo;
    *second = forward_of(t) ? lo : hi;
}

int trmm_leaf(const Trsm &t, Range r, const TrmmScratch &w, cudaStream_t s) {
    const size_t es = elem_size(t.dt);
    const int64_t bs = r.size();
    const char *A = static_cast<const char *>(t.A);
    char *B = static_cast<char *>(t.B);
    BX_CUDA(cudaMemcpy2DAsync(w.diag, size_t(kTrmmLeaf) * es, A + (r.lo + r.lo * t.lda) * es, size_t(t.lda) * es,
                              size_t(bs) * es, size_t(bs), cudaMemcpyDeviceToDevice, s));
    const int form = t.lower ? (t.unit ? kTriLowerUnit : kTriLower) : (t.unit ? kTriUpperUnit : kTriUpper);
    BX_TRY(launch_complete_operand(t.dt, form, w.diag, kTrmmLeaf, bs, s));
    const int tr = (t.trans == ConjT && !is_complex(t.dt)) ? TransT : t.trans;
    Gemm g;
    g.dt = t.dt;
    g.alpha = t.alpha;
    g.beta = cplx{0.0, 0.0};
    g.K = bs;
    if (t.left) {  // rows r of B: B_r = alpha op(A_rr) B_r
        BX_CUDA(cudaMemcpy2DAsync(w.temp, size_t(w.ldt) * es, B + r.lo * es, size_t(t.ldb) * es, size_t(bs) * es,
                                  size_t(t.N), cudaMemcpyDeviceToDevice, s));
        g.M = bs; g.N = t.N;
        g.ta = tr; g.A = w.diag; g.lda = kTrmmLeaf;
        g.tb = NoTrans; g.B = w.temp; g.ldb = w.ldt;
        g.C = B + r.lo * es;
    } else {  // columns r of B: B_r = alpha B_r op(A_rr)
        BX_CUDA(cudaMemcpy2DAsync(w.temp, size_t(w.ldt) * es, B + r.lo * t.ldb * es, size_t(t.ldb) * es,
                                  size_t(t.M) * es, size_t(bs), cudaMemcpyDeviceToDevice, s));
        g.M = t.M; g.N = bs;
        g.ta = NoTrans; g.A = w.temp; g.lda = w.ldt;
        g.tb = tr; g.B = w.diag; g.ldb = kTrmmLeaf;
        g.C = B + r.lo * t.ldb * es;
    }
    g.ldc = t.ldb;
    return dmma_supported(g) ? launch_gemm_dmma(g, s) : launch_gemm_simt(g, s);
}

int multiply(const Trsm &t, Range r, const TrmmScratch &w, cudaStream_t s, bool *emulated) {
    if (r.size() <= kTrmmLeaf) return trmm_leaf(t, r, w, s);
    Range first, second;
    trmm_split(t, r, &first, &second);
    BX_TRY(multiply(t, first, w, s, emulated));
    BX_TRY(device_gemm(update_gemm(t, first, second, t.alpha, kOne), s));
    if (call_stats().path == 2) *emulated = true;
    return multiply(t, second, w, s, emulated);
}

// The same product out of place: part r of dst (B's layout) = alpha S_rr
// B_r, B unchanged. A leaf multiplies B's rows (or columns) by the completed
// diagonal block straight into dst, with no staging copy; every update
// reads B's original values, so the halves may go in either order.
int leaf_into(const Trsm &t, void *dst, Range r, const TrmmScratch &w, cudaStream_t s) {
    const size_t es = elem_size(t.dt);
    const int64_t bs = r.size();
    const char *A = static_cast<const char *>(t.A);
    const char *B = static_cast<const char *>(t.B);
    char *D = static_cast<char *>(dst);
    BX_CUDA(cudaMemcpy2DAsync(w.diag, size_t(kTrmmLeaf) * es, A + (r.lo + r.lo * t.lda) * es, size_t(t.lda) * es,
                              size_t(bs) * es, size_t(bs), cudaMemcpyDeviceToDevice, s));
    const int form = t.lower ? (t.unit ? kTriLowerUnit : kTriLower) : (t.unit ? kTriUpperUnit : kTriUpper);
    BX_TRY(launch_complete_operand(t.dt, form, w.diag, kTrmmLeaf, bs, s));
    const int tr = (t.trans == ConjT && !is_complex(t.dt)) ? TransT : t.trans;
    Gemm g;
    g.dt = t.dt;
    g.alpha = t.alpha;
    g.beta = cplx{0.0, 0.0};
    g.K = bs;
    if (t.left) {  // rows r: D_r = alpha op(A_rr) B_r
        g.M = bs; g.N = t.N;
        g.ta = tr; g.A = w.diag; g.lda = kTrmmLeaf;
        g.tb = NoTrans; g.B = B + r.lo * es; g.ldb = t.ldb;
        g.C = D + r.lo * es;
    } else {  // columns r: D_r = alpha B_r op(A_rr)
        g.M = t.M; g.N = bs;
        g.ta = NoTrans; g.A = B + r.lo * t.ldb * es; g.lda = t.ldb;
        g.tb = tr; g.B = w.diag; g.ldb = kTrmmLeaf;
        g.C = D + r.lo * t.ldb * es;
    }
    g.ldc = t.ldb;
    return dmma_supported(g) ? launch_gemm_dmma(g, s) : launch_gemm_simt(g, s);
}

int multiply_into(const Trsm &t, void *dst, Range r, const TrmmScratch &w, cudaStream_t s, bool *emulated) {
    if (r.size() <= kTrmmLeaf) return leaf_into(t, dst, r, w, s);
    Range first, second;
    trmm_split(t, r, &first, &second);
    BX_TRY(multiply_into(t, dst, first, w, s, emulated));
    Gemm g = update_gemm(t, first, second, t.alpha, kOne);
    g.C = static_cast<char *>(dst) + (static_cast<char *>(g.C) - static_cast<char *>(t.B));
    BX_TRY(device_gemm(g, s));
    if (call_stats().path == 2) *emulated = true;
    return multiply_into(t, dst, second, w, s, emulated);
}

}  // namespace

bool tri_forward(const Trsm &t) { return forward_of(t); }

Gemm tri_update_gemm(const Trsm &t, int64_t tgt_lo, int64_t tgt_hi, int64_t src_lo, int64_t src_hi) {
    return update_gemm(t, Range{tgt_lo, tgt_hi}, Range{src_lo, src_hi}, t.alpha, kOne);
}

int trsm_solve_part(const Trsm &t, int64_t lo, int64_t hi, cplx scale, cudaStream_t s, bool *emulated) {
    return solve(t, Range{lo, hi}, scale, s, emulated);
}

int trsm_update_part(const Trsm &t, int64_t tgt_lo, int64_t tgt_hi, int64_t src_lo, int64_t src_hi, cplx scale,
                     cudaStream_t s, bool *emulated) {
    BX_TRY(device_gemm(update_gemm(t, Range{tgt_lo, tgt_hi}, Range{src_lo, src_hi}, kMinusOne, scale), s));
    if (call_stats().path == 2) *emulated = true;
    return BLASX_OK;
}

Gemm trsm_top_update(const Trsm &t) {
    const Range all{0, t.order()};
    if (all.size() <= kBlock) {
        Gemm g = update_gemm(t, all, all, kMinusOne, t.alpha);
        g.K = 0;
        return g;
    }
    Range first, second;
    split(t, all, &first, &second);
    return update_gemm(t, second, first, kMinusOne, t.alpha);
}

int trsm_device(const Trsm &t, cudaStream_t s, bool *emulated) {
    *emulated = false;
    if (t.M == 0 || t.N == 0) return BLASX_OK;
    if (t.alpha.re == 0 && t.alpha.im == 0) {  // X = 0; A is not read
        Gemm z;
        z.dt = t.dt;
        z.ta = z.tb = NoTrans;
        z.M = t.M; z.N = t.N; z.K = 0;
        z.alpha = cplx{0.0, 0.0}; z.beta = cplx{0.0, 0.0};
        z.A = nullptr; z.lda = 1; z.B = nullptr; z.ldb = 1;
        z.C = t.B; z.ldc = t.ldb;
        return launch_scale(z, s);
    }
    return solve(t, Range{0, t.order()}, t.alpha, s, emulated);
}

}  // namespace bx

namespace bx {

TrmmScratch trmm_scratch_sizes(const Trsm &t) {
    TrmmScratch w;
    const size_t es = elem_size(t.dt);
    w.ldt = t.left ? kTrmmLeaf : (t.M + 31) / 32 * 32;
    w.diag_bytes = size_t(kTrmmLeaf) * kTrmmLeaf * es;
    w.temp_bytes = size_t(w.ldt) * size_t(t.left ? t.N : kTrmmLeaf) * es;
    return w;
}

int trmm_part_into(const Trsm &t, void *dst, int64_t lo, int64_t hi, const TrmmScratch &w, cudaStream_t s,
                   bool *emulated) {
    return multiply_into(t, dst, Range{lo, hi}, w, s, emulated);
}

int trmm_update_into(const Trsm &t, void *dst, int64_t tgt_lo, int64_t tgt_hi, int64_t src_lo, int64_t src_hi,
                     cudaStream_t s, bool *emulated) {
    Gemm g = update_gemm(t, Range{tgt_lo, tgt_hi}, Range{src_lo, src_hi}, t.alpha, kOne);
    g.C = static_cast<char *>(dst) + (static_cast<char *>(g.C) - static_cast<char *>(t.B));
    BX_TRY(device_gemm(g, s));
    if (call_stats().path == 2) *emulated = true;
    return BLASX_OK;
}

Gemm trmm_top_update(const Trsm &t) {
    const Range all{0, t.order()};
    if (all.size() <= kTrmmLeaf) {
        Gemm g = update_gemm(t, all, all, t.alpha, kOne);
        g.K = 0;
        return g;
    }
    Range first, second;
    trmm_split(t, all, &first, &second);
    return update_gemm(t, first, second, t.alpha, kOne);
}

int trmm_device(const Trsm &t, const TrmmScratch &w, cudaStream_t s, bool *emulated) {
    *emulated = false;
    if (t.M == 0 || t.N == 0) return BLASX_OK;
    if (t.alpha.re == 0 && t.alpha.im == 0) {  // B = 0; A is not read
        Gemm z;
        z.dt = t.dt;
        z.ta = z.tb = NoTrans;
        z.M = t.M; z.N = t.N; z.K = 0;
        z.alpha = cplx{0.0, 0.0}; z.beta = cplx{0.0, 0.0};
        z.A = nullptr; z.lda = 1; z.B = nullptr; z.ldb = 1;
        z.C = t.B; z.ldc = t.ldb;
        return launch_scale(z, s);
    }
    return multiply(t, Range{0, t.order()}, w, s, emulated);
}

}  // namespace bx
