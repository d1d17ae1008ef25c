// ozaki.cu -- scaling, slicing, modulus-count decision and CRT reconstruction
// of the emulated GEMM (see ozaki.h for the method), and its driver.
//
// Pipeline on one stream, with no host synchronisation:
//   stats + decide      -> per-row max|x| and sum x^2 of both operands; modulus
//                          count N (0 = native) and norm bound Q
//   slice(A), slice(B)  -> row exponents, int8 residues for l < N
//   residue GEMM        -> uint8 residues of every product (tcgen05)
//   reconstruct         -> exact CRT, unscale, alpha/beta epilogue
//   native guard        -> the native kernel runs only when N == 0
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "kernels.h"
#include "ozaki.h"
#include "ozaki_dev.cuh"
#include "ozaki_stats.cuh"
#include "profile.h"

namespace bx {
namespace oz {

const int kModuli[kMaxModuli] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227,
                                 223, 217, 211, 199, 197, 193, 191, 181, 179, 173};

namespace {

// ---- the standalone kernels: one body block per CUDA block -------------------

// The pair sample's blocks come first: a row of the grid of an operand's own
// launch (its chunks are at most the blocks along k).
template <typename T, int ROLE>
__global__ void __launch_bounds__(256, ROLE == 0 ? 4 : (ROLE == 1 ? 3 : 2)) slice_kc_kernel(View v, RowStats st, const Decision *dec, int *expo,
                                                       SliceOut o, const __grid_constant__ PairVeto pv) {
    __shared__ __align__(16) __nv_bfloat16 smem[kPairShared];
    const int row0 = pv.p.chunks ? 1 : 0;
    if (blockIdx.y < row0) {
        if (int(blockIdx.x) < pv.p.chunks) pair_veto_block<T>(pv, blockIdx.x, threadIdx.x, smem);
        return;
    }
    slice_kc_body<T, ROLE>(v, st, dec, expo, o, blockIdx.x, blockIdx.y - row0, threadIdx.x);
}

template <typename T, int ROLE>
__global__ void __launch_bounds__(256, ROLE == 0 ? 4 : (ROLE == 1 ? 3 : 2)) slice_rc_kernel(View v, RowStats st, const Decision *dec, int *expo,
                                                       SliceOut o, const __grid_constant__ PairVeto pv) {
    __shared__ __align__(16) unsigned char smem[slice_rc_smem_bytes<ROLE>()];
    static_assert(sizeof smem >= kPairShared * sizeof(__nv_bfloat16), "the pair sample's stage");
    const int row0 = pv.p.chunks ? 1 : 0;
    if (blockIdx.y < row0) {
        if (int(blockIdx.x) < pv.p.chunks) pair_veto_block<T>(pv, blockIdx.x, threadIdx.x, smem);
        return;
    }
    slice_rc_body<T, ROLE>(v, st, dec, expo, o, blockIdx.x, blockIdx.y - row0, threadIdx.x, smem);
}

// Both operands of a real GEMM: after the pair sample's, blocks [0, na) slice
// op(A), the others op(B).
struct SliceSide {
    View v;
    RowStats st;
    int *expo;
    SliceOut o;
    int gx;  // blocks along k
};
template <typename T, bool AKC, bool BKC>
__global__ void __launch_bounds__(256, 4) slice_both_kernel(SliceSide a, SliceSide b, int na, const Decision *dec,
                                                            const __grid_constant__ PairVeto pv) {
    __shared__ __align__(16) unsigned char smem[(AKC && BKC) ? kPairShared * sizeof(__nv_bfloat16) : slice_rc_smem_bytes<0>()];
    const int i = int(blockIdx.x) - pv.p.chunks;
    if (i < 0) {
        pair_veto_block<T>(pv, blockIdx.x, threadIdx.x, smem);
    } else if (i < na) {
        if (AKC) slice_kc_body<T, 0>(a.v, a.st, dec, a.expo, a.o, i % a.gx, i / a.gx, threadIdx.x);
        else slice_rc_body<T, 0>(a.v, a.st, dec, a.expo, a.o, i % a.gx, i / a.gx, threadIdx.x, smem);
    } else {
        const int j = i - na;
        if (BKC) slice_kc_body<T, 0>(b.v, b.st, dec, b.expo, b.o, j % b.gx, j / b.gx, threadIdx.x);
        else slice_rc_body<T, 0>(b.v, b.st, dec, b.expo, b.o, j % b.gx, j / b.gx, threadIdx.x, smem);
    }
}

// Where the call's decision and error word go in pinned host memory (null:
// nowhere). One thread stores them there: as two copies behind the call's last
// kernel they took 12 us of every call (FP64 2048^3: 243 -> 231 us).
struct Report {
    Decision *dec;
    int *err;
    const int *device_err;
};

// Ten blocks per SM (48 registers): the gathers of residues wait on memory,
// and two more blocks than 64 registers allow cover it (complex128 2401 x 1639
// x 1203: 446 -> 435 us a call, FP32 3001 x 1777 x 999: 143 -> 137; 8192^3 the
// same).
template <typename T, bool CPLX>
__global__ void __launch_bounds__(128, 10) reconstruct_kernel(const ReconArgs a, const Decision *dec,
                                                              const Report rep) {
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        if (rep.dec) *rep.dec = *dec;
        if (rep.err) *rep.err = *rep.device_err;
    }
    __shared__ __align__(16) double sh[4 * kReconShared<CPLX>];
    reconstruct_body<T, CPLX>(a, dec, blockIdx.x, blockIdx.y, threadIdx.x, sh);
}

std::once_flag g_tables_once;
int g_tables_status = BLASX_OK;

}  // namespace

int upload_crt_tables() {
    std::call_once(g_tables_once, [] {
        if (upload_tables() != cudaSuccess) g_tables_status = BLASX_ERR_CUDA;
    });
    if (g_tables_status != BLASX_OK) return set_error(g_tables_status, "CRT table upload failed");
    return BLASX_OK;
}

int prepare_crt_tables_current_device() {
    BX_CUDA(upload_tables());
    return BLASX_OK;
}

}  // namespace oz

// --------------------------------------------------------------------------
// driver
// --------------------------------------------------------------------------

namespace {

// Statistics of both operands and the decision. The arrival counters (the
// row-flag arrays and Decision::pad) are zero on entry. The whole
// call fell from 342 to 265 us at FP64 2048^3, from 643 to 525 us for a
// complex128 product of 2401 x 1639 x 1203 and from 173 to 154 us for an
// FP32 one of 3001 x 1777 x 999 against per-operand kernels with atomics and
// a one-block decision.
template <typename T>
int launch_stats(const oz::View &va, bool akc, const oz::RowStats &sa, const oz::View &vb, bool bkc,
                 const oz::RowStats &sb, bool alias, const oz::Parts &pt, double unit, int mode, cudaStream_t s) {
    oz::StatsArgs a;
    a.s[0] = oz::stats_side(va, sa, akc, pt.Y);
    a.s[1] = alias ? a.s[0] : oz::stats_side(vb, sb, bkc, pt.X);
    a.sides = alias ? 1 : 2;
    a.total_groups = a.s[0].groups + (alias ? 0 : a.s[1].groups);
    a.arrive = &pt.dec->pad;
    a.K = va.K;
    a.unit = unit;
    a.mode = mode;
    a.forced = oz::forced_moduli();
    a.dec = pt.dec;
    const int64_t blocks = int64_t(a.s[0].groups) * a.s[0].chunks +
                           (alias ? 0 : int64_t(a.s[1].groups) * a.s[1].chunks);
    oz::stats_decide_kernel<T><<<unsigned(blocks), oz::kStatsThreads, 0, s>>>(a);
    BX_CUDA(cudaGetLastError());
    count_launch();
    return BLASX_OK;
}

template <typename T, int ROLE>
int launch_slice(const oz::View &v, bool kc, const oz::RowStats &st, const oz::Decision *dec,
                 int *expo, const oz::SliceOut &o, int64_t Kc, const oz::PairVeto &pv, cudaStream_t s) {
    const unsigned rows = unsigned(o.Rp / 64) + (pv.p.chunks ? 1 : 0);
    if (kc) {
        dim3 grid(unsigned(Kc / 64), rows);
        oz::slice_kc_kernel<T, ROLE><<<grid, 256, 0, s>>>(v, st, dec, expo, o, pv);
    } else {
        const int kt = ROLE ? 32 : 64;
        dim3 grid(unsigned(Kc / kt), rows);
        oz::slice_rc_kernel<T, ROLE><<<grid, 256, 0, s>>>(v, st, dec, expo, o, pv);
    }
    BX_CUDA(cudaGetLastError());
    count_launch();
    return BLASX_OK;
}

// Both operands of a real GEMM in one launch (one tail instead of two: at
// 2048^3 an operand alone is 1.7 waves of blocks). False when the grid would
// be too large.
template <typename T>
bool slice_both_fits(const oz::SliceOut &oa, const oz::SliceOut &ob, int64_t Kc) {
    return (Kc / 64) * (oa.Rp / 64 + ob.Rp / 64 + 1) <= INT32_MAX;
}
template <typename T>
int launch_slice_both(const oz::View &va, bool akc, const oz::RowStats &sa, int *ea, const oz::SliceOut &oa,
                      const oz::View &vb, bool bkc, const oz::RowStats &sb, int *fb, const oz::SliceOut &ob,
                      const oz::Decision *dec, int64_t Kc, const oz::PairVeto &pv, cudaStream_t s) {
    const int gx = int(Kc / 64), na = int(gx * (oa.Rp / 64)), nb = int(gx * (ob.Rp / 64));
    const oz::SliceSide a{va, sa, ea, oa, gx}, b{vb, sb, fb, ob, gx};
    const unsigned grid = unsigned(pv.p.chunks) + unsigned(na) + unsigned(nb);
    if (akc) {
        if (bkc) oz::slice_both_kernel<T, true, true><<<grid, 256, 0, s>>>(a, b, na, dec, pv);
        else oz::slice_both_kernel<T, true, false><<<grid, 256, 0, s>>>(a, b, na, dec, pv);
    } else {
        if (bkc) oz::slice_both_kernel<T, false, true><<<grid, 256, 0, s>>>(a, b, na, dec, pv);
        else oz::slice_both_kernel<T, false, false><<<grid, 256, 0, s>>>(a, b, na, dec, pv);
    }
    BX_CUDA(cudaGetLastError());
    count_launch();
    return BLASX_OK;
}

// The whole emulated pipeline on a caller-provided workspace of
// make_plan(g).bytes bytes: no allocation. The device decision and error
// flag are written to the given host slots (pinned, mapped memory) when they
// are not null.
template <typename T>
int ozaki_run(const Gemm &g, cudaStream_t s, int mode, void *ws, int num_sms, void *dec_host,
              int *err_host, const PanelHooks *hooks = nullptr, bool clear_err = true) {
    constexpr bool CPLX = oz::Elem<T>::cplx;
    const oz::Plan pl = oz::make_plan(g);
    const int64_t M = pl.M, N = pl.N, K = pl.K, Kh = pl.Kh, Kp = pl.Kp, Kc = pl.Kc;
    const int64_t Ip = pl.Ip, Jp = pl.Jp, Jx = pl.Jx;
    const oz::Parts pt = oz::carve_parts(g, pl, ws);
    int *err = pt.err;
    oz::Decision *dec = pt.dec;
    const oz::RowStats sa = pt.sa, sb = pt.sb;
    int *ea = pt.ea, *fb = pt.fb;
    int8_t *Y = pt.Y, *X = pt.X;
    uint8_t *U = pt.U;
    cudaEvent_t ev0 = prof::mark(s);
    // the error word (unless a sequence of steps keeps it), the decision and
    // the arrival counters of the statistics
    char *zero = reinterpret_cast<char *>(clear_err ? static_cast<void *>(err) : static_cast<void *>(dec));
    BX_CUDA(cudaMemsetAsync(zero, 0, size_t(reinterpret_cast<char *>(sa.amax) - zero), s));

    // op(A) rows i over k; op(B) columns j over k
    oz::View va{g.A, g.lda, M, K, g.ta == ConjT};
    oz::View vb{g.B, g.ldb, N, K, g.tb == ConjT};
    const bool akc = g.ta != NoTrans, bkc = g.tb == NoTrans;
    int *fbd = pl.alias ? ea : fb;  // aliased: the columns of op(B) are the rows of op(A)
    const double unit = oz::Elem<T>::single ? std::ldexp(1.0, -24) : std::ldexp(1.0, -53);
    BX_TRY(launch_stats<T>(va, akc, sa, vb, bkc, sb, pl.alias, pt, unit, mode, s));

    oz::SliceOut oy{Y, Ip, Kp, Kh, Ip * Kp};
    oz::SliceOut ox{X, Jp, Kp, Kh, Jx * Kp};
    // auto mode: the pair sample, with the slices of the operand that has more
    // rows, which hide it best (complex64 3560 x 704 x 320: 133 us a call with
    // the other's, 128 so), unless its row of blocks would exceed the grid.
    // Its counters are the last
    // words of op(A)'s flags, padded to a multiple of 64: the arrival counters
    // of op(A)'s groups, one for eight rows, end before them.
    oz::PairVeto none{}, pv{};
    if (mode == 0 && oz::forced_moduli() == 0)
        pv = oz::pair_veto(va, akc, sa, vb, bkc, pl.alias ? sa : sb, g.uplo, g.diag, pt,
                           sb.flags - oz::kPairCounters, dec);
    bool pv_first = pl.alias || oy.Rp >= ox.Rp;
    if (!pl.alias && (pv_first ? oy : ox).Rp / 64 >= 65535) pv_first = !pv_first;
    if constexpr (CPLX) {
        BX_TRY((launch_slice<T, 1>(va, akc, sa, dec, ea, oy, Kc, pv_first ? pv : none, s)));
        BX_TRY((launch_slice<T, 2>(vb, bkc, sb, dec, fb, ox, Kc, pv_first ? none : pv, s)));
    } else {
        if (!pl.alias && slice_both_fits<T>(oy, ox, Kc)) {
            BX_TRY(launch_slice_both<T>(va, akc, sa, ea, oy, vb, bkc, sb, fb, ox, dec, Kc, pv, s));
        } else {
            BX_TRY((launch_slice<T, 0>(va, akc, sa, dec, ea, oy, Kc, pv_first ? pv : none, s)));
            if (!pl.alias) BX_TRY((launch_slice<T, 0>(vb, bkc, sb, dec, fb, ox, Kc, pv_first ? none : pv, s)));
        }
    }
    // residue GEMMs and reconstruction, in column panels of C when asked.
    // (Running a panel's reconstruction on a second stream beside the next
    // panel's residue GEMM was measured slower: under the power cap the
    // concurrent integer work lowers the clock of the tensor work.)
    // the residue GEMMs are done when a reconstruction runs: the error word is
    // final with the last of them
    const oz::Report report{static_cast<oz::Decision *>(dec_host), err_host, err};
    const int64_t tiles_j = Jp / oz::kTileJ;
    const int panels = (CPLX || !hooks) ? 1 : int(std::max<int64_t>(1, std::min<int64_t>(hooks->panels, tiles_j)));
    cudaEvent_t ev1 = prof::mark(s), ev2 = nullptr;
    for (int pnl = 0; pnl < panels; ++pnl) {
        const int64_t tj0 = tiles_j * pnl / panels, tj1 = tiles_j * (pnl + 1) / panels;
        const int64_t j0 = tj0 * oz::kTileJ, j1 = std::min<int64_t>(N, tj1 * oz::kTileJ);
        if (panels == 1) {
            BX_TRY(oz::launch_residue_gemm(X, Y, U, Jx, Ip, Kp, dec, err, num_sms, s, 0, -1, g.max_cta_tiles,
                                           g.uplo, g.diag, Jp));
        } else {
            BX_TRY(oz::launch_residue_gemm(X, Y, U, Jx, Ip, Kp, dec, err, num_sms, s, tj0, tj1 - tj0,
                                           g.max_cta_tiles, g.uplo, g.diag, Jp));
        }
        if (pnl == 0) ev2 = prof::mark(s);
        if (hooks && hooks->before_reconstruct && j1 > j0)
            BX_TRY(hooks->before_reconstruct(hooks->ctx, j0, j1));
        // grid.y is limited to 65535 columns per launch
        for (int64_t c0 = j0; c0 < j1; c0 += 65535) {
            const int64_t c1 = std::min<int64_t>(j1, c0 + 65535);
            dim3 rgrid(unsigned((M + 4 * 128 - 1) / (4 * 128)), unsigned(c1 - c0));
            oz::ReconArgs ra{U, Jp, Ip, M, N, ea, fbd, g.alpha.re, g.alpha.im, g.beta.re, g.beta.im,
                             g.beta_zero() ? 1 : 0, g.C, g.ldc, c0, g.uplo, g.diag};
            oz::reconstruct_kernel<T, CPLX><<<rgrid, 128, 0, s>>>(ra, dec, report);
            BX_CUDA(cudaGetLastError());
            count_launch();
        }
        if (hooks && j1 > j0) {
            // native fallback for this panel's columns (runs only when nmod == 0),
            // so that the panel's write-back also follows the fallback
            Gemm gp = g;
            gp.N = j1 - j0;
            gp.B = static_cast<const char *>(g.B) +
                   (g.tb == NoTrans ? j0 * g.ldb : j0) * int64_t(elem_size(g.dt));
            gp.C = static_cast<char *>(g.C) + j0 * g.ldc * int64_t(elem_size(g.dt));
            gp.diag = g.diag + j0;
            gp.guard = &dec->nmod;
            gp.queue = &dec->pad;
            if (dmma_supported(gp)) BX_TRY(launch_gemm_dmma(gp, s));
            else BX_TRY(launch_gemm_simt(gp, s));
        }
        if (hooks && hooks->after_panel) BX_TRY(hooks->after_panel(hooks->ctx, j0, j1));
    }
    cudaEvent_t ev3 = prof::mark(s);

    // native fallback, decided on the device (runs only when nmod == 0);
    // with panels it already ran panel by panel
    if (!hooks) {
        Gemm gn = g;
        gn.guard = &dec->nmod;
        gn.queue = &dec->pad;
        if (dmma_supported(gn)) BX_TRY(launch_gemm_dmma(gn, s));
        else BX_TRY(launch_gemm_simt(gn, s));
    }
    cudaEvent_t ev4 = prof::mark(s);
    prof::span(prof::kSlice, ev0, ev1);
    prof::span(prof::kResidueGemm, ev1, ev2);
    prof::span(prof::kReconstruct, ev2, ev3);
    prof::span(prof::kNative, ev3, ev4);

    call_stats().path = 2;
    call_stats().moduli = -1;  // decided on the device: resolved from dec_host once the stream has passed
    return BLASX_OK;
}

template <typename T> int ozaki_t(const Gemm &g, cudaStream_t s, int mode, bool optional) {
    Context *ctx = context();
    if (!ctx) return last_status();
    BX_TRY(oz::upload_crt_tables());
    const oz::Plan pl = oz::make_plan(g);
    void *ws = nullptr;
    const cudaError_t got = dev_malloc_async(&ws, pl.bytes, s);
    if (got == cudaErrorMemoryAllocation && optional) {
        cudaGetLastError();
        return kNoScratch;
    }
    BX_CUDA(got);
    struct Free {
        void *p;
        cudaStream_t s;
        ~Free() { cudaFreeAsync(p, s); }
    } free_ws{ws, s};
    return ozaki_run<T>(g, s, mode, ws, ctx->num_sms, ctx->last_decision, ctx->last_error_flag);
}

}  // namespace

int ozaki_gemm(const Gemm &g, cudaStream_t s, int mode, bool optional) {
    switch (g.dt) {
        case DType::F64: return ozaki_t<double>(g, s, mode, optional);
        case DType::F32: return ozaki_t<float>(g, s, mode, optional);
        case DType::C64: return ozaki_t<oz::cpair>(g, s, mode, optional);
        default: return ozaki_t<oz::zpair>(g, s, mode, optional);
    }
}

size_t ozaki_scratch_bytes(const Gemm &g) { return oz::make_plan(g).bytes; }

int ozaki_gemm_panels(const Gemm &g, cudaStream_t s, int mode, void *ws, int num_sms,
                      const PanelHooks &hooks, bool clear_err) {
    Context *ctx = context();
    if (!ctx) return last_status();
    BX_TRY(oz::upload_crt_tables());
    switch (g.dt) {
        case DType::F64:
            return ozaki_run<double>(g, s, mode, ws, num_sms, ctx->last_decision, ctx->last_error_flag, &hooks,
                                     clear_err);
        case DType::C64:
            return ozaki_run<oz::cpair>(g, s, mode, ws, num_sms, ctx->last_decision, ctx->last_error_flag, &hooks,
                                        clear_err);
        case DType::F32:
            return ozaki_run<float>(g, s, mode, ws, num_sms, ctx->last_decision, ctx->last_error_flag, &hooks,
                                    clear_err);
        default:
            return ozaki_run<oz::zpair>(g, s, mode, ws, num_sms, ctx->last_decision, ctx->last_error_flag,
                                        &hooks, clear_err);
    }
}

int ozaki_gemm_step(const Gemm &g, cudaStream_t s, int mode, void *ws, int num_sms, bool first,
                    bool last) {
    Context *ctx = context();
    if (!ctx) return last_status();
    BX_TRY(oz::upload_crt_tables());
    void *dec_host = last ? ctx->last_decision : nullptr;
    int *err_host = last ? ctx->last_error_flag : nullptr;
    switch (g.dt) {
        case DType::F64: return ozaki_run<double>(g, s, mode, ws, num_sms, dec_host, err_host, nullptr, first);
        case DType::F32: return ozaki_run<float>(g, s, mode, ws, num_sms, dec_host, err_host, nullptr, first);
        case DType::C64: return ozaki_run<oz::cpair>(g, s, mode, ws, num_sms, dec_host, err_host, nullptr, first);
        default: return ozaki_run<oz::zpair>(g, s, mode, ws, num_sms, dec_host, err_host, nullptr, first);
    }
}

int ozaki_gemm_in(const Gemm &g, cudaStream_t s, int mode, void *ws, int num_sms) {
    switch (g.dt) {
        case DType::F64: return ozaki_run<double>(g, s, mode, ws, num_sms, nullptr, nullptr);
        case DType::F32: return ozaki_run<float>(g, s, mode, ws, num_sms, nullptr, nullptr);
        case DType::C64: return ozaki_run<oz::cpair>(g, s, mode, ws, num_sms, nullptr, nullptr);
        default: return ozaki_run<oz::zpair>(g, s, mode, ws, num_sms, nullptr, nullptr);
    }
}

}  // namespace bx
