// dispatch.cu -- picks the device kernel path for a device-resident GEMM.
//
// Precision mode (blasx_set_dgemm_mode / BLASX_DGEMM_MODE):
//   native  -- FP64 / complex128 on the DMMA kernel, FP32 on the SIMT kernel;
//   auto    -- the INT8 Ozaki path where it measured faster than native
//              (ozaki_selected), K within its exact range; it still falls
//              back to native on the device when the measured spread of the
//              operands needs more than 20 moduli;
//   ozaki   -- the Ozaki path whenever K is within its exact range.
#include <algorithm>

#include "kernels.h"
#include "ozaki.h"
#include "profile.h"

namespace bx {

namespace {
// Whether auto mode emulates g, from `f64` (`c128`) multiply-adds on.
bool auto_emulates(const Gemm &g, double f64, double c128) {
    if (std::min(g.M, g.N) < 256) return false;
    const double work = double(g.M) * double(g.N) * double(g.K);
    switch (g.dt) {
        case DType::F64: return g.K >= 512 && work >= f64;
        case DType::F32: return g.K >= 256 && work >= 3e8;
        case DType::C64: return g.K >= 256 && work >= 1.5e8;
        default: return g.K >= 256 && work >= c128;
    }
}
bool exact_k(const Gemm &g) { return g.K <= (is_complex(g.dt) ? oz::kMaxK / 2 : oz::kMaxK); }
}  // namespace

// Device-resident calls emulate from 2e9 (FP64) and 7e8 (complex128)
// multiply-adds. Measured, native / emulated: FP64 1024^3 91 / 82 us, 1280^3
// 162 / 109, 1024 x 2048 x 1024 171 / 109, 1792^3 433 / 184; complex128 768^3
// 138 / 116, 900^3 231 / 157, 1024^3 304 / 161. Below the line the gain is
// smaller than what operands of wide spread pay for finding out (35 us). A
// triangular output halves the native work and not all of the emulation's:
// its line lies at twice that.
// Calls that plan their memory under an HBM budget keep the lines from which
// their scratch has always been planned, 6e9 and 2e9.
bool ozaki_selected(const Gemm &g, int mode) {
    if (!exact_k(g) || mode == 1) return false;
    if (mode == 2) return true;
    const double half = g.uplo ? 2.0 : 1.0;
    return g.resident ? auto_emulates(g, 2e9 * half, 7e8 * half) : auto_emulates(g, 6e9, 2e9);
}

int device_gemm(const Gemm &g, cudaStream_t s) {
    if (g.M == 0 || g.N == 0) return BLASX_OK;
    if (g.alpha_zero() || g.K == 0) return launch_scale(g, s);
    const int mode = config().dgemm_mode.load();
    if (ozaki_selected(g, mode)) {
        // between the two lines the native kernels serve a call whose scratch
        // does not fit
        const bool optional = mode == 0 && !auto_emulates(g, 6e9, 2e9);
        const int st = ozaki_gemm(g, s, mode, optional);
        if (st != kNoScratch) return st;
    }
    call_stats().path = 1;
    call_stats().moduli = 0;
    cudaEvent_t e0 = prof::mark(s);
    const int st = dmma_supported(g) ? launch_gemm_dmma(g, s) : launch_gemm_simt(g, s);
    prof::span(prof::kNative, e0, prof::mark(s));
    return st;
}

}  // namespace bx
