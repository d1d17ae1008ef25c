// kernels_sgemm.cu -- FP32 GEMM on the CUDA cores with the 128 x 128 tile of
// simt_tile.cuh, one CTA per C tile: large products whose operands cannot be
// copied 16 bytes at a time.
#include "kernels.h"
#include "simt_tile.cuh"

namespace bx {
namespace {

using namespace dev;

__global__ void __launch_bounds__(sg::THR, 2) sgemm128_kernel(const SimtParams<float> p, const int *guard) {
    if (guard && *guard != 0) return;  // the emulated path produced C
    __shared__ __align__(16) float smem[sgemm128_smem_bytes() / sizeof(float)];
    sgemm128_tile(p, blockIdx.x, blockIdx.y, smem);
}

constexpr int64_t kSms = 148;

// Not 16 bytes per copy in fma_tile.cuh.
bool narrow_copies(const void *p, int64_t ld) { return ld % 4 != 0 || reinterpret_cast<uintptr_t>(p) % 16 != 0; }

}  // namespace

// The FMA kernels copy such an operand 4 bytes at a time, four times the copies,
// which at 64x64 tiles take issue slots from the multiply-adds; this tile reads
// it through registers, each element for 128 outputs. Measured, FMA / this one,
// both operands narrow: 8000 x 8000 x 2000 NN 7.89 / 6.51 ms, NT 7.99 / 6.41;
// 4000 x 4000 x 1000 NN 1042 / 881 us; 2500 x 2500 x 600 NT 272 / 241; 3000 x
// 3000 x 256 NN 169 / 165; 2100 x 2150 NT x 250 95 / 86, x 200 81 / 73, x 160 66
// / 66, x 80 42 / 51; 4000 x 4000 x 100 155 / 165. One of them: 8000 x
// 8000 x 2000 6.78 to 7.33 / 6.5, 3000 x 3000 x 1000 507 to 546 / 494, 8000 x
// 4000 x 512 914 to 1006 / 950, 3000 x 3000 x 256 147 to 157 / 164. With 16-byte
// copies FMA is as fast or faster everywhere. Two of these CTAs share an SM and
// a tile is four 64x64 ones: the last round's idle SMs count against it (2400 x
// 2400 x 300, 361 tiles: 134 / 146; 4000 x 2000 x 700, 512: 390 / 360). These
// read C (beta 0.5), which costs this tile's epilogue more than FMA's; with beta
// = 0 its lines lie lower: both narrow 8000 x 4000 NT x 250 572 / 473 us, x 140
// 354 / 302, x 96 260 / 232, x 64 193 / 184; one, x 400 725 to 791 / 700, x 200
// 415 to 440 / 391, x 100 254 to 266 / 245, 4000 x 4000 x 64 90 to 96 / 98.
bool sgemm128_preferred(const Gemm &g) {
    using namespace dev::sg;
    if (g.dt != DType::F32 || g.M > INT32_MAX || g.N > INT32_MAX || g.K > INT32_MAX) return false;
    const int narrow = narrow_copies(g.A, g.lda) + narrow_copies(g.B, g.ldb);
    const bool reads_c = !g.beta_zero();
    if (narrow == 0 || g.K < (reads_c ? (narrow == 2 ? 192 : 640) : 96)) return false;
    const double area = narrow == 2 ? 1.19 : (reads_c ? 1.08 : 1.13);
    const int64_t tiles = ((g.M + TM - 1) / TM) * ((g.N + TN - 1) / TN);
    const int64_t small = ((g.M + 63) / 64) * ((g.N + 63) / 64);
    const int64_t rounds = (tiles + kSms - 1) / kSms;  // tiles of the busiest SM
    return (g.N + TN - 1) / TN <= 65535 && double(rounds * kSms * 4) < area * double(small);
}

int launch_sgemm128(const Gemm &g, cudaStream_t s) {
    using namespace dev::sg;
    dim3 grid(unsigned((g.M + TM - 1) / TM), unsigned((g.N + TN - 1) / TN));
    const SimtParams<float> p{g.ta, g.tb, int(g.M), int(g.N), int(g.K), float(g.alpha.re), float(g.beta.re),
                              static_cast<const float *>(g.A), g.lda, static_cast<const float *>(g.B), g.ldb,
                              static_cast<float *>(g.C), g.ldc, g.beta_zero() ? 1 : 0, g.uplo, g.diag};
    sgemm128_kernel<<<grid, sg::THR, 0, s>>>(p, g.guard);
    BX_CUDA(cudaGetLastError());
    count_launch();
    return BLASX_OK;
}

}  // namespace bx
