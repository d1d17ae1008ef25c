// ozaki_stats.cuh -- operand statistics and the modulus decision of a
// standalone emulated GEMM, as one launch over both operands.
//
// What bounds it: the operands are read once (HBM), so a block must keep many
// loads in flight and the grid must fill the GPU for a row-contiguous operand
// of a few thousand rows too. An operand is cut into groups of rows (8 for a
// k-contiguous source, one warp per row; 64 for a row-contiguous one, warps
// striding over k) times chunks of k; the chunk count follows from the number
// of groups, so that kStatsBlocks blocks exist where the least chunk allows it
// (two k-contiguous operands of 2048 x 2048 make 1024). Each chunk leaves its
// partial sums in scratch, the block that arrives last at its group adds them
// in chunk order (the result does not depend on timing), and the block that
// arrives last of all reduces the groups and decides.
//
// One thread per row over 512 k with atomics, a second launch for the other
// operand and a one-block decision kernel took 81 + 12 + 16 us at 2048^3 and
// 138 + 15 + 18 us for a complex128 product of 2401 x 1639 x 1203; see the
// launch in ozaki.cu for what this form takes.
#pragma once

#include <algorithm>

#include "ozaki_dev.cuh"

namespace bx {
namespace oz {
namespace {

constexpr int kStatsThreads = 256;
constexpr int kStatsBlocks = 148 * 12;  // blocks aimed at, both operands together
constexpr int kKcRows = 8, kRcRows = 64;   // rows per group
constexpr int kKcMinChunk = 1024, kRcMinChunk = 128;  // least k per chunk

struct StatsSide {
    View v;
    RowStats st;
    int kc;       // k-contiguous source
    int groups, chunks;
    int64_t kchunk;
    double *part;    // [chunks][3][R]: max, sum of squares, sum of magnitudes (max = -1: non-finite seen)
    double *grho, *gratio;  // per group: max rho, min ||x||_2 / max|x|
    int *arrive;     // per group, zeroed
};
struct StatsArgs {
    StatsSide s[2];
    int sides;       // 1 when op(B) is op(A)^T
    int total_groups;
    int *arrive;     // zeroed
    int64_t K;
    double unit;
    int mode, forced;
    Decision *dec;
};

// Geometry of one operand; scratch is its own slice buffer, written only
// after the decision (at least 20 bytes per padded row and k, the partials
// take 24 bytes per row and chunk of 128 k or more and 16 per group).
inline StatsSide stats_side(const View &v, const RowStats &st, bool kc, void *scratch) {
    StatsSide s;
    s.v = v;
    s.st = st;
    s.kc = kc;
    const int rows = kc ? kKcRows : kRcRows;
    s.groups = int((v.R + rows - 1) / rows);
    const int64_t least = kc ? kKcMinChunk : kRcMinChunk;
    const int64_t most = (v.K + least - 1) / least;
    const int64_t want = std::max<int64_t>(1, kStatsBlocks / (2 * int64_t(s.groups)));
    s.chunks = int(std::min(want, most));
    s.kchunk = (v.K + s.chunks - 1) / s.chunks;
    s.grho = static_cast<double *>(scratch);
    s.gratio = s.grho + s.groups;
    s.part = s.gratio + s.groups;
    s.arrive = st.flags;
    return s;
}

// One element's contribution.
__device__ __forceinline__ void stats_add(double re, double im, double &amax, double &ssq, double &sab, bool &bad) {
    bad = bad || !(isfinite(re) && isfinite(im));
    const double ar = fabs(re), ai = fabs(im);
    amax = fmax(amax, fmax(ar, ai));
    ssq = fma(re, re, fma(im, im, ssq));
    sab += ar + ai;
}

template <typename T>
__device__ __forceinline__ void stats_load(const T *p, double &re, double &im) {
    if constexpr (Elem<T>::cplx) {
        using R = typename Elem<T>::R;
        const R *q = reinterpret_cast<const R *>(p);
        re = double(q[0]);
        im = double(q[1]);  // its sign does not matter here
    } else {
        re = double(*p);
        im = 0.0;
    }
}

// rho = ||x||_2 sqrt(K) / ||x||_1 and ||x||_2 / max|x| of one row from its
// sums; the neutral values for a zero row.
__device__ __forceinline__ void row_spread(double amax, double ssq, double sab, double rootk, double &rho,
                                           double &ratio) {
    rho = 0.0;
    ratio = 1e300;
    if (sab > 0) {
        const double n2 = sqrt(ssq);
        rho = n2 * rootk / sab;
        ratio = n2 / amax;
    }
}

// The modulus count from the extremes over all rows, by one warp: lane n
// evaluates kMinModuli + n moduli (the estimate of decide_body).
__device__ __forceinline__ void decide_warp(const StatsArgs &a, const double (&rho)[2], const double (&ratio)[2],
                                            bool bad, int lane) {
    const double ra = fmax(rho[0], 1.0), rb = fmax(rho[1], 1.0);
    const double ha = ratio[0] > 1e299 ? 0.0 : log2(ratio[0]);
    const double hb = ratio[1] > 1e299 ? 0.0 : log2(ratio[1]);
    const int ni = min(lane, kNumN - 1), n = ni + kMinModuli;
    const double qa = fmin(double(c_crt.Q[ni]), kP + ha);
    const double qb = fmin(double(c_crt.Q[ni]), kP + hb);
    const double est = 3.0 * ra * rb * exp2(-fmin(qa, qb)) / a.unit;
    const bool ok = lane < kNumN && (a.forced ? n == a.forced : est <= 0.5);
    const unsigned hit = __ballot_sync(0xffffffffu, ok);
    const int at = hit ? __ffs(int(hit)) - 1 : kNumN - 1;
    const double est_at = __shfl_sync(0xffffffffu, est, at);
    if (lane != 0) return;
    int chosen = hit ? at + kMinModuli : 0;
    if (!chosen && a.mode == 2) chosen = kMaxModuli;
    if (bad) chosen = 0;  // Inf/NaN: the native kernel propagates them
    Decision d;
    d.nmod = d.slices = chosen;
    d.spread = ra * rb;
    d.q = chosen ? c_crt.Q[chosen - kMinModuli] : 0;
    d.estimate = est_at;
    d.nonfinite = bad;
    d.pad = 0;
    *a.dec = d;
}

// Block `b` of one side (a group and a chunk of it); true when the block
// finished its group, with the group's extremes stored.
template <typename T>
__device__ __forceinline__ bool stats_group(const StatsSide &s, int64_t b, double rootk, int tid) {
    __shared__ double sm[3][8][kRcRows];  // per warp: the rows' partial values
    __shared__ double s_rho[kRcRows], s_ratio[kRcRows];
    __shared__ int s_last;
    const int lane = tid & 31, warp = tid >> 5;
    const int group = int(b / s.chunks), chunk = int(b % s.chunks);
    const int64_t R = s.v.R;
    const int64_t k0 = chunk * s.kchunk, k1 = min(s.v.K, k0 + s.kchunk);
    const T *p = static_cast<const T *>(s.v.p);
    const int rows = s.kc ? kKcRows : kRcRows;
    const int64_t r0 = int64_t(group) * rows;
    if (s.kc) {
        constexpr int U = Elem<T>::cplx ? 4 : 8;  // loads in flight per lane
        const int64_t r = r0 + warp;
        double amax = 0, ssq = 0, sab = 0;
        bool bad = false;
        if (r < R) {
            const T *q = p + r * s.v.ld;
            for (int64_t k = k0 + lane; k < k1; k += 32 * U) {
                double re[U], im[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    re[u] = im[u] = 0.0;
                    if (k + 32 * u < k1) stats_load<T>(q + k + 32 * u, re[u], im[u]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) stats_add(re[u], im[u], amax, ssq, sab, bad);
            }
        }
        for (int o = 16; o; o >>= 1) {
            amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
            sab += __shfl_xor_sync(0xffffffffu, sab, o);
        }
        bad = __any_sync(0xffffffffu, bad);
        if (lane == 0) {
            sm[0][0][warp] = bad ? -1.0 : amax;
            sm[1][0][warp] = ssq;
            sm[2][0][warp] = sab;
        }
        __syncthreads();
    } else {
        // a lane holds rows lane and lane + 32 of the group
        constexpr int U = 4;
        double amax[2] = {0, 0}, ssq[2] = {0, 0}, sab[2] = {0, 0};
        bool bad[2] = {false, false};
        const bool in[2] = {r0 + lane < R, r0 + lane + 32 < R};
        const T *q = p + r0 + lane;
        for (int64_t k = k0 + warp; k < k1; k += 8 * U) {
            double re[2][U], im[2][U];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    re[h][u] = im[h][u] = 0.0;
                    if (in[h] && k + 8 * u < k1) stats_load<T>(q + (k + 8 * u) * s.v.ld + 32 * h, re[h][u], im[h][u]);
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int h = 0; h < 2; ++h) stats_add(re[h][u], im[h][u], amax[h], ssq[h], sab[h], bad[h]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            sm[0][warp][lane + 32 * h] = bad[h] ? -1.0 : amax[h];
            sm[1][warp][lane + 32 * h] = ssq[h];
            sm[2][warp][lane + 32 * h] = sab[h];
        }
        __syncthreads();
        if (tid < kRcRows) {
            double m = sm[0][0][tid], q2 = sm[1][0][tid], q1 = sm[2][0][tid];
            bool neg = m < 0;
#pragma unroll
            for (int w = 1; w < 8; ++w) {
                neg = neg || sm[0][w][tid] < 0;
                m = fmax(m, sm[0][w][tid]);
                q2 += sm[1][w][tid];
                q1 += sm[2][w][tid];
            }
            sm[0][0][tid] = neg ? -1.0 : m;
            sm[1][0][tid] = q2;
            sm[2][0][tid] = q1;
        }
    }
    // the first `rows` threads hold one row each from here on
    const int64_t r = r0 + tid;
    const bool mine = tid < rows && r < R;
    if (s.chunks > 1) {
        if (mine) {
            double *w = s.part + int64_t(chunk) * 3 * R + r;
#pragma unroll
            for (int q = 0; q < 3; ++q) w[q * R] = sm[q][0][tid];
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(s.arrive + group, 1) == s.chunks - 1;
        __syncthreads();
        if (!s_last) return false;
        __threadfence();
    }
    double rho = 0.0, ratio = 1e300;
    bool bad = false;
    if (mine) {
        double m, q2, q1;
        if (s.chunks > 1) {
            m = q2 = q1 = 0.0;
            const double *w = s.part + r;
#pragma unroll 4
            for (int c = 0; c < s.chunks; ++c, w += 3 * R) {
                const double wm = __ldcg(w);
                bad = bad || wm < 0;
                m = fmax(m, wm);
                q2 += __ldcg(w + R);
                q1 += __ldcg(w + 2 * R);
            }
        } else {
            m = sm[0][0][tid];
            bad = m < 0;
            q2 = sm[1][0][tid];
            q1 = sm[2][0][tid];
        }
        s.st.amax[r] = m;
        s.st.sumsq[r] = q2;
        row_spread(m, q2, q1, rootk, rho, ratio);
        if (bad) ratio = -1.0;  // marks the group; the other values no longer matter
    }
    if (tid < rows) {
        s_rho[tid] = rho;
        s_ratio[tid] = ratio;
    }
    __syncthreads();
    if (warp == 0) {
        for (int i = lane + 32; i < rows; i += 32) {
            rho = fmax(rho, s_rho[i]);
            ratio = fmin(ratio, s_ratio[i]);
        }
        for (int o = 16; o; o >>= 1) {
            rho = fmax(rho, __shfl_xor_sync(0xffffffffu, rho, o));
            ratio = fmin(ratio, __shfl_xor_sync(0xffffffffu, ratio, o));
        }
        if (lane == 0) {
            s.grho[group] = rho;
            s.gratio[group] = ratio;
        }
    }
    return true;
}

// Blocks [0, groups * chunks) of side 0, then those of side 1.
template <typename T> __global__ void __launch_bounds__(kStatsThreads) stats_decide_kernel(const StatsArgs a) {
    __shared__ int s_final;
    __shared__ double s_ext[4][8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double rootk = sqrt(double(a.K));
    const int64_t n0 = int64_t(a.s[0].groups) * a.s[0].chunks;
    const int64_t b = blockIdx.x;
    const bool second = b >= n0;
    if (!stats_group<T>(second ? a.s[1] : a.s[0], second ? b - n0 : b, rootk, tid)) return;
    if (tid == 0) {
        __threadfence();
        s_final = atomicAdd(a.arrive, 1) == a.total_groups - 1;
    }
    __syncthreads();
    if (!s_final) return;
    __threadfence();
    double rho[2] = {0, 0}, ratio[2] = {1e300, 1e300};
    for (int sd = 0; sd < a.sides; ++sd)
        for (int i = tid; i < a.s[sd].groups; i += kStatsThreads) {
            rho[sd] = fmax(rho[sd], __ldcg(a.s[sd].grho + i));
            ratio[sd] = fmin(ratio[sd], __ldcg(a.s[sd].gratio + i));
        }
    for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int sd = 0; sd < 2; ++sd) {
            rho[sd] = fmax(rho[sd], __shfl_xor_sync(0xffffffffu, rho[sd], o));
            ratio[sd] = fmin(ratio[sd], __shfl_xor_sync(0xffffffffu, ratio[sd], o));
        }
    if (lane == 0) {
        s_ext[0][warp] = rho[0];
        s_ext[1][warp] = rho[1];
        s_ext[2][warp] = ratio[0];
        s_ext[3][warp] = ratio[1];
    }
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (int w = 0; w < 8; ++w)
#pragma unroll
        for (int sd = 0; sd < 2; ++sd) {
            rho[sd] = fmax(rho[sd], s_ext[sd][w]);
            ratio[sd] = fmin(ratio[sd], s_ext[2 + sd][w]);
        }
    if (a.sides == 1) {
        rho[1] = rho[0];
        ratio[1] = ratio[0];
    }
    decide_warp(a, rho, ratio, ratio[0] < 0 || ratio[1] < 0, lane);
}

// ---- the pair sample beside the slices ------------------------------------------
//
// In auto mode the first blocks of a slice launch take the pair sample; the
// last of them sets the modulus count to zero, so that the residue GEMM and
// the reconstruction do nothing and the native kernel runs, when the operands'
// large entries do not meet. (Decision::slices keeps the count for the slices
// that run meanwhile.) As part of the statistics the sample's chain of loads
// and hand-overs delayed the decision: 7.6 us at FP64 2048^3, 10.3 at FP32
// 3001 x 1777 x 999. Beside the slices it costs about 1 us there. The chunks are
// added in two levels, groups of 16 or the square root of their number.
constexpr int kPairMaxGroup = 32, kPairCounters = kPairMaxGroup + 1;
struct PairVeto {
    PairSample p;  // no chunks: no sample
    int group;     // chunks per group
    int *arrive;   // zeroed: per group, then for the groups
    Decision *dec;
};
// counters: kPairCounters words.
inline PairVeto pair_veto(const View &va, bool akc, const RowStats &sa, const View &vb, bool bkc, const RowStats &sb,
                          int uplo, int64_t diag, const Parts &pt, int *counters, Decision *dec) {
    PairVeto a;
    // (128 chunks fit the smallest scratch; slots for the groups and the result)
    const int64_t room = std::max<int64_t>(128, pt.pair_slots - kPairCounters - 1);
    a.p = pair_sample(va, akc, sa, vb, bkc, sb, uplo, diag,
                      int(std::min<int64_t>(room, kPairMaxGroup * kPairMaxGroup)), pt.pair);
    a.group = 16;
    while (a.group * a.group < a.p.chunks) ++a.group;
    a.arrive = counters;
    a.dec = dec;
    return a;
}

// Counts one arrival of `of` at `counter`; true in every thread of the block
// that is the last one, which may then read what the others left.
__device__ __forceinline__ bool last_arrival(int *counter, int of, int tid) {
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(counter, 1) == of - 1;
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
    return true;
}

template <typename T>
__device__ __noinline__ void pair_veto_block(const PairVeto &a, int chunk, int tid, void *sh) {
    const PairSample &p = a.p;
    if (a.dec->slices == 0) return;  // native already
    const int per = a.group, groups = (p.chunks + per - 1) / per, group = chunk / per;
    const int n = min(per, p.chunks - group * per);
    float *sums = p.part + int64_t(p.chunks) * kPairPart;
    pair_chunk_body<T>(p, chunk, tid, static_cast<__nv_bfloat16 *>(sh));
    if (!last_arrival(a.arrive + group, n, tid)) return;
    const float *in = p.part;
    int count = n;
    if (groups > 1) {
        reinterpret_cast<float4 *>(sums + int64_t(group) * kPairPart)[tid] =
            pair_add(p.part + int64_t(group) * per * kPairPart, n, tid);
        if (!last_arrival(a.arrive + kPairMaxGroup, groups, tid)) return;
        in = sums;
        count = groups;
    }
    const float least = pair_reduce(p, in, count, tid, static_cast<float *>(sh));
    if (tid == 0) {
        const double est = paired_estimate(a.dec->estimate, a.dec->spread, least);
        a.dec->estimate = est;
        if (!(est <= 0.5)) a.dec->nmod = 0;
    }
}

}  // namespace
}  // namespace oz
}  // namespace bx
