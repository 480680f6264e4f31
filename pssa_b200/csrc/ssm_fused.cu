// Fused selective-SSM stage: discretise, scan and read out in one pass, state in registers.
//
//   a = exp(delta_i * A_ij);  b = delta_i * B_j;  h_ij <- a*h_ij + b*x_i;  y_i = sum_j h_ij * C_j
//
// Replaces the reference's three kernels ssm_prepare / affine_scan / ssm_materialize
// (src/cuda/stages.ptx:8-65, launched from src/cuda/stages.rs:260-356), which write three
// [T, d*s] arrays to HBM and read them back twice, and the CPU stage src/gpu_batch.rs:543-680.
// Here the only HBM traffic is the inputs (delta, x, B, C: (2d + 2s) floats per token), y, and the
// carry once per lane; the per-token maps never leave registers. The kernel is therefore bound by
// the exp throughput (d*s per token), not by HBM.
//
// Work split: one CTA = one lane (independent sequence) x CH consecutive channels i; a channel's
// s states are spread over G threads of one warp holding ST states each (G*ST >= s), in pieces of four that
// alternate between the groups. Inside a warp the 32/G threads that own the same group sit in adjacent lanes, so the
// B_j / C_j pieces a thread needs are one shared-memory address per group (a broadcast) and the groups' pieces lie side
// by side (no bank conflicts); y is completed over the G groups by shuffles.
// Time is walked serially by every thread; token tiles (delta, x, B, C rows) are staged through a
// cp.async ring in shared memory so the global-load latency is hidden behind the previous tile's exps.
//
// Two arithmetic modes:
//   FAST  ex2.approx on delta*(A*log2 e) (the reference's own GPU recipe, stages.ptx:21-22),
//         FMA contraction, y summed per thread then by a shuffle tree over the G threads.
//   EXACT exp_exact, separately rounded multiply/add in the reference's order (src/pssa.rs:1131-1144);
//         with G == 1 the sum over j is the reference's sequential sum.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <math_constants.h>

#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "bounds.hpp"
#include "context.hpp"
#include "kernels.hpp"

namespace pssa {
namespace {

constexpr int kThreads = 256;  // default CTA size; the 16-state fast configuration also comes with 352 (see launch_ssm_fused)
// tokens per staged tile; the widest state split keeps 8 so its stages stay inside the shared memory of one SM. The
// 64-state configuration (four lanes per channel) takes 32 tokens in two stages: the same shared memory as 16 tokens in
// three, half as many CTA-wide barriers (12.07 against 12.19 ms per step for the twelve launches of the benchmark)
template <int G>
constexpr int kTileTokensFor = G >= 32 ? 8 : (G == 4 ? 32 : 16);
// The 16-state fast configuration is capped at 64 registers so four CTAs (32 warps) share an SM: the kernel is bound by
// dependent-issue latency, not by a pipe, and the extra warps are worth more than the 16 bytes of spill they cost.
constexpr int kMinCtasFast = 4;
constexpr int kStages = 2;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// exp for the exact mode: x = n ln 2 + r by a two-part ln 2, e^r = 1 + (r + r^2 q(r)) with a quartic q (least largest relative
// error on |r| <= ln 2 / 2, fitted by linear programming: 2^-28.3), n added to the exponent. For the decays of the
// recurrence (-0.08 < x <= 0) 97 % of the results are the correctly rounded ones (largest error 0.57 ulp), which is what the
// reference's host libm returns, so its states are met in far more bits than with a 1 to 2 ulp exp; and the XU pipe is not
// used. Below -1 90 % are, and the largest error is 1.0 ulp. Results near or below the smallest normal number, and overflow, are left to expf.
__device__ __forceinline__ float exp_exact(float x) {
    const float t = fmaf(x, 1.4426950408889634f, 12582912.0f);  // 1.5 * 2^23: the integer part ends up in the low bits
    const float n = t - 12582912.0f;
    float r = fmaf(n, -0.693145751953125f, x);
    r = fmaf(n, -1.4286068202862268e-06f, r);
    float q = 0.0013814537087455392f;
    q = fmaf(q, r, 0.00836874544620514f);
    q = fmaf(q, r, 0.04166838899254799f);
    q = fmaf(q, r, 0.1666652113199234f);
    q = fmaf(q, r, 0.4999999403953552f);
    const float e = 1.0f + fmaf(q, __fmul_rn(r, r), r);
    const float y = __int_as_float(__float_as_int(e) + (__float_as_int(t) << 23));
    return fabsf(x) < 87.0f ? y : expf(x);
}

// Packed fp32 pairs (one instruction, two IEEE-rounded results): the kernel is bound by instruction issue, and the
// per-state multiply / fma work is half the instruction stream.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// to [-126, 128], where 2^128 is infinity; a NaN stays one
__device__ __forceinline__ float clamp_exp2(float x) {
    float y;
    asm("max.NaN.f32 %0, %1, 0fC2FC0000;\n\tmin.NaN.f32 %0, %0, 0f43000000;" : "=f"(y) : "f"(x));
    return y;
}
// 2^x for a pair of x on the FMA pipe: x = n + f with |f| <= 1/2 by adding and taking off 1.5 * 2^23, 2^f by a degree-5
// polynomial with p(0) = 1 (least largest relative error under that constraint, fitted by linear programming: 2^-22.5 after
// fp32 rounding, mean -2e-8), n added to the exponent. Below 2^-126 the result stays at that size instead of going to zero.
__device__ __forceinline__ f32x2 exp2_poly2(f32x2 x) {
    float x0, x1;
    unpack2(x, x0, x1);
    x = pack2(clamp_exp2(x0), clamp_exp2(x1));
    const f32x2 t = add2(x, pack2(12582912.0f, 12582912.0f));
    const f32x2 f = fma2(add2(t, pack2(-12582912.0f, -12582912.0f)), pack2(-1.0f, -1.0f), x);
    f32x2 r = pack2(0.001326472731307149f, 0.001326472731307149f);
    r = fma2(r, f, pack2(0.009671512991189957f, 0.009671512991189957f));
    r = fma2(r, f, pack2(0.05550733581185341f, 0.05550733581185341f));
    r = fma2(r, f, pack2(0.24022242426872253f, 0.24022242426872253f));
    r = fma2(r, f, pack2(0.6931470036506653f, 0.6931470036506653f));
    r = fma2(r, f, pack2(1.0f, 1.0f));
    float t0, t1, r0, r1;
    unpack2(t, t0, t1);
    unpack2(r, r0, r1);
    r = pack2(__int_as_float(__float_as_int(r0) + (__float_as_int(t0) << 23)), __int_as_float(__float_as_int(r1) + (__float_as_int(t1) << 23)));
    return fma2(x, pack2(0.0f, 0.0f), r);  // a NaN, which the additions to the exponent turn into a number, is one again
}
// 2^x for a pair of x in [-0.4, 0]: no range reduction, a degree-4 polynomial with p(0) = 1 (least largest relative error under that
// constraint, fitted by linear programming: 2^-23.4 after fp32 rounding, rms 2^-25.0; ex2.approx has 2^-22.9 and 2^-24.6 there).
constexpr float kSmallArg = 0.4f;
__device__ __forceinline__ f32x2 exp2_small2(f32x2 x) {
    f32x2 r = pack2(0.008396584540605545f, 0.008396584540605545f);
    r = fma2(r, x, pack2(0.05509750917553902f, 0.05509750917553902f));
    r = fma2(r, x, pack2(0.24017220735549927f, 0.24017220735549927f));
    r = fma2(r, x, pack2(0.6931449174880981f, 0.6931449174880981f));
    return fma2(r, x, pack2(1.0f, 1.0f));
}
__device__ __forceinline__ f32x2 exp2_approx2(f32x2 x) {
    float x0, x1;
    unpack2(x, x0, x1);
    return pack2(ex2_approx(x0), ex2_approx(x1));
}

// Which CTA of the lanes x channel blocks this one is. CTAs go to the SMs in rounds; lanes of different lengths come longest first, and
// every second round runs backwards, so that an SM with a long lane's CTA of one round gets a shorter one's of the next (seven
// prompts of 33 to 1501 tokens at d 768: 157 us a launch in the caller's order and with early starts, 143 in this).
__device__ __forceinline__ unsigned ssm_cta(unsigned per_round) {
    const unsigned b = blockIdx.x;
    if (per_round == 0) return b;
    const unsigned round = b / per_round, first = round * per_round;
    return (round & 1) && first + per_round <= gridDim.x ? first + (per_round - 1 - (b - first)) : b;
}

// MAPS: the first of the two passes over time chunks. It leaves every chunk's affine map at `sum_delta` (sum of delta, then the
// end state from a zero carry) and no y: what would form and store it, a third of the instructions, is not in it.
template <int ST, int G, bool EXACT, bool TAPE, int THR = kThreads, int CPT = 1, bool MAPS = false>
__global__ void __launch_bounds__(THR, (ST <= 16 && !TAPE && !EXACT) ? (CPT > 1 ? 3 : THR > 256 ? 2 : kMinCtasFast) : 1) ssm_fused_kernel(SsmParams p) {
    // CPT channels per thread (fast mode without tape only): a token's B and C rows are loaded once for both channels and
    // the two recurrences are independent instruction streams, so a warp-token of twice the work takes fewer than twice
    // the instructions.
    static_assert(CPT == 1 || (CPT == 2 && !EXACT && !TAPE), "two channels per thread exist for the fast mode only");
    pdl_trigger();  // the next kernel in the stream may start its prologue now ...
    pdl_wait();     // ... and this one, if launched as a dependent, waits here for its own predecessor
    constexpr int kThreads = THR;     // shadows the default: every stride below follows this instantiation's CTA size
    constexpr int CH = kThreads / G * CPT;  // channels per CTA
    constexpr int kTileTokens = kTileTokensFor<G>;
    constexpr int LPG = 32 / G;       // lanes of a warp that share one state group
    constexpr int SP = ST * G;        // floats per token row of B / C in shared memory
    constexpr int QS = 4 * G;         // a thread's states lie in pieces of four, this far apart
    extern __shared__ __align__(16) float smem[];
    float* sm_delta = smem;                                   // [kStages][kTileTokens][CH]
    float* sm_x = sm_delta + kStages * kTileTokens * CH;      // [kStages][kTileTokens][CH]
    float* sm_b = sm_x + kStages * kTileTokens * CH;          // [kStages][kTileTokens][SP]
    float* sm_c = sm_b + kStages * kTileTokens * SP;          // [kStages][kTileTokens][SP]

    const int tid = threadIdx.x;
    const int lane_id = tid & 31;
    const int g = lane_id / LPG;
    const int c = (tid >> 5) * LPG + lane_id % LPG;
    const int ncb = (p.d + CH - 1) / CH;
    const unsigned cta = ssm_cta(p.ragged);
    const int lane = cta / ncb;
    const int i0 = (cta % ncb) * CH;
    const int i = i0 + CPT * c;  // a two-channel thread owns the adjacent channels CPT * c and CPT * c + 1
    const bool valid = i < p.d;
    const size_t row0 = p.offsets ? p.offsets[lane] : 0;
    const int len = p.lengths ? (int)p.lengths[lane] : (int)p.rows;
    const int d = p.d, s = p.s;
    const size_t ds = (size_t)d * s;
    const int j0 = g * 4;
    const size_t ldd = p.ld_delta ? p.ld_delta : (size_t)d;
    const size_t ldbc = p.ld_bc ? p.ld_bc : (size_t)s;
    float* carry = p.carry && !MAPS ? p.carry + (size_t)(p.lane_slots ? p.lane_slots[lane] : lane) * (p.carry_stride ? p.carry_stride : ds)
                                    : nullptr;

    float A[ST], h[ST];
    float A1[CPT > 1 ? ST : 1], h1[CPT > 1 ? ST : 1];  // the second channel of a two-channel thread
    const int i1 = i + 1;
    const bool valid1 = CPT > 1 && i1 < p.d;
    // pieces of four states: 16-byte accesses when the layout allows
    const bool vec_state = p.aligned && (s & 3) == 0 && (reinterpret_cast<uintptr_t>(p.rates) & 15) == 0 &&
                           (reinterpret_cast<uintptr_t>(carry) & 15) == 0;
    auto load_state = [&](float* Av, float* hv, int ch, bool ok_ch) {
        if (vec_state) {
#pragma unroll
            for (int q = 0; q < ST / 4; ++q) {
                const bool ok = ok_ch && (j0 + q * QS) < s;
                const float4 r4 = ok ? __ldg(reinterpret_cast<const float4*>(p.rates + (size_t)ch * s + j0 + q * QS)) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 h4 = (ok && carry) ? *(reinterpret_cast<const float4*>(carry + (size_t)ch * s + j0 + q * QS)) : make_float4(0.f, 0.f, 0.f, 0.f);
                Av[q * 4] = r4.x, Av[q * 4 + 1] = r4.y, Av[q * 4 + 2] = r4.z, Av[q * 4 + 3] = r4.w;
                hv[q * 4] = h4.x, hv[q * 4 + 1] = h4.y, hv[q * 4 + 2] = h4.z, hv[q * 4 + 3] = h4.w;
            }
            if (!EXACT) {
#pragma unroll
                for (int jj = 0; jj < ST; ++jj) Av[jj] *= 1.4426950408889634f;
            }
        } else {
#pragma unroll
            for (int jj = 0; jj < ST; ++jj) {
                const int j = j0 + jj / 4 * QS + jj % 4;
                bool ok = ok_ch && j < s;
                float rate = ok ? __ldg(p.rates + (size_t)ch * s + j) : 0.0f;
                Av[jj] = EXACT ? rate : rate * 1.4426950408889634f;
                hv[jj] = (ok && carry) ? carry[(size_t)ch * s + j] : 0.0f;
            }
        }
    };
    load_state(A, h, i, valid);
    if constexpr (CPT > 1) load_state(A1, h1, i1, valid1);
    // Small arguments. A slow state's delta * A is near zero, and there the exponential is four packed multiply-adds without a range
    // reduction, cheap enough to share the exponentials between the XU and the FMA pipe. Two of a thread's eight pairs (three in the map
    // pass, which forms no y) take that way in every tile whose arguments allow it; a thread's states are interleaved with the other
    // groups' so that its last pieces come from the slow end of a table of ascending timescales. Us a launch at 32 x 2048, 24 x 2048, 16 x
    // 2048 and 1 x 8192 tokens (d 768), with one general polynomial pair in eight before: 945 -> 889, 697 -> 619, 539 -> 474, 115 -> 107;
    // the map pass of 8192 tokens 104 -> 86. The apply pass with 0 / 1 / 3 / 4 pairs: 960 / 922 / 894 / 944.
    // amax: the largest |rate| of those states; infinite if one is positive or NaN
    constexpr bool HAS_SMALL = ST == 16 && G == 4 && !TAPE && !EXACT;
    constexpr int kSmallFrom = ST - (MAPS ? 6 : 4);
    float amax = 0.0f;
    if constexpr (HAS_SMALL) {
#pragma unroll
        for (int jj = kSmallFrom; jj < ST; ++jj) {
            amax = A[jj] <= 0.0f ? fmaxf(amax, -A[jj]) : CUDART_INF_F;
            if constexpr (CPT > 1) amax = A1[jj] <= 0.0f ? fmaxf(amax, -A1[jj]) : CUDART_INF_F;
        }
    }
    float sum_t = 0.0f, sum_t1 = 0.0f;  // MAPS: delta summed over the tile, and over the chunk in f64
    double sum_d = 0.0, sum_d1 = 0.0;

    const int ntiles = (len + kTileTokens - 1) / kTileTokens;

    auto load_tile = [&](int k) {
        if (k < ntiles) {
            const int st = k % kStages;
            const int t0 = k * kTileTokens;
            const int nt = min(kTileTokens, len - t0);
            float* dd = sm_delta + st * kTileTokens * CH;
            float* dx = sm_x + st * kTileTokens * CH;
            float* db = sm_b + st * kTileTokens * SP;
            float* dc = sm_c + st * kTileTokens * SP;
            if (p.aligned) {
                constexpr int CQ = CH / 4 > 0 ? CH / 4 : 1;
                for (int idx = tid; idx < nt * CQ; idx += kThreads) {
                    int tt = idx / CQ, q = idx % CQ;
                    int col = i0 + q * 4;
                    size_t gro = (row0 + t0 + tt) * (size_t)d + col;
                    if (CH >= 4 && col < d) {
                        cp_async16(dd + tt * CH + q * 4, p.delta + (row0 + t0 + tt) * ldd + col);
                        cp_async16(dx + tt * CH + q * 4, p.x_norm + gro);
                    } else if (CH >= 4) {
                        *reinterpret_cast<float4*>(dd + tt * CH + q * 4) = make_float4(0, 0, 0, 0);
                        *reinterpret_cast<float4*>(dx + tt * CH + q * 4) = make_float4(0, 0, 0, 0);
                    }
                }
                constexpr int SQ = ST * G / 4;
                for (int idx = tid; idx < nt * SQ; idx += kThreads) {
                    int tt = idx / SQ, q = idx % SQ;
                    int j = q * 4;
                    int dst = tt * SP + j;
                    size_t gro = (row0 + t0 + tt) * ldbc + j;
                    if (j < s) {
                        cp_async16(db + dst, p.b_proj + gro);
                        cp_async16(dc + dst, p.c_proj + gro);
                    } else {
                        *reinterpret_cast<float4*>(db + dst) = make_float4(0, 0, 0, 0);
                        *reinterpret_cast<float4*>(dc + dst) = make_float4(0, 0, 0, 0);
                    }
                }
            } else {
                for (int idx = tid; idx < nt * CH; idx += kThreads) {
                    int tt = idx / CH, q = idx % CH;
                    int col = i0 + q;
                    size_t gro = (row0 + t0 + tt) * (size_t)d + col;
                    dd[tt * CH + q] = col < d ? __ldg(p.delta + (row0 + t0 + tt) * ldd + col) : 0.0f;
                    dx[tt * CH + q] = col < d ? __ldg(p.x_norm + gro) : 0.0f;
                }
                for (int idx = tid; idx < nt * ST * G; idx += kThreads) {
                    int tt = idx / (ST * G), j = idx % (ST * G);
                    int dst = tt * SP + j;
                    size_t gro = (row0 + t0 + tt) * ldbc + j;
                    db[dst] = j < s ? __ldg(p.b_proj + gro) : 0.0f;
                    dc[dst] = j < s ? __ldg(p.c_proj + gro) : 0.0f;
                }
            }
        }
        cp_async_commit();
    };

#pragma unroll
    for (int k = 0; k < kStages - 1; ++k) load_tile(k);

    for (int k = 0; k < ntiles; ++k) {
        // tile k has landed once at most kStages-2 newer groups are in flight; the barrier also means every thread is
        // done with tile k-1 (its stage is the one the prefetch below overwrites)
        cp_async_wait<kStages - 2>();
        __syncthreads();
        load_tile(k + kStages - 1);
        const int st = k % kStages;
        const int t0 = k * kTileTokens;
        const int nt = min(kTileTokens, len - t0);
        float* dd = sm_delta + st * kTileTokens * CH;
        const float* dx = sm_x + st * kTileTokens * CH;
        const float* db = sm_b + st * kTileTokens * SP + j0;
        const float* dc = sm_c + st * kTileTokens * SP + j0;
        // one token's recurrence; yp, ypb: this thread's part of y
        auto token = [&](int tt, auto small_args, float& yp, float& ypb) {
            constexpr bool SMALL = decltype(small_args)::value;
            float dl, xv, dlb = 0.0f, xvb = 0.0f;
            if constexpr (CPT > 1) {  // both channels' values with one 8-byte load each
                const float2 d2 = *reinterpret_cast<const float2*>(dd + tt * CH + 2 * c);
                const float2 x2 = *reinterpret_cast<const float2*>(dx + tt * CH + 2 * c);
                dl = d2.x, dlb = d2.y, xv = x2.x, xvb = x2.y;
            } else {
                dl = dd[tt * CH + c], xv = dx[tt * CH + c];
            }
            const size_t row = row0 + t0 + tt;
            static_assert(ST % 4 == 0, "states per thread are loaded as float4");
            float bj[ST], cj[ST];
#pragma unroll
            for (int q = 0; q < ST / 4; ++q) {
                float4 vb = *reinterpret_cast<const float4*>(db + tt * SP + q * QS);
                float4 vc = make_float4(0.f, 0.f, 0.f, 0.f);
                if constexpr (!MAPS) vc = *reinterpret_cast<const float4*>(dc + tt * SP + q * QS);
                bj[q * 4] = vb.x, bj[q * 4 + 1] = vb.y, bj[q * 4 + 2] = vb.z, bj[q * 4 + 3] = vb.w;
                cj[q * 4] = vc.x, cj[q * 4 + 1] = vc.y, cj[q * 4 + 2] = vc.z, cj[q * 4 + 3] = vc.w;
            }
            yp = 0.0f, ypb = 0.0f;
            float av[TAPE ? ST : 1], bv[TAPE ? ST : 1];
            if (EXACT) {
#pragma unroll
                for (int jj = 0; jj < ST; ++jj) {
                    float a = exp_exact(__fmul_rn(dl, A[jj]));
                    float bb = __fmul_rn(dl, bj[jj]);
                    h[jj] = __fadd_rn(__fmul_rn(a, h[jj]), __fmul_rn(bb, xv));
                    yp = __fadd_rn(yp, __fmul_rn(h[jj], cj[jj]));
                    if (TAPE) av[jj] = a, bv[jj] = bb;
                }
            } else {
                const float w = dl * xv;
                const f32x2 dl2 = pack2(dl, dl), w2 = pack2(w, w);
                f32x2 y2 = pack2(0.0f, 0.0f);
                const float wb = dlb * xvb;
                const f32x2 dlb2 = pack2(dlb, dlb), wb2 = pack2(wb, wb);
                f32x2 yb2 = pack2(0.0f, 0.0f);
#pragma unroll
                for (int jj = 0; jj < ST; jj += 2) {
                    const f32x2 b2 = pack2(bj[jj], bj[jj + 1]), c2 = pack2(cj[jj], cj[jj + 1]);
                    // one pair of exponentials in eight goes to the FMA pipe (the benchmark's launch: 976 us with none, 952 with
                    // one, 1059 with two, whose extra issue slots cost more than the XU pipe gains)
                    // (the map pass, which has no y to form, takes two: 109 -> 105 us for 8192 tokens)
                    const bool poly = !SMALL && ST == 16 && G == 4 && !TAPE && (jj == 0 || (MAPS && jj == 8));
                    auto exp2_of = [&](f32x2 x) { return SMALL && jj >= kSmallFrom ? exp2_small2(x) : poly ? exp2_poly2(x) : exp2_approx2(x); };
                    const f32x2 a2 = exp2_of(mul2(dl2, pack2(A[jj], A[jj + 1])));
                    f32x2 h2 = fma2(a2, pack2(h[jj], h[jj + 1]), mul2(w2, b2));
                    unpack2(h2, h[jj], h[jj + 1]);
                    if constexpr (!MAPS) y2 = fma2(h2, c2, y2);
                    if (TAPE) unpack2(a2, av[jj], av[jj + 1]), bv[jj] = dl * bj[jj], bv[jj + 1] = dl * bj[jj + 1];
                    if constexpr (CPT > 1) {
                        f32x2 hb2 = fma2(exp2_of(mul2(dlb2, pack2(A1[jj], A1[jj + 1]))), pack2(h1[jj], h1[jj + 1]), mul2(wb2, b2));
                        unpack2(hb2, h1[jj], h1[jj + 1]);
                        if constexpr (!MAPS) yb2 = fma2(hb2, c2, yb2);
                    }
                }
                float y_lo, y_hi;
                unpack2(y2, y_lo, y_hi);
                yp = y_lo + y_hi;
                if constexpr (CPT > 1) {
                    unpack2(yb2, y_lo, y_hi);
                    ypb = y_lo + y_hi;
                }
            }
            if constexpr (MAPS) sum_t += dl, sum_t1 += dlb;
            if (TAPE) {
#pragma unroll
                for (int jj = 0; jj < ST; ++jj) {
                    const int j = j0 + jj / 4 * QS + jj % 4;
                    if (valid && j < s) {
                        size_t o = row * ds + (size_t)i * s + j;
                        if (p.states) p.states[o] = h[jj];
                        if (p.bar_a) p.bar_a[o] = av[jj];
                        if (p.bar_b) p.bar_b[o] = bv[jj];
                    }
                }
            }
        };
        // y of one token: a shuffle tree over the G groups. (Every reader of the delta slot it goes to sits in this warp and has read it.)
        auto finish = [&](int tt, float yp, float ypb) {
            if constexpr (MAPS) return;
#pragma unroll
            for (int m = LPG; m < 32; m <<= 1) yp += __shfl_xor_sync(0xffffffffu, yp, m);
            if constexpr (CPT > 1) {
#pragma unroll
                for (int m = LPG; m < 32; m <<= 1) ypb += __shfl_xor_sync(0xffffffffu, ypb, m);
                if (g == 0) *reinterpret_cast<float2*>(dd + tt * CH + 2 * c) = make_float2(yp, ypb);
            } else {
                if (g == 0) dd[tt * CH + c] = yp;
            }
        };
        // The same sums for four tokens over four groups at once, each group ending with its token: three shuffles instead of eight and one
        // store instead of four, and the tokens' operand loads are not held up behind one another's stores.
        auto sum_four = [&](const float* v) {
            const bool odd = g & 1, high = g & 2;
            const float r0 = (odd ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[1], LPG);
            const float r1 = (odd ? v[3] : v[2]) + __shfl_xor_sync(0xffffffffu, odd ? v[2] : v[3], LPG);
            return (high ? r1 : r0) + __shfl_xor_sync(0xffffffffu, high ? r0 : r1, 2 * LPG);
        };
        const std::false_type any{};
        auto tile = [&](auto small_args) {
            int tt = 0;
            if (G == 4 && (decltype(small_args)::value || nt == kTileTokens)) {
#pragma unroll 1
                for (int t4 = 0; t4 < kTileTokens; t4 += 4) {
                    float yv[4], yw[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) token(t4 + u, small_args, yv[u], yw[u]);
                    if constexpr (MAPS) continue;
                    const float y = sum_four(yv);
                    if constexpr (CPT > 1) {
                        *reinterpret_cast<float2*>(dd + (t4 + g) * CH + 2 * c) = make_float2(y, sum_four(yw));
                    } else {
                        dd[(t4 + g) * CH + c] = y;
                    }
                }
                return;
            } else if (nt == kTileTokens) {
#pragma unroll 4
                for (; tt < kTileTokens; ++tt) {
                    float yp, ypb;
                    token(tt, small_args, yp, ypb);
                    finish(tt, yp, ypb);
                }
            }
            for (; tt < nt; ++tt) {
                float yp, ypb;
                token(tt, any, yp, ypb);
                finish(tt, yp, ypb);
            }
        };
        bool small = HAS_SMALL && p.small_args && nt == kTileTokens;
        if constexpr (HAS_SMALL) {
            // largest delta of the warp's channels over the tile, each group of lanes looking at its share of the tokens: bit
            // patterns compare like the numbers, and negative deltas and NaNs lie above all others
            unsigned top = 0;
#pragma unroll
            for (int t = 0; t < kTileTokens / G; ++t) {
                const float* dp = dd + (t * G + g) * CH + CPT * c;
                if constexpr (CPT > 1) {
                    const uint2 v = *reinterpret_cast<const uint2*>(dp);
                    top = max(top, max(v.x, v.y));
                } else {
                    top = max(top, *reinterpret_cast<const unsigned*>(dp));
                }
            }
#pragma unroll
            for (int m = LPG; m < 32; m <<= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, m));
            small = __all_sync(0xffffffffu, small && __uint_as_float(top) * amax <= kSmallArg && top < 0x80000000u);
        }
        if (HAS_SMALL && small) tile(std::integral_constant<bool, HAS_SMALL>{});
        else tile(any);
        if constexpr (MAPS) {
            sum_d += (double)sum_t, sum_d1 += (double)sum_t1, sum_t = sum_t1 = 0.0f;
            continue;
        }
        __syncthreads();
        // write the tile's y rows out together: 16-byte stores instead of one predicated scalar store per token
        if (p.aligned) {
            constexpr int CQ = CH / 4;
            for (int idx = tid; idx < nt * CQ; idx += kThreads) {
                const int tt = idx / CQ, q = idx % CQ;
                const int col = i0 + q * 4;
                if (col < d) {
                    const float4 v = *reinterpret_cast<const float4*>(dd + tt * CH + q * 4);
                    const size_t o = (row0 + t0 + tt) * (size_t)d + col;
                    *reinterpret_cast<float4*>(p.y + o) = v;
                    if (p.y_bf16) {
                        __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
                        uint2 pk;
                        pk.x = *reinterpret_cast<unsigned*>(&lo);
                        pk.y = *reinterpret_cast<unsigned*>(&hi);
                        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.y_bf16) + o) = pk;
                    }
                }
            }
        } else {
            for (int idx = tid; idx < nt * CH; idx += kThreads) {
                const int tt = idx / CH, q = idx % CH;
                if (i0 + q < d) {
                    const size_t o = (row0 + t0 + tt) * (size_t)d + i0 + q;
                    p.y[o] = dd[tt * CH + q];
                    if (p.y_bf16) reinterpret_cast<__nv_bfloat16*>(p.y_bf16)[o] = __float2bfloat16_rn(dd[tt * CH + q]);
                }
            }
        }
    }
    cp_async_wait<0>();
    if constexpr (MAPS) {
        float* rec = p.sum_delta + (size_t)lane * p.sum_delta_stride;
        auto store_map = [&](const float* hv, int ch, bool ok_ch, double sum) {
            if (g == 0 && ok_ch) rec[ch] = (float)sum;
#pragma unroll
            for (int q = 0; q < ST / 4; ++q)
                if (ok_ch && j0 + q * QS < s)
                    *reinterpret_cast<float4*>(rec + d + (size_t)ch * s + j0 + q * QS) = make_float4(hv[q * 4], hv[q * 4 + 1], hv[q * 4 + 2], hv[q * 4 + 3]);
        };
        store_map(h, i, valid, sum_d);
        if constexpr (CPT > 1) store_map(h1, i1, valid1, sum_d1);
        return;
    }
    if (carry && len > 0) {
        auto store_state = [&](const float* hv, int ch, bool ok_ch) {
            if (vec_state) {
#pragma unroll
                for (int q = 0; q < ST / 4; ++q)
                    if (ok_ch && j0 + q * QS < s)
                        *reinterpret_cast<float4*>(carry + (size_t)ch * s + j0 + q * QS) = make_float4(hv[q * 4], hv[q * 4 + 1], hv[q * 4 + 2], hv[q * 4 + 3]);
            } else {
#pragma unroll
                for (int jj = 0; jj < ST; ++jj) {
                    const int j = j0 + jj / 4 * QS + jj % 4;
                    if (ok_ch && j < s) carry[(size_t)ch * s + j] = hv[jj];
                }
            }
        };
        store_state(h, i, valid);
        if constexpr (CPT > 1) store_state(h1, i1, valid1);
    }
}

// Few lanes. The kernel above gives a warp eight channels, so one sequence of a 768-channel model is 96 warps on 592
// schedulers; and cutting such sequences into time chunks pays every exponential twice. Here a channel's states are spread
// over more lanes: LPC lanes hold SPL states each, 32 / LPC channels to a warp.
//   * a lane owns pieces of V adjacent states, the pieces LPC * V apart, and neighbouring lanes hold the same states of
//     different channels: a token's B and C are conflict-free 16-byte loads that neighbours share, and the tape (states,
//     bar_a, bar_b) leaves in whole lines.
//   * y needs a sum over the LPC lanes for every token: the lanes leave their partials in shared memory and the tile's sums
//     are taken at its end, a lane per token, so no shuffle sits in the token loop. The exact mode sums the s products of
//     a token one after another there, as the reference does.
//   * few lanes leave a warp alone on its scheduler, so everything has to overlap inside it: see the token loop.
//   * a tile's tail is padded with delta = 0, which leaves the state as it is (exp(0) = 1, input 0).
// What bounds it: alone, a token's dependent instructions (about 85 cycles, 32 of them exponentials); with many warps the
// shared-memory pipe (0.67 of its wavefronts at 8 lanes of 768 channels) and the XU pipe (0.62) side by side.
constexpr int kWideStages = 3;
constexpr int kWideWarps = 4;
template <int LPC, int SPL, int TT, bool EXACT>
constexpr size_t wide_smem_floats() {
    const int ch = kWideWarps * (32 / LPC), s = LPC * SPL;
    return (size_t)kWideStages * TT * (2 * s + 2 * (ch + 4)) + 2 * TT * (ch + 4) + 2 * (size_t)TT * (ch + 1) * 4 +
           (EXACT ? (size_t)kWideWarps * 32 * (s + 1) : (size_t)kWideWarps * TT * 36);
}

__device__ __forceinline__ void cp_async16_zfill(void* smem, const void* gmem, bool live) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(live ? 16 : 0));
}

template <int V> struct WideVec;
template <> struct WideVec<2> { typedef float2 type; };
template <> struct WideVec<4> { typedef float4 type; };

template <int LPC, int SPL, int TT, bool EXACT, bool TAPE>
__global__ void __launch_bounds__(kWideWarps * 32) ssm_wide_kernel(SsmParams p) {
    pdl_trigger();
    pdl_wait();
    constexpr int WARPS = kWideWarps;      // TT: tokens per staged tile
    constexpr int S = LPC * SPL;           // states per channel
    constexpr int V = SPL < 4 ? SPL : 4;   // adjacent states of a lane: one 8- or 16-byte access
    constexpr int NQ = SPL / V;            // such pieces per lane, LPC * V states apart
    constexpr int NP = SPL / 2;            // state pairs per lane
    constexpr int CPW = 32 / LPC;          // channels per warp
    constexpr int CH = WARPS * CPW;        // channels per CTA
    constexpr int THR = WARPS * 32;
    constexpr int CQ = CH / 4, SQ = S / 4;
    constexpr int DP = CH + 4, WP = CH + 1;  // token pitches that spread the banks over tokens
    typedef typename WideVec<V>::type vec;
    static_assert(CH % 4 == 0 && (!EXACT || TT % LPC == 0) && TT % 8 == 0, "tile shapes");
    extern __shared__ __align__(16) float smem[];
    float* sm_b = smem;                                   // [stages][TT][S]
    float* sm_c = sm_b + kWideStages * TT * S;            // [stages][TT][S]
    float* sm_d = sm_c + kWideStages * TT * S;            // [stages][TT][DP]
    float* sm_x = sm_d + kWideStages * TT * DP;           // [stages][TT][DP]
    float* sm_y = sm_x + kWideStages * TT * DP;           // [2][TT][DP]
    float4* sm_dw = reinterpret_cast<float4*>(sm_y + 2 * TT * DP);        // [2][TT][WP]
    float* sm_p = reinterpret_cast<float*>(sm_dw + 2 * WP * TT);          // exact: [WARPS][32][S + 1]; fast: [WARPS][TT][36]

    const int tid = threadIdx.x, wid = tid >> 5, lane_id = tid & 31;
    const int jl = lane_id / CPW, cw = lane_id % CPW;
    const int c = wid * CPW + cw;
    const int ncb = (p.d + CH - 1) / CH;
    const unsigned cta = ssm_cta(p.ragged);
    const int lane = cta / ncb;
    const int i0 = (cta % ncb) * CH;
    const int i = i0 + c;
    const bool valid = i < p.d;
    const size_t row0 = p.offsets ? p.offsets[lane] : 0;
    const int len = p.lengths ? (int)p.lengths[lane] : (int)p.rows;
    if (len <= 0) return;
    const int d = p.d;
    const size_t ds = (size_t)d * S;
    const size_t ldd = p.ld_delta ? p.ld_delta : (size_t)d;
    const size_t ldbc = p.ld_bc ? p.ld_bc : (size_t)S;
    float* carry = p.carry ? p.carry + (size_t)(p.lane_slots ? p.lane_slots[lane] : lane) * (p.carry_stride ? p.carry_stride : ds) : nullptr;
    const size_t so = (size_t)i * S + V * jl;
    float A[SPL], h[SPL];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        vec a{}, hv{};
        if (valid) a = __ldg(reinterpret_cast<const vec*>(p.rates + so + q * V * LPC));
        if (valid && carry) hv = *reinterpret_cast<const vec*>(carry + so + q * V * LPC);
#pragma unroll
        for (int v = 0; v < V; ++v) A[q * V + v] = reinterpret_cast<const float*>(&a)[v], h[q * V + v] = reinterpret_cast<const float*>(&hv)[v];
    }
    // an infinite rate (times log2 e, in the fast mode) would make a NaN of the padding's delta 0: the largest finite one does the
    // same for any other delta
    constexpr float kRateMax = EXACT ? FLT_MAX : FLT_MAX / 1.45f;
#pragma unroll
    for (int q = 0; q < SPL; ++q) A[q] = fabsf(A[q]) > kRateMax ? copysignf(kRateMax, A[q]) : A[q];
    auto put = [&](float* base, int t, int q, const float* v) {  // one piece of a tape row
        vec o;
#pragma unroll
        for (int u = 0; u < V; ++u) reinterpret_cast<float*>(&o)[u] = v[u];
        *reinterpret_cast<vec*>(base + (row0 + t) * ds + so + q * V * LPC) = o;
    };

    const int ntiles = (len + TT - 1) / TT;
    auto load_tile = [&](int k) {
        if (k < ntiles) {
            const int st = k % kWideStages, t0 = k * TT;
            for (int idx = tid; idx < TT * SQ; idx += THR) {
                const int tt = idx / SQ, j = idx % SQ * 4;
                const bool live = t0 + tt < len;
                const size_t o = (row0 + (live ? t0 + tt : 0)) * ldbc + j;
                cp_async16_zfill(sm_b + (st * TT + tt) * S + j, p.b_proj + o, live);
                cp_async16_zfill(sm_c + (st * TT + tt) * S + j, p.c_proj + o, live);
            }
            for (int idx = tid; idx < TT * CQ; idx += THR) {
                const int tt = idx / CQ, q = idx % CQ;
                const bool live = t0 + tt < len && i0 + q * 4 < d;
                const size_t row = row0 + (live ? t0 + tt : 0), col = live ? i0 + q * 4 : 0;
                cp_async16_zfill(sm_d + (st * TT + tt) * DP + q * 4, p.delta + row * ldd + col, live);
                cp_async16_zfill(sm_x + (st * TT + tt) * DP + q * 4, p.x_norm + row * d + col, live);
            }
        }
        cp_async_commit();
    };
    // y of a finished tile: 16-byte pieces of CH channels per token
    auto store_y = [&](int k) {
        const int t0 = k * TT, nt = min(TT, len - t0);
        for (int idx = tid; idx < nt * CQ; idx += THR) {
            const int tt = idx / CQ, q = idx % CQ;
            if (i0 + q * 4 < d) {
                const float4 v = *reinterpret_cast<const float4*>(sm_y + ((k & 1) * TT + tt) * DP + q * 4);
                const size_t o = (row0 + t0 + tt) * (size_t)d + i0 + q * 4;
                *reinterpret_cast<float4*>(p.y + o) = v;
                if (p.y_bf16) {
                    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
                    uint2 pk;
                    pk.x = *reinterpret_cast<unsigned*>(&lo), pk.y = *reinterpret_cast<unsigned*>(&hi);
                    *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.y_bf16) + o) = pk;
                }
            }
        }
    };
    // (delta, delta, delta * x, delta * x) of the group's channel for every token of a landed tile, spread over its lanes
    auto prepare = [&](int k) {
        const int st = k % kWideStages;
#pragma unroll
        for (int t = jl; t < TT; t += LPC) {
            const float dl = sm_d[(st * TT + t) * DP + c], xv = sm_x[(st * TT + t) * DP + c];
            sm_dw[((k & 1) * TT + t) * WP + c] = EXACT ? make_float4(dl, xv, 0.f, 0.f) : make_float4(dl, dl, dl * xv, dl * xv);
        }
    };
    load_tile(0);
    load_tile(1);
    if constexpr (EXACT) {
        for (int k = 0; k < ntiles; ++k) {
            cp_async_wait<1>();
            __syncthreads();  // tile k has landed; every warp is done with tile k - 1 and its y values are complete
            load_tile(k + 2);
            if (k > 0) store_y(k - 1);
            prepare(k);
            __syncwarp();
            const int st = k % kWideStages, t0 = k * TT;
#pragma unroll 1
            for (int s0 = 0; s0 < TT; s0 += LPC) {
                if (s0 > 0 && t0 + s0 >= len) break;
                const float4* dw = sm_dw + ((k & 1) * TT + s0) * WP + c;
                const int sj = (st * TT + s0) * S + V * jl;
#pragma unroll 8
                for (int tt = 0; tt < LPC; ++tt) {
                    const float4 w4 = dw[tt * WP];
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        const vec bv = *reinterpret_cast<const vec*>(sm_b + sj + tt * S + q * V * LPC);
                        const vec cv = *reinterpret_cast<const vec*>(sm_c + sj + tt * S + q * V * LPC);
                        float a[V], bb[V];
#pragma unroll
                        for (int v = 0; v < V; ++v) {
                            a[v] = exp_exact(__fmul_rn(w4.x, A[q * V + v]));
                            bb[v] = __fmul_rn(w4.x, reinterpret_cast<const float*>(&bv)[v]);
                            h[q * V + v] = __fadd_rn(__fmul_rn(a[v], h[q * V + v]), __fmul_rn(bb[v], w4.y));
                            sm_p[(wid * 32 + cw * LPC + tt) * (S + 1) + q * V * LPC + V * jl + v] =
                                __fmul_rn(h[q * V + v], reinterpret_cast<const float*>(&cv)[v]);
                        }
                        if (TAPE && valid && t0 + s0 + tt < len) {
                            if (p.states) put(p.states, t0 + s0 + tt, q, h + q * V);
                            if (p.bar_a) put(p.bar_a, t0 + s0 + tt, q, a);
                            if (p.bar_b) put(p.bar_b, t0 + s0 + tt, q, bb);
                        }
                    }
                }
                // lane (cw, jl) sums token jl of channel cw over the states in order
                __syncwarp();
                const float* pr = sm_p + (wid * 32 + cw * LPC + jl) * (S + 1);
                float y = 0.0f;
#pragma unroll 16
                for (int j = 0; j < S; ++j) y = __fadd_rn(y, pr[j]);
                sm_y[((k & 1) * TT + s0 + jl) * DP + c] = y;
                __syncwarp();
            }
        }
    } else {
        // The tokens form one stream of TB-token batches across tile borders: while batch b goes through the recurrence,
        // batch b + 1's exponentials are formed and batch b + 2's operands are on their way from shared memory. Two register
        // sets, used in turn, so that nothing is moved between them.
        constexpr int TB = 2, TG = 4 * TB;
        f32x2 A2[NP], h2[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q)
            A2[q] = pack2(A[2 * q] * 1.4426950408889634f, A[2 * q + 1] * 1.4426950408889634f), h2[q] = pack2(h[2 * q], h[2 * q + 1]);
        struct Ops { ulonglong2 w[TB]; f32x2 b[TB][NP]; };
        struct Exps { f32x2 e[TB][NP], u[TB][NP]; };
        struct Cs { f32x2 c[TB][NP]; };
        auto load_pairs = [&](const float* src, f32x2* dst) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                if constexpr (V == 4) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(src + q * V * LPC);
                    dst[2 * q] = v.x, dst[2 * q + 1] = v.y;
                } else {
                    dst[q] = *reinterpret_cast<const f32x2*>(src + q * V * LPC);
                }
            }
        };
        // sb / sd: this lane's first state of a group of TG tokens in sm_b (sm_c lies a constant away), its channel's row of sm_dw
        auto fetch = [&](const float* sb, const float4* sd, int b, Ops& o) {
#pragma unroll
            for (int u = 0; u < TB; ++u) {
                o.w[u] = *reinterpret_cast<const ulonglong2*>(sd + (b * TB + u) * WP);
                load_pairs(sb + (b * TB + u) * S, o.b[u]);
            }
        };
        auto fetch_c = [&](const float* sb, int b, Cs& o) {
#pragma unroll
            for (int u = 0; u < TB; ++u) load_pairs(sb + kWideStages * TT * S + (b * TB + u) * S, o.c[u]);
        };
        auto expand = [&](const Ops& o, Exps& x) {
            f32x2 arg[TB][NP];
#pragma unroll
            for (int u = 0; u < TB; ++u)
#pragma unroll
                for (int q = 0; q < NP; ++q) arg[u][q] = mul2(o.w[u].x, A2[q]);
#pragma unroll
            for (int u = 0; u < TB; ++u)
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    x.e[u][q] = exp2_approx2(arg[u][q]);
                    x.u[u][q] = mul2(o.w[u].y, o.b[u][q]);
                }
        };
        auto recur = [&](const float* sb, const float4* sd, float* part, int t0, int b, const Exps& x, const Cs& cc) {
            f32x2 hs[TB][NP], y2[TB];
#pragma unroll
            for (int u = 0; u < TB; ++u)
#pragma unroll
                for (int q = 0; q < NP; ++q) hs[u][q] = fma2(x.e[u][q], u == 0 ? h2[q] : hs[u - 1][q], x.u[u][q]);
#pragma unroll
            for (int q = 0; q < NP; ++q)
#pragma unroll
                for (int u = 0; u < TB; ++u) y2[u] = q == 0 ? mul2(hs[u][q], cc.c[u][q]) : fma2(hs[u][q], cc.c[u][q], y2[u]);
#pragma unroll
            for (int q = 0; q < NP; ++q) h2[q] = hs[TB - 1][q];
#pragma unroll
            for (int u = 0; u < TB; ++u) {
                float lo, hi;
                unpack2(y2[u], lo, hi);
                part[(b * TB + u) * 36] = lo + hi;
                const int t = t0 + b * TB + u;
                if (TAPE && valid && t < len) {
                    const float dl = sd[(b * TB + u) * WP].x;
                    f32x2 bp[NP];
                    load_pairs(sb + (b * TB + u) * S, bp);
                    float hv[SPL], av[SPL], bw[SPL];
#pragma unroll
                    for (int q = 0; q < NP; ++q) {
                        unpack2(hs[u][q], hv[2 * q], hv[2 * q + 1]);
                        unpack2(x.e[u][q], av[2 * q], av[2 * q + 1]);
                        unpack2(mul2(pack2(dl, dl), bp[q]), bw[2 * q], bw[2 * q + 1]);
                    }
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        if (p.states) put(p.states, t, q, hv + q * V);
                        if (p.bar_a) put(p.bar_a, t, q, av + q * V);
                        if (p.bar_b) put(p.bar_b, t, q, bw + q * V);
                    }
                }
            }
        };
        Ops oa, ob;
        Exps ea, eb;
        Cs ca, cb;
        for (int k = 0; k < ntiles; ++k) {
            cp_async_wait<0>();
            __syncthreads();  // tiles k and k + 1 have landed; every warp is done with tile k - 1 and its y values are complete
            load_tile(k + 2);
            if (k > 0) store_y(k - 1);
            if (k == 0) prepare(0);
            prepare(k + 1);
            __syncwarp();
            const float* sb = sm_b + (k % kWideStages) * TT * S + V * jl;
            const float4* sd = sm_dw + (k & 1) * WP * TT + c;
            const float* const sb_next = sm_b + ((k + 1) % kWideStages) * TT * S + V * jl;
            const float4* const sd_next = sm_dw + ((k + 1) & 1) * WP * TT + c;
            float* part = sm_p + wid * TT * 36 + cw * LPC + jl;
            if (k == 0) {
                fetch(sb, sd, 0, oa);
                fetch(sb, sd, 1, ob);
                fetch_c(sb, 0, ca);
                expand(oa, ea);
            }
#pragma unroll 1
            for (int g = 0; g < TT / TG; ++g) {
                const float* nb = g == TT / TG - 1 ? sb_next : sb + TG * S;
                const float4* nd = g == TT / TG - 1 ? sd_next : sd + TG * WP;
                const int tg = k * TT + g * TG;
                fetch(sb, sd, 2, oa);
                fetch_c(sb, 1, cb);
                recur(sb, sd, part, tg, 0, ea, ca);
                expand(ob, eb);
                fetch(sb, sd, 3, ob);
                fetch_c(sb, 2, ca);
                recur(sb, sd, part, tg, 1, eb, cb);
                expand(oa, ea);
                fetch(nb, nd, 0, oa);
                fetch_c(sb, 3, cb);
                recur(sb, sd, part, tg, 2, ea, ca);
                expand(ob, eb);
                fetch(nb, nd, 1, ob);
                fetch_c(nb, 0, ca);
                recur(sb, sd, part, tg, 3, eb, cb);
                expand(oa, ea);
                sb = nb, sd = nd, part += TG * 36;
            }
            // the tile's sums over the LPC lanes of a channel: lane (cw, jl) finishes tokens jl, jl + LPC, ... of channel cw
            __syncwarp();
#pragma unroll
            for (int t = jl; t < TT; t += LPC) {
                const float4* pr = reinterpret_cast<const float4*>(sm_p + (wid * TT + t) * 36 + cw * LPC);
                float4 acc = pr[0];
#pragma unroll
                for (int q = 1; q < LPC / 4; ++q) {
                    const float4 v = pr[q];
                    acc.x += v.x, acc.y += v.y, acc.z += v.z, acc.w += v.w;
                }
                sm_y[((k & 1) * TT + t) * DP + c] = (acc.x + acc.y) + (acc.z + acc.w);
            }
            __syncwarp();
        }
#pragma unroll
        for (int q = 0; q < NP; ++q) unpack2(h2[q], h[2 * q], h[2 * q + 1]);
    }
    cp_async_wait<0>();
    __syncthreads();
    store_y(ntiles - 1);
    if (carry && valid) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            vec o;
#pragma unroll
            for (int v = 0; v < V; ++v) reinterpret_cast<float*>(&o)[v] = h[q * V + v];
            *reinterpret_cast<vec*>(carry + so + q * V * LPC) = o;
        }
    }
}

// Decode step: every lane advances by one token, so the launch is one pass over the carries (2 * d * s * 4 bytes per
// lane in and out) and nothing else matters. A thread owns four consecutive states of one channel: rates, carry in and
// carry out are 16-byte accesses that a warp makes over a contiguous 512 bytes; y is finished by a shuffle tree over the
// TPC threads of the channel. Same arithmetic as the fast mode of the tiled kernel (ex2.approx, fused multiply-adds), or as the
// exact one: then the products h * C wait in shared memory for one thread per channel to add them in order.
template <int TPC, bool EXACT>
__global__ void __launch_bounds__(256) ssm_step_kernel(SsmParams p) {
    pdl_trigger();  // the next kernel in the stream may start its prologue now ...
    pdl_wait();     // ... and this one, if launched as a dependent, waits here for its own predecessor
    constexpr int CPB = 256 / TPC;  // channels per CTA
    __shared__ float prod[EXACT ? CPB * (4 * TPC + 1) : 1];
    const int tid = threadIdx.x;
    const int q = tid % TPC, c = tid / TPC;
    const int ncb = (p.d + CPB - 1) / CPB;
    const int lane = blockIdx.x / ncb;
    const int i = (blockIdx.x % ncb) * CPB + c;
    const int len = p.lengths ? (int)p.lengths[lane] : (int)p.rows;
    if (len <= 0) return;  // idle lane: carry and y untouched
    const size_t row = p.offsets ? p.offsets[lane] : 0;
    const int d = p.d, s = p.s;
    const size_t ds = (size_t)d * s;
    const size_t ldd = p.ld_delta ? p.ld_delta : (size_t)d;
    const size_t ldbc = p.ld_bc ? p.ld_bc : (size_t)s;
    float* carry = p.carry ? p.carry + (size_t)(p.lane_slots ? p.lane_slots[lane] : lane) * (p.carry_stride ? p.carry_stride : ds)
                           : nullptr;
    const bool live = i < d && q * 4 < s;
    float yp = 0.0f;
    if (live) {
        const size_t so = (size_t)i * s + q * 4;
        const float4 a4 = __ldg(reinterpret_cast<const float4*>(p.rates + so));
        const float4 h4 = carry ? *reinterpret_cast<const float4*>(carry + so) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 b4 = __ldg(reinterpret_cast<const float4*>(p.b_proj + row * ldbc + q * 4));
        const float4 c4 = __ldg(reinterpret_cast<const float4*>(p.c_proj + row * ldbc + q * 4));
        const float dl = __ldg(p.delta + row * ldd + i);
        const float w = dl * __ldg(p.x_norm + row * d + i);
        float4 h;
        if constexpr (EXACT) {
            const float xv = __ldg(p.x_norm + row * d + i);
            h.x = __fadd_rn(__fmul_rn(exp_exact(__fmul_rn(dl, a4.x)), h4.x), __fmul_rn(__fmul_rn(dl, b4.x), xv));
            h.y = __fadd_rn(__fmul_rn(exp_exact(__fmul_rn(dl, a4.y)), h4.y), __fmul_rn(__fmul_rn(dl, b4.y), xv));
            h.z = __fadd_rn(__fmul_rn(exp_exact(__fmul_rn(dl, a4.z)), h4.z), __fmul_rn(__fmul_rn(dl, b4.z), xv));
            h.w = __fadd_rn(__fmul_rn(exp_exact(__fmul_rn(dl, a4.w)), h4.w), __fmul_rn(__fmul_rn(dl, b4.w), xv));
            float* pr = prod + c * (4 * TPC + 1) + q * 4;
            pr[0] = __fmul_rn(h.x, c4.x), pr[1] = __fmul_rn(h.y, c4.y), pr[2] = __fmul_rn(h.z, c4.z), pr[3] = __fmul_rn(h.w, c4.w);
        } else {
            const float k = dl * 1.4426950408889634f;
            h.x = fmaf(ex2_approx(k * a4.x), h4.x, w * b4.x);
            h.y = fmaf(ex2_approx(k * a4.y), h4.y, w * b4.y);
            h.z = fmaf(ex2_approx(k * a4.z), h4.z, w * b4.z);
            h.w = fmaf(ex2_approx(k * a4.w), h4.w, w * b4.w);
            yp = fmaf(h.x, c4.x, fmaf(h.y, c4.y, fmaf(h.z, c4.z, h.w * c4.w)));
        }
        if (carry) *reinterpret_cast<float4*>(carry + so) = h;
    }
    if constexpr (EXACT) {
        __syncthreads();
        if (q == 0 && i < d)
            for (int j = 0; j < s; ++j) yp = __fadd_rn(yp, prod[c * (4 * TPC + 1) + j]);
    } else {
#pragma unroll
        for (int m = 1; m < TPC; m <<= 1) yp += __shfl_xor_sync(0xffffffffu, yp, m);
    }
    if (q == 0 && i < d) {
        p.y[row * d + i] = yp;
        if (p.y_bf16) reinterpret_cast<__nv_bfloat16*>(p.y_bf16)[row * d + i] = __float2bfloat16_rn(yp);
    }
}

template <int TPC, bool EXACT>
int32_t launch_step(pssa_b200_ctx* ctx, const SsmParams& p) {
    constexpr int CPB = 256 / TPC;
    size_t blocks = (size_t)((p.d + CPB - 1) / CPB) * p.lanes;
    if (blocks > 0x7fffffffull)
        return fail(ctx, PSSA_B200_ERR_SHAPE, "B200 SSM grid (%zu, 1) exceeds grid limits; refusing launch", blocks);
    PSSA_CUDA(ctx, launch_dependent(ssm_step_kernel<TPC, EXACT>, dim3((unsigned)blocks), dim3(256), 0, ctx->stream, p));
    return after_launch(ctx, "ssm_step_kernel");
}

// Sum of delta over each lane's rows, per channel (the decay half of a time shard's affine map: the product of
// exp(delta_t * A) over the shard is exp(A * sum of delta)). One CTA = one lane x 32 channels; 8 row-strided partial sums
// per channel in f64, combined in a fixed order.
__global__ void __launch_bounds__(256) sum_delta_kernel(const float* __restrict__ delta, size_t ldd, const uint32_t* __restrict__ offsets,
                                                        const uint32_t* __restrict__ lengths, int d, float* __restrict__ out,
                                                        size_t out_stride) {
    __shared__ double part[8][32];
    const int lane = blockIdx.y;
    const int c = threadIdx.x & 31, tq = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + c;
    const size_t row0 = offsets[lane];
    const int len = (int)lengths[lane];
    double acc = 0.0;
    if (i < d)
        for (int t = tq; t < len; t += 8) acc += (double)__ldg(delta + (row0 + t) * ldd + i);
    part[tq][c] = acc;
    __syncthreads();
    if (tq == 0 && i < d) {
        double sum = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) sum += part[k][c];
        out[(size_t)lane * out_stride + i] = (float)sum;
    }
}

// One thread per (lane, channel, state): walks the shard maps of every rank and time chunk in time order. The records do not depend
// on h, so a batch of them is always on its way while the batch before goes through its dependent multiply-adds: what is left
// is a few trips to L2, where the map pass has just left the records (37 chunks of 768 x 64 states: 31 -> 12 us, of which about 5 are
// the launch; before, a division per record and loads that waited for the batch before them).
__global__ void __launch_bounds__(128) seqpar_fold_kernel(const float* __restrict__ gathered, size_t rec, int world, int rank,
                                                          int chunks, size_t rank_stride, const float* __restrict__ rates,
                                                          float* __restrict__ state, size_t state_stride,
                                                          const uint32_t* __restrict__ lane_slots, float* __restrict__ carry_in,
                                                          int d, int s) {
    pdl_trigger();
    pdl_wait();
    const size_t ds = (size_t)d * s;
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = blockIdx.y;
    if (e >= ds) return;
    const int i = (int)((unsigned)e / (unsigned)s);
    float* st = state + (size_t)(lane_slots ? lane_slots[lane] : lane) * state_stride;
    const float a = rates[e];
    float h = st[e];
    constexpr int U = 10;
    for (int k = 0; k < world; ++k) {
        const float* r = gathered + (size_t)k * rank_stride + (size_t)lane * chunks * rec;
        float* out = k == rank ? carry_in + (size_t)lane * chunks * ds + e : nullptr;
        float sum[U], add[U];
        auto request = [&](int left) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (u < left) sum[u] = __ldcg(r + i), add[u] = __ldcg(r + d + e), r += rec;
        };
        request(chunks);
        for (int c = 0; c < chunks; c += U) {
            float pk[U], ad[U];
#pragma unroll
            for (int u = 0; u < U; ++u) pk[u] = sum[u], ad[u] = add[u];
            request(chunks - c - U);
#pragma unroll
            for (int u = 0; u < U; ++u) pk[u] = u < chunks - c ? exp_exact(__fmul_rn(a, pk[u])) : 0.0f;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (u < chunks - c) {
                    if (out) *out = h, out += ds;
                    h = __fadd_rn(__fmul_rn(pk[u], h), ad[u]);
                }
        }
    }
    st[e] = h;
}

template <int ST, int G, bool EXACT, bool TAPE, int THR = kThreads, int CPT = 1, bool MAPS = false>
int32_t launch_cfg(pssa_b200_ctx* ctx, const SsmParams& p) {
    constexpr int kThreads = THR;
    constexpr int CH = kThreads / G * CPT;
    constexpr int SP = ST * G;
    constexpr int kTileTokens = kTileTokensFor<G>;
    size_t smem = (size_t)kStages * kTileTokens * (2 * CH + 2 * SP) * sizeof(float);
    auto kern = ssm_fused_kernel<ST, G, EXACT, TAPE, THR, CPT, MAPS>;
    static PerDeviceOnce attr_set;  // per instantiation and per device
    if (smem > 48 * 1024 && attr_set.need(ctx->device)) {
        PSSA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set.done(ctx->device);
    }
    int ncb = (p.d + CH - 1) / CH;
    size_t blocks = (size_t)ncb * p.lanes;
    if (blocks > 0x7fffffffull)
        return fail(ctx, PSSA_B200_ERR_SHAPE, "B200 SSM grid (%zu, 1) exceeds grid limits; refusing launch", blocks);
    static PerDeviceCount resident;
    SsmParams q = p;
    q.ragged = p.ragged ? ctx->sm_count : 0;
    // which tiles are small is a warp's verdict over its channels, whose number depends on the lanes: not for prompts of under 256
    // tokens, whose bits are the same in any batch
    q.small_args = p.tiled || p.max_len == 0 || p.max_len >= 256;
    PSSA_CUDA(ctx, launch_spread(resident, p.ragged ? 0 : 1, ctx->device, ctx->sm_count, kern, dim3((unsigned)blocks), dim3(kThreads), smem,
                                 ctx->stream, q));
    return after_launch(ctx, MAPS ? "ssm_fused_kernel[chunk maps]" : "ssm_fused_kernel");
}

template <int LPC, int SPL, int TT, bool EXACT, bool TAPE>
int32_t launch_wide_cfg(pssa_b200_ctx* ctx, const SsmParams& p) {
    constexpr int CH = kWideWarps * (32 / LPC);
    constexpr size_t smem = wide_smem_floats<LPC, SPL, TT, EXACT>() * sizeof(float);
    auto kern = ssm_wide_kernel<LPC, SPL, TT, EXACT, TAPE>;
    static PerDeviceOnce attr_set;
    if (smem > 48 * 1024 && attr_set.need(ctx->device)) {
        PSSA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set.done(ctx->device);
    }
    const size_t blocks = (size_t)((p.d + CH - 1) / CH) * p.lanes;
    if (blocks > 0x7fffffffull)
        return fail(ctx, PSSA_B200_ERR_SHAPE, "B200 SSM grid (%zu, 1) exceeds grid limits; refusing launch", blocks);
    static PerDeviceCount resident;
    SsmParams q = p;
    q.ragged = p.ragged ? ctx->sm_count : 0;
    PSSA_CUDA(ctx, launch_spread(resident, p.ragged ? 0 : 1, ctx->device, ctx->sm_count, kern, dim3((unsigned)blocks), dim3(kWideWarps * 32), smem,
                                 ctx->stream, q));
    return after_launch(ctx, "ssm_fused_kernel[few lanes]");
}
template <int LPC, int SPL, int TT>
int32_t launch_wide(pssa_b200_ctx* ctx, const SsmParams& p, bool exact) {
    const bool tape = p.states || p.bar_a || p.bar_b;
    if (exact) return tape ? launch_wide_cfg<LPC, SPL, 32, true, true>(ctx, p) : launch_wide_cfg<LPC, SPL, 32, true, false>(ctx, p);
    return tape ? launch_wide_cfg<LPC, SPL, TT, false, true>(ctx, p) : launch_wide_cfg<LPC, SPL, TT, false, false>(ctx, p);
}

// The tape outputs (states, bar_a, bar_b: the reference's training tape) cost d*s floats per token
// each; inference never asks for them, so they live in a separate instantiation.
template <int ST, int G, bool EXACT>
int32_t launch_one(pssa_b200_ctx* ctx, const SsmParams& p) {
    if (p.states || p.bar_a || p.bar_b) return launch_cfg<ST, G, EXACT, true>(ctx, p);
    return launch_cfg<ST, G, EXACT, false>(ctx, p);
}

// CTA shape by wave balance. Every CTA of a launch is resident at once and a warp's time per token is fixed by
// its exponentials (16 per lane and channel, 8 cycles each on its scheduler's XU pipe), so the launch lasts as
// long as the busiest scheduler: count, per shape, the channel-warps the fullest SM puts on one scheduler.
// 256 threads = 64 channels per CTA (4 CTAs per SM), 352 threads = 88 channels (2 per SM), 128 threads with two
// channels per thread = 64 channels (3 per SM). With d = 768 and 32 lanes: 384 CTAs put 3 x 8 warps on most SMs
// (6 per scheduler), 288 of 352 threads put 2 x 11 (6 on two schedulers, 5 on the others), 384 two-channel CTAs
// put 3 x 4 double warps (6). On a tie the two-channel shape wins: a token's B and C rows are loaded once
// for both channels (11.93 -> 11.67 ms for the 12 launches of the benchmark step).
struct TiledShape {
    int kind;  // 0 = 256 threads, 1 = 352, 2 = 128 with two channels per thread
    long long busiest;
};
TiledShape tiled_shape(const pssa_b200_ctx* ctx, int d, int lanes) {
    auto busiest = [&](int threads, int cpt, int cap) -> long long {
        const int ch = threads / 4 * cpt;
        const long long blocks = (long long)((d + ch - 1) / ch) * lanes;
        const long long per_sm = (blocks + ctx->sm_count - 1) / ctx->sm_count;
        if (per_sm > cap) return 1ll << 40;  // more than one wave: not considered
        return (per_sm * (threads / 32) + 3) / 4 * cpt;
    };
    const long long two = busiest(128, 2, 3), wide = busiest(352, 1, 2), plain = busiest(256, 1, 4);
    if (two <= wide && two <= plain) {
        const long long all = ((long long)d * lanes / 8 + 4 * ctx->sm_count - 1) / (4 * ctx->sm_count);  // several waves
        return {2, two < (1ll << 40) ? two : all};
    }
    if (wide < plain) return {1, wide};
    return {0, plain};
}

// shapes the few-lanes kernel takes: state pairs that fill 4 to 32 lanes, 16-byte rows and states
bool ssm_wide_ok(const SsmParams& p) {
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    return !p.tiled && (p.s == 16 || p.s == 32 || p.s == 64) && p.aligned && al16(p.rates) && al16(p.carry) && al16(p.states) &&
           al16(p.bar_a) && al16(p.bar_b) && p.carry_stride % 4 == 0;
}

}  // namespace

int32_t launch_seqpar_fold(pssa_b200_ctx* ctx, const float* gathered, size_t rec, int world, int rank, int chunks, int lanes,
                           size_t rank_stride, const float* rates, float* state, size_t state_stride, const uint32_t* lane_slots,
                           float* carry_in, int d, int s) {
    const size_t ds = (size_t)d * s;
    dim3 grid((unsigned)((ds + 127) / 128), (unsigned)lanes);
    if (lanes < 1 || lanes > 65535) return fail(ctx, PSSA_B200_ERR_SHAPE, "chunk fold: %d lanes outside 1..65535", lanes);
    PSSA_CUDA(ctx, launch_dependent(seqpar_fold_kernel, grid, dim3(128), 0, ctx->stream, gathered, rec, world, rank, chunks, rank_stride, rates, state,
                                    state_stride, lane_slots, carry_in, d, s));
    return after_launch(ctx, "seqpar_fold_kernel");
}

size_t ssm_time_chunks(const pssa_b200_ctx* ctx, const SsmParams& p, bool exact) {
    const size_t longest = (size_t)p.max_len, ctas = (size_t)p.lanes * ((p.d + 63) / 64), schedulers = 4 * (size_t)ctx->sm_count;
    // Two passes pay every exponential twice. Where the few-lanes kernel applies they are the faster way only for a long
    // sequence that leaves it at few channels a scheduler.
    if (ssm_wide_ok(p)) {
        if (exact || p.s < 64) {
            if (!exact || longest < 4096 || 2 * p.rows * (size_t)p.d > 3 * longest * schedulers) return 1;
        } else {
            // CTAs of 64 channels, three to an SM. Us per pass of the 12-block model (d 768), few lanes against this: 1 lane of 512
            // tokens 1231 and 1339, 1024 1508 -> 1476, 2048 2210 -> 1961, 8192 6246 -> 4288; 2 lanes of 2048 2825 and 2842, 4096
            // 4789 -> 4364; 3 lanes of 8192 9968 and 10726. One block of d 192: 1 lane of 1024 105 -> 103, 4096 213 -> 129, 4 lanes 300 -> 226,
            // 8 lanes 418 -> 378.
            const size_t n = std::min<size_t>({(size_t)kMaxTimeChunks, 3 * (size_t)ctx->sm_count / std::max<size_t>(1, ctas), longest / 64});
            const size_t channels = (size_t)p.lanes * p.d;
            return channels <= 3 * schedulers && longest >= (2 * channels <= 3 * schedulers ? 1024u : 2560u) ? n : 1;
        }
    }
    if (ctas > (size_t)ctx->sm_count) return 1;
    return std::min({(size_t)16, std::max<size_t>(1, schedulers / ctas), std::max<size_t>(1, longest / 128)});
}

bool ssm_writes_maps(const SsmParams& p, bool exact) {
    return p.sum_delta && !exact && p.s > 32 && p.s <= 64 && p.aligned && p.offsets && p.lengths && (reinterpret_cast<uintptr_t>(p.rates) & 15) == 0 &&
           (reinterpret_cast<uintptr_t>(p.sum_delta) & 15) == 0 && p.sum_delta_stride % 4 == 0 && p.carry == p.sum_delta + p.d &&
           p.carry_stride == p.sum_delta_stride;
}

int32_t launch_ssm_fused(pssa_b200_ctx* ctx, const SsmParams& p, bool exact) {
    const int s = p.s;
    if (ssm_writes_maps(p, exact)) return launch_cfg<16, 4, false, false, 128, 2, true>(ctx, p);
    if (p.sum_delta) {
        if (!p.offsets || !p.lengths) return fail(ctx, PSSA_B200_ERR_INVALID_ARGUMENT, "B200 SSM: sum_delta needs lane offsets and lengths");
        if (p.lanes > 65535) return fail(ctx, PSSA_B200_ERR_SHAPE, "B200 SSM: sum_delta supports at most 65535 lanes; refusing launch");
        dim3 grid((unsigned)((p.d + 31) / 32), (unsigned)p.lanes);
        sum_delta_kernel<<<grid, 256, 0, ctx->stream>>>(p.delta, p.ld_delta ? p.ld_delta : (size_t)p.d, p.offsets, p.lengths, p.d,
                                                       p.sum_delta, p.sum_delta_stride);
        int32_t rc = after_launch(ctx, "sum_delta_kernel");
        if (rc != PSSA_B200_OK) return rc;
    }
    const bool tape = p.states || p.bar_a || p.bar_b;
    if (p.single_token && !tape && (!exact || s <= 64) && p.aligned && s <= 128 && (reinterpret_cast<uintptr_t>(p.rates) & 15) == 0 &&
        (reinterpret_cast<uintptr_t>(p.carry) & 15) == 0 && ((p.carry_stride ? p.carry_stride : (size_t)p.d * s) & 3) == 0) {
        // (above 64 states the exact mode sums y over shuffled groups: the tiled kernel's order stays)
        if (s <= 16) return exact ? launch_step<4, true>(ctx, p) : launch_step<4, false>(ctx, p);
        if (s <= 32) return exact ? launch_step<8, true>(ctx, p) : launch_step<8, false>(ctx, p);
        if (s <= 64) return exact ? launch_step<16, true>(ctx, p) : launch_step<16, false>(ctx, p);
        return launch_step<32, false>(ctx, p);
    }
    if (ssm_wide_ok(p)) {
        // Channels in flight: lanes counted by their share of the longest one. With 64 states, up to one channel per scheduler
        // takes 32 lanes a channel, above that 16; 32-token tiles while two CTAs an SM hold everything, 16-token ones
        // (half the shared memory) beyond. With 64 states a full machine is the tiled kernel's: us per 1024 tokens at d = 768,
        // tiled against this one: 1 lane 214 -> 52, 4 lanes 214 -> 91, 8 lanes 214 -> 171, 13 lanes 275 -> 237, but 24 lanes
        // 344 and 402: the two lines below are fits of both. With 32 and 16 states this one is ahead at every size
        // (384 x 32: 1 lane 226 -> 40, 64 lanes 369 -> 336; 192 x 16: 106 -> 40, 137 -> 104), and in the exact mode
        // (64 states, 1 lane 1600 -> 107, 32 lanes 1742 -> 1604). The tape's stores decide where it is asked for: whole lines
        // here, 4-byte pieces there. The lane splits sum y in different orders, so for calls of under 256 tokens a lane
        // (from there on time chunks depend on the lanes too) the split follows the shape alone and a stream sees the same bits
        // alone and in a batch; the exact mode's order is always the same.
        const size_t longest = p.max_len ? (size_t)p.max_len : (p.lengths ? 1 : p.rows);
        // (never more than there are: `rows` may count rows of no lane)
        const int lanes = (int)std::max<size_t>(1, p.max_len || !p.lengths ? std::min<size_t>(p.rows / std::max<size_t>(1, longest), (size_t)p.lanes) : (size_t)p.lanes);
        const size_t channels = (size_t)lanes * p.d, schedulers = 4 * (size_t)ctx->sm_count;
        const bool by_shape = !exact && longest < 256;
        if (s == 16) return channels <= 4 * schedulers && !by_shape ? launch_wide<8, 2, 32>(ctx, p, exact) : launch_wide<4, 4, 16>(ctx, p, exact);
        if (s == 32) return channels <= 2 * schedulers && !by_shape ? launch_wide<16, 2, 32>(ctx, p, exact) : launch_wide<8, 4, 32>(ctx, p, exact);
        if (channels <= (exact ? 2 : 1) * schedulers && !by_shape) return launch_wide<32, 2, 32>(ctx, p, exact);
        // (resident CTAs count every lane, however short)
        if (channels <= 4 * schedulers && (size_t)p.lanes * p.d <= 4 * schedulers) return launch_wide<16, 4, 32>(ctx, p, exact);
        // (five CTAs of the 16 x 4 split fit an SM: a sixth would run behind them. Four channels a warp then, 8 x 8, three CTAs to an SM. Us
        // a launch of 1024 tokens, inputs from HBM: 8 and 9 lanes of d 768 185 -> 169, 31 of d 192 182 -> 167, 16 and 18 of d 384 184 -> 168, 4 of
        // d 1536 183 -> 166, 6 of d 1024 182 -> 167, 62 and 74 of d 96 183 -> 166, 24 and 27 of d 256 183 -> 166; 300 tokens 68 to 71 -> 63 to 65. Below
        // and above it loses at each of these widths: 7 lanes of d 768 155 and 168, 10 lanes 202 and 233)
        const size_t ctas = channels / 8, sms = (size_t)ctx->sm_count;
        if (!exact && !tape && !by_shape && !p.ragged && ctas > 5 * sms && ctas <= 6 * sms) return launch_wide<8, 8, 16>(ctx, p, exact);
        const double wide_us = 13.8 * (double)channels / (double)schedulers;
        const double tiled_us = 60.0 + 64.5 * (double)tiled_shape(ctx, p.d, lanes).busiest;
        if (exact || tape || by_shape || wide_us < tiled_us) return launch_wide<16, 4, 16>(ctx, p, exact);
    }
    if (exact) {
        if (s <= 4) return launch_one<4, 1, true>(ctx, p);
        if (s <= 16) return launch_one<16, 1, true>(ctx, p);
        if (s <= 64) return launch_one<64, 1, true>(ctx, p);
        if (s <= 128) return launch_one<16, 8, true>(ctx, p);
        if (s <= 512) return launch_one<16, 32, true>(ctx, p);
    } else {
        if (s <= 4) return launch_one<4, 1, false>(ctx, p);
        if (s <= 8) return launch_one<4, 2, false>(ctx, p);
        if (s <= 16) return launch_one<4, 4, false>(ctx, p);
        if (s <= 32) return launch_one<16, 2, false>(ctx, p);
        if (s <= 64) {
            if (!tape) {
                const TiledShape t = tiled_shape(ctx, p.d, p.lanes);
                if (t.kind == 2) return launch_cfg<16, 4, false, false, 128, 2>(ctx, p);
                if (t.kind == 1) return launch_cfg<16, 4, false, false, 352>(ctx, p);
            }
            return launch_one<16, 4, false>(ctx, p);
        }
        if (s <= 128) return launch_one<16, 8, false>(ctx, p);
        if (s <= 256) return launch_one<16, 16, false>(ctx, p);
        if (s <= 512) return launch_one<16, 32, false>(ctx, p);
    }
    return fail(ctx, PSSA_B200_ERR_UNSUPPORTED, "B200 SSM: state width %d exceeds 512; refusing launch", s);
}

}  // namespace pssa
