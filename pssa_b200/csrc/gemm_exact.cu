// Y[M,N] = X[M,K] * W[N,K]^T in fp32 with the reference's per-dot reduction order.
//
// Replaces `gemm_cpu_into` / `matvec` (src/backend.rs:832-871, src/pssa.rs:109-116): every output is one
// `dot_slice` (src/linalg.rs:184-298). On an AVX2/FMA host that is 4 accumulators x 8 lanes fed with
// fused multiply-adds over 32-element strides, extra 8-element blocks into accumulator 0, a fixed
// fold ((acc0+acc1)+(acc2+acc3), high half onto low half, two horizontal adds) and a scalar tail; for
// lengths 1..7 and 9..15 it is the portable 4-accumulator loop. A warp reproduces exactly that: lane l
// owns partial sum l of the 32, the fold is the same sequence of additions done with shuffles. This is
// the verification / exact path; the throughput path for the projections is the tensor-core GEMM.
#include "bounds.hpp"
#include "context.hpp"
#include "device_math.cuh"
#include "kernels.hpp"

namespace pssa {
namespace {

constexpr int RT = 4, CT = 4;  // outputs per warp: RT rows x CT columns

__global__ void __launch_bounds__(256) gemm_xwt_exact_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                             float* out, size_t M, int N, int K, size_t ldo, int epi,
                                                             float alpha) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t row0 = ((size_t)blockIdx.x * 4 + (warp >> 1)) * RT;
    const int col0 = (blockIdx.y * 2 + (warp & 1)) * CT;
    if (row0 >= M || col0 >= N) return;
    const float* xr[RT];
    const float* wc[CT];
#pragma unroll
    for (int r = 0; r < RT; ++r) xr[r] = x + (row0 + r < M ? row0 + r : M - 1) * (size_t)K;
#pragma unroll
    for (int c = 0; c < CT; ++c) wc[c] = w + (size_t)(col0 + c < N ? col0 + c : N - 1) * K;
    float acc[RT][CT];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int c = 0; c < CT; ++c) acc[r][c] = 0.0f;
    int i = 0;
    const unsigned full = 0xffffffffu;
    if (K == 8 || K >= 16) {  // linalg.rs:212-279
        for (; i + 32 <= K; i += 32) {
            float xa[RT], wb[CT];
#pragma unroll
            for (int r = 0; r < RT; ++r) xa[r] = __ldg(xr[r] + i + lane);
#pragma unroll
            for (int c = 0; c < CT; ++c) wb[c] = __ldg(wc[c] + i + lane);
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int c = 0; c < CT; ++c) acc[r][c] = fmaf(xa[r], wb[c], acc[r][c]);
        }
        for (; i + 8 <= K; i += 8) {  // remaining whole vectors go to accumulator 0 (lanes 0..7)
            if (lane < 8) {
#pragma unroll
                for (int r = 0; r < RT; ++r)
#pragma unroll
                    for (int c = 0; c < CT; ++c) acc[r][c] = fmaf(__ldg(xr[r] + i + lane), __ldg(wc[c] + i + lane), acc[r][c]);
            }
        }
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int c = 0; c < CT; ++c) {
                float v = acc[r][c];
                v = __fadd_rn(v, __shfl_down_sync(full, v, 8));   // acc0+acc1 (lanes 0-7), acc2+acc3 (lanes 16-23)
                v = __fadd_rn(v, __shfl_down_sync(full, v, 16));  // (acc0+acc1)+(acc2+acc3)
                v = __fadd_rn(v, __shfl_down_sync(full, v, 4));   // low 128 bits + high 128 bits
                v = __fadd_rn(v, __shfl_down_sync(full, v, 1));   // hadd: f0+f1, f2+f3
                v = __fadd_rn(v, __shfl_down_sync(full, v, 2));   // hadd: (f0+f1)+(f2+f3)
                acc[r][c] = v;
            }
    } else {  // linalg.rs:282-298
        for (; i + 4 <= K; i += 4) {
            if (lane < 4) {
#pragma unroll
                for (int r = 0; r < RT; ++r)
#pragma unroll
                    for (int c = 0; c < CT; ++c)
                        acc[r][c] = __fadd_rn(acc[r][c], __fmul_rn(__ldg(xr[r] + i + lane), __ldg(wc[c] + i + lane)));
            }
        }
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int c = 0; c < CT; ++c) {
                float v = acc[r][c];
                v = __fadd_rn(v, __shfl_down_sync(full, v, 1));  // acc0+acc1, acc2+acc3
                v = __fadd_rn(v, __shfl_down_sync(full, v, 2));  // (acc0+acc1)+(acc2+acc3)
                acc[r][c] = v;
            }
    }
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int c = 0; c < CT; ++c) {
                if (row0 + r >= M || col0 + c >= N) continue;
                float sum = acc[r][c];
                for (int t = i; t < K; ++t) sum = __fadd_rn(sum, __fmul_rn(xr[r][t], wc[c][t]));
                float* o = out + (row0 + r) * ldo + col0 + c;
                *o = apply_epilogue(epi, sum, alpha, epi == EPI_ADD_OUT ? *o : 0.0f);
            }
    }
}

// ---- tiled form for K == 8 or K >= 16. What bounded the kernel above was its fold (five shuffles for every output of a warp) and,
// with few rows, one round trip to HBM per 32 columns of W. Here
//   * the fold is a butterfly that halves a lane's outputs at every level: the additions pair the same sums as the reference's
//     (a + b and b + a are the same number), so RT * CT outputs cost RT * CT - 1 shuffles and end one to a lane;
//   * with few rows (AHEAD > 0) a warp requests AHEAD steps of its W rows at once and X is staged in shared memory;
//   * several products of one X (the six x-side projections) are one launch.
// Us, before -> now: 1 x 16384 x 768 39 -> 16. Used up to four rows, and where rows are not 16-byte aligned.
constexpr int kMaxParts = 6;
constexpr int kMaxStagedX = 200 * 1024;
struct ExactPart {
    const float* w;
    float* out;
    int n, tile0, epi;  // columns, first column tile
};
struct ExactParts {
    ExactPart p[kMaxParts];
    int count, tiles;
};
// The partial sums of NO outputs, one of 32 per lane each, to whole outputs: acc0+acc1 / acc2+acc3 (distance 8), their sum (16), low + high
// half (4), the two horizontal adds (1, 2). Returns the first output that this lane ends up with.
template <int NO, int LEVEL = 0, int SIZE>
__device__ __forceinline__ int fold_partials(float (&acc)[SIZE], int lane) {
    if constexpr (LEVEL == 5) {
        return 0;
    } else {
        constexpr int m = LEVEL == 0 ? 8 : LEVEL == 1 ? 16 : LEVEL == 2 ? 4 : LEVEL == 3 ? 1 : 2;
        if constexpr (NO > 1) {
            constexpr int half = NO / 2;
            const bool up = (lane & m) != 0;
#pragma unroll
            for (int o = 0; o < half; ++o) {
                const float send = up ? acc[o] : acc[o + half], keep = up ? acc[o + half] : acc[o];
                acc[o] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, m));
            }
            return (up ? half : 0) + fold_partials<half, LEVEL + 1>(acc, lane);
        } else {
            acc[0] = __fadd_rn(acc[0], __shfl_xor_sync(0xffffffffu, acc[0], m));
            return fold_partials<1, LEVEL + 1>(acc, lane);
        }
    }
}

// ---- many rows. The kernel below it reads every row of W once per eight rows of X, and a third of its instructions are addresses (ncu, 1000 x
// 1536 x 768: issue slots 66 % taken, fma pipe 37 %). Here a CTA's warps share a tile of operands that comes through a cp.async ring in
// shared memory, KB columns a stage, from pointers that only move on; the sums are the same ones in the same order. Small CTAs, three or
// four to an SM, so that one's first loads and fold run beside another's products. Us, W in HBM, before -> now: 8 x 768 x 768 8.3 -> 5.6
// (the launch), 16 x 768 x 1536 15.1 -> 6.8, 16 x 16384 x 768 35 -> 18, 300 x 1536 x 768 50 -> 28, 1000 x 1536 x 768 136 -> 86. What bounds
// it: a load for four multiply-adds (8 x 16 outputs a warp: half the loads, but two warps a scheduler do not hide them: 140 us;
// partials four to a lane with packed multiply-adds and 16-byte loads: 146).
constexpr int kRingStages = 4;
template <int RT, int CT, int WR, int WC, int KB>
__global__ void __launch_bounds__(32 * WR * WC) gemm_xwt_exact_ring_kernel(const float* __restrict__ x, const __grid_constant__ ExactParts parts, size_t M,
                                                                         int K, size_t ldo, float alpha) {
    extern __shared__ __align__(16) float ring[];  // [stages][BR + BC][KB]
    constexpr int NO = RT * CT, BR = RT * WR, BC = CT * WC, THR = 32 * WR * WC, Q = KB / 4;
    constexpr int RPP = THR / Q, NX = BR / RPP, NW = BC / RPP;  // rows a pass of all threads copies, passes for X and for W
    static_assert(BR % RPP == 0 && BC % RPP == 0, "whole passes");
    const int tid = threadIdx.x, lane = tid & 31, wr = (tid >> 5) / WC, wc = (tid >> 5) % WC;
    const int ct = (int)(blockIdx.x % parts.tiles);
    const size_t row0 = (size_t)(blockIdx.x / parts.tiles) * BR;
    int pi = 0;
#pragma unroll
    for (int i = 1; i < kMaxParts; ++i)
        if (i < parts.count && ct >= parts.p[i].tile0) pi = i;
    const ExactPart part = parts.p[pi];
    const int col0 = (ct - part.tile0) * BC;
    const int klen = K & ~31, blocks = (klen + KB - 1) / KB;
    const int cr = tid / Q, ck = tid % Q * 4;  // this thread's row of a pass and its columns
    const float *xsrc[NX], *wsrc[NW];  // rows past the end repeat the last one
#pragma unroll
    for (int j = 0; j < NX; ++j) xsrc[j] = x + (row0 + cr + j * RPP < M ? row0 + cr + j * RPP : M - 1) * (size_t)K + ck;
#pragma unroll
    for (int j = 0; j < NW; ++j) wsrc[j] = part.w + (size_t)min(col0 + cr + j * RPP, part.n - 1) * K + ck;
    const unsigned dst = (unsigned)__cvta_generic_to_shared(ring + cr * KB + ck);
    constexpr unsigned kStage = (BR + BC) * KB * 4;
    auto copy = [](unsigned to, const float* from) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from)); };
    auto load_x = [&](int b) {
        if (b * KB + ck < klen)
#pragma unroll
            for (int j = 0; j < NX; ++j) copy(dst + (b % kRingStages) * kStage + j * RPP * KB * 4, xsrc[j] + b * KB);
    };
    auto load_w = [&](int b) {
        if (b * KB + ck < klen)
#pragma unroll
            for (int j = 0; j < NW; ++j) copy(dst + (b % kRingStages) * kStage + (BR + j * RPP) * KB * 4, wsrc[j] + b * KB);
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    // W towards L2 before the wait (a prefetch reads nothing: the kernel before may have written W)
    for (int idx = tid; idx < BC * ((K + 31) / 32); idx += THR)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(part.w + (size_t)min(col0 + idx % BC, part.n - 1) * K + idx / BC * 32));
    pdl_trigger();
    pdl_wait();
#pragma unroll
    for (int b = 0; b < kRingStages - 1; ++b) load_x(b), load_w(b), commit();
    float acc[NO];
#pragma unroll
    for (int o = 0; o < NO; ++o) acc[o] = 0.0f;
    for (int b = 0; b < blocks; ++b) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kRingStages - 2) : "memory");
        __syncthreads();  // block b has landed, and everybody is done with the stage that is filled next
        load_x(b + kRingStages - 1), load_w(b + kRingStages - 1), commit();
        const float* xs = ring + (b % kRingStages) * (BR + BC) * KB + wr * RT * KB + lane;
        const float* ws = ring + (b % kRingStages) * (BR + BC) * KB + (BR + wc * CT) * KB + lane;
#pragma unroll
        for (int s = 0; s < KB / 32; ++s) {
            if (b * KB + s * 32 >= klen) break;
            float xa[RT], wb[CT];
#pragma unroll
            for (int r = 0; r < RT; ++r) xa[r] = xs[r * KB + s * 32];
#pragma unroll
            for (int c = 0; c < CT; ++c) wb[c] = ws[c * KB + s * 32];
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int c = 0; c < CT; ++c) acc[r * CT + c] = fmaf(xa[r], wb[c], acc[r * CT + c]);
        }
    }
    const size_t wrow = row0 + wr * RT;
    const int wcol = col0 + wc * CT;
    int i = klen;
    for (; i + 8 <= K; i += 8)  // remaining whole vectors go to accumulator 0 (lanes 0..7)
        if (lane < 8) {
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int c = 0; c < CT; ++c)
                    acc[r * CT + c] = fmaf(__ldg(x + (wrow + r < M ? wrow + r : M - 1) * (size_t)K + i + lane),
                                           __ldg(part.w + (size_t)min(wcol + c, part.n - 1) * K + i + lane), acc[r * CT + c]);
        }
    const int mine = fold_partials<NO>(acc, lane);
    constexpr int kDup = NO >= 32 ? 0 : NO == 16 ? 2 : 3;  // lanes that hold the same output
    if (NO < 32 && (lane & kDup)) return;
#pragma unroll
    for (int o = 0; o < (NO >= 32 ? NO / 32 : 1); ++o) {
        const int r = (mine + o) / CT, c = (mine + o) % CT;
        if (wrow + r >= M || wcol + c >= part.n) continue;
        float sum = acc[o];
        const float *xt = x + (wrow + r) * (size_t)K, *wt = part.w + (size_t)(wcol + c) * K;
        for (int t = i; t < K; ++t) sum = __fadd_rn(sum, __fmul_rn(xt[t], wt[t]));
        float* dst_o = part.out + (wrow + r) * ldo + wcol + c;
        *dst_o = apply_epilogue(part.epi, sum, alpha, part.epi == EPI_ADD_OUT ? *dst_o : 0.0f);
    }
}

template <int RT, int CT, int AHEAD>
__global__ void __launch_bounds__(256) gemm_xwt_exact_tiled_kernel(const float* __restrict__ x, const __grid_constant__ ExactParts parts, size_t M,
                                                                   int K, size_t ldo, float alpha) {
    extern __shared__ __align__(16) float sm_x[];  // AHEAD > 0: [RT][K], the only row tile
    constexpr int NO = RT * CT;
    const int lane = threadIdx.x & 31;
    const size_t row_tiles = (M + RT - 1) / RT, job0 = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5), jobs = row_tiles * parts.tiles;
    const size_t job = job0 < jobs ? job0 : jobs - 1;
    if (AHEAD == 0) {
        pdl_trigger();
        pdl_wait();
        if (job0 >= jobs) return;
    }
    const int ct = (int)(job % parts.tiles);
    const size_t row0 = job / parts.tiles * RT;
    int pi = 0;
#pragma unroll
    for (int i = 1; i < kMaxParts; ++i)
        if (i < parts.count && ct >= parts.p[i].tile0) pi = i;
    const ExactPart part = parts.p[pi];
    const int col0 = (ct - part.tile0) * CT;
    const float* xr[RT];
    const float* wc[CT];
#pragma unroll
    for (int r = 0; r < RT; ++r) xr[r] = x + (row0 + r < M ? row0 + r : M - 1) * (size_t)K + lane;
#pragma unroll
    for (int c = 0; c < CT; ++c) wc[c] = part.w + (size_t)min(col0 + c, part.n - 1) * K + lane;
    float acc[NO];
#pragma unroll
    for (int o = 0; o < NO; ++o) acc[o] = 0.0f;
    const int steps = K >> 5;
    if constexpr (AHEAD > 0) {
        // W towards L2 before the wait (a prefetch reads nothing), X whole into shared memory: one trip to memory each
#pragma unroll
        for (int c = 0; c < CT; ++c)
            for (int k = lane * 32; k < K; k += 1024) asm volatile("prefetch.global.L2 [%0];" ::"l"(wc[c] - lane + k));
        pdl_trigger();
        pdl_wait();
        if ((K & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
            const int q = K >> 2, rows = M < RT ? (int)M : RT;
            for (int r = 0; r < rows; ++r)
                for (int k = threadIdx.x; k < q; k += 256)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(sm_x + r * K + k * 4)), "l"(x + (size_t)r * K + k * 4));
            asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
        } else {
            for (int idx = threadIdx.x; idx < (int)(M < RT ? M : RT) * K; idx += 256) sm_x[idx] = x[idx];
        }
        __syncthreads();
        if (job0 >= jobs) return;
        for (int s0 = 0; s0 < steps; s0 += AHEAD) {
            float wb[AHEAD][CT];
#pragma unroll
            for (int s = 0; s < AHEAD; ++s)
#pragma unroll
                for (int c = 0; c < CT; ++c) wb[s][c] = s0 + s < steps ? __ldg(wc[c] + (s0 + s) * 32) : 0.0f;
#pragma unroll
            for (int s = 0; s < AHEAD; ++s)
                if (s0 + s < steps) {
                    float xa[RT];
#pragma unroll
                    for (int r = 0; r < RT; ++r) xa[r] = sm_x[(r < (int)M ? r : (int)M - 1) * K + (s0 + s) * 32 + lane];
#pragma unroll
                    for (int r = 0; r < RT; ++r)
#pragma unroll
                        for (int c = 0; c < CT; ++c) acc[r * CT + c] = fmaf(xa[r], wb[s][c], acc[r * CT + c]);
                }
        }
    } else {
#pragma unroll 2
        for (int s = 0; s < steps; ++s) {
            float xa[RT], wb[CT];
#pragma unroll
            for (int r = 0; r < RT; ++r) xa[r] = __ldg(xr[r] + s * 32);
#pragma unroll
            for (int c = 0; c < CT; ++c) wb[c] = __ldg(wc[c] + s * 32);
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int c = 0; c < CT; ++c) acc[r * CT + c] = fmaf(xa[r], wb[c], acc[r * CT + c]);
        }
    }
    int i = steps << 5;
    for (; i + 8 <= K; i += 8)  // remaining whole vectors go to accumulator 0 (lanes 0..7)
        if (lane < 8) {
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int c = 0; c < CT; ++c) acc[r * CT + c] = fmaf(__ldg(xr[r] + i), __ldg(wc[c] + i), acc[r * CT + c]);
        }
    const int mine = fold_partials<NO>(acc, lane);  // which output ends in this lane (its first, where a lane keeps several)
    constexpr int OWN = NO >= 32 ? NO / 32 : 1;
    // with fewer than 32 outputs the lanes that differ in the last levels hold the same one: one of them stores
    constexpr int kDup = NO >= 32 ? 0 : NO == 16 ? 2 : NO == 8 ? 3 : NO == 4 ? 7 : 31;
    if (NO < 32 && (lane & kDup)) return;
#pragma unroll
    for (int o = 0; o < OWN; ++o) {
        const int r = (mine + o) / CT, c = (mine + o) % CT;
        if (row0 + r >= M || col0 + c >= part.n) continue;
        float sum = acc[o];
        const float *xs = x + (row0 + r) * (size_t)K, *ws = part.w + (size_t)(col0 + c) * K;
        for (int t = i; t < K; ++t) sum = __fadd_rn(sum, __fmul_rn(xs[t], ws[t]));
        float* dst = part.out + (row0 + r) * ldo + col0 + c;
        *dst = apply_epilogue(part.epi, sum, alpha, part.epi == EPI_ADD_OUT ? *dst : 0.0f);
    }
}

template <int RT, int CT, int AHEAD>
int32_t launch_tiled(pssa_b200_ctx* ctx, const float* x, ExactParts& parts, size_t M, size_t K, size_t ldo, float alpha) {
    parts.tiles = 0;
    for (int i = 0; i < parts.count; ++i) parts.p[i].tile0 = parts.tiles, parts.tiles += (parts.p[i].n + CT - 1) / CT;
    const size_t jobs = (M + RT - 1) / RT * parts.tiles, blocks = (jobs + 7) / 8;
    if (blocks > 0x7fffffffull) return fail(ctx, PSSA_B200_ERR_SHAPE, "B200 GEMM grid (%zu, 1) exceeds grid limits; refusing launch", blocks);
    const size_t smem = AHEAD ? (size_t)RT * K * sizeof(float) : 0;
    static PerDeviceOnce attr_set;
    if (smem > 48 * 1024 && attr_set.need(ctx->device)) {
        PSSA_CUDA(ctx, cudaFuncSetAttribute(gemm_xwt_exact_tiled_kernel<RT, CT, AHEAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxStagedX));
        attr_set.done(ctx->device);
    }
    PSSA_CUDA(ctx, launch_dependent(gemm_xwt_exact_tiled_kernel<RT, CT, AHEAD>, dim3((unsigned)blocks), dim3(256), smem, ctx->stream, x, parts, M, (int)K, ldo, alpha));
    return after_launch(ctx, "gemm_xwt_exact_kernel");
}
template <int RT, int CT, int WR, int WC, int KB>
int32_t launch_ring(pssa_b200_ctx* ctx, const float* x, ExactParts& parts, size_t M, size_t K, size_t ldo, float alpha) {
    constexpr int BR = RT * WR, BC = CT * WC;
    parts.tiles = 0;
    for (int i = 0; i < parts.count; ++i) parts.p[i].tile0 = parts.tiles, parts.tiles += (parts.p[i].n + BC - 1) / BC;
    const size_t blocks = (M + BR - 1) / BR * parts.tiles;
    if (blocks > 0x7fffffffull) return fail(ctx, PSSA_B200_ERR_SHAPE, "B200 GEMM grid (%zu, 1) exceeds grid limits; refusing launch", blocks);
    constexpr size_t smem = (size_t)kRingStages * (BR + BC) * KB * sizeof(float);
    auto kern = gemm_xwt_exact_ring_kernel<RT, CT, WR, WC, KB>;
    static PerDeviceOnce attr_set;
    if (smem > 48 * 1024 && attr_set.need(ctx->device)) {
        PSSA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set.done(ctx->device);
    }
    // few rows: the early start's prefetch of W is worth more than an even spread (a scored step of 16 streams 977 us, 1119 spread); 300
    // rows, whose 64-wide query product is a CTA to every other SM: 3309 and 3139
    static PerDeviceCount resident;
    PSSA_CUDA(ctx, launch_spread(resident, M <= 128 ? 1 << 20 : 1, ctx->device, ctx->sm_count, kern, dim3((unsigned)blocks), dim3(32 * WR * WC),
                                 smem, ctx->stream, x, parts, M, (int)K, ldo, alpha));
    return after_launch(ctx, "gemm_xwt_exact_kernel");
}
int32_t launch_parts(pssa_b200_ctx* ctx, const float* x, ExactParts& parts, size_t M, size_t K, size_t ldo, float alpha) {
    // Up to four rows a warp takes all of them and two columns of W, so that W's rows are spread over the most warps (16384 columns, 4 rows:
    // 17.4 us; tiles of eight rows 16.3, but 8.7 to 9.5 for 1536 columns where this takes 5.5). Above, tiles of 8 rows x 16 columns where
    // 16 x 16 would be half empty (17 rows of K = 1536: 7.3 and 11.4 us).
    if (M <= 4 && 4 * K * 4 <= kMaxStagedX) return launch_tiled<4, 2, 24>(ctx, x, parts, M, K, ldo, alpha);
    bool vec = K % 4 == 0 && K >= 32 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    for (int i = 0; i < parts.count; ++i) vec = vec && (reinterpret_cast<uintptr_t>(parts.p[i].w) & 15) == 0;
    if (!vec) {
        // Rows that the ring cannot copy. Tiles of 8 x 8 load a word for four multiply-adds instead of 2.7, but hold twice the registers (16
        // warps to an SM) and leave more of a last wave empty; short sums hide that sooner. Us, 8 x 4 and 8 x 8: 1000 x 192 x 16 6.4 and
        // 5.7, 4096 x 768 x 16 79 and 64, 2048 x 1536 x 191 169 and 149, 1000 x 1536 x 767 175 and 167; under the line 300 x 768 x 191 15.3 and
        // 15.5, 300 x 592 x 767 24.4 and 26.8, 300 x 1536 x 767 57.1 and 57.6. Few rows need nothing of their own (16 x 16384 x 767 32; 40
        // with X staged in shared memory).
        size_t n = 0;
        for (int i = 0; i < parts.count; ++i) n += parts.p[i].n;
        const size_t wide = (M + 7) / 8 * ((n + 7) / 8);
        if (wide >= (K < 64 ? 20 : K < 256 ? 30 : 56) * (size_t)ctx->sm_count) return launch_tiled<8, 8, 0>(ctx, x, parts, M, K, ldo, alpha);
        return launch_tiled<8, 4, 0>(ctx, x, parts, M, K, ldo, alpha);
    }
    if (M <= 8 || (M > 16 && M <= 24)) return launch_ring<8, 4, 1, 4, 64>(ctx, x, parts, M, K, ldo, alpha);
    return launch_ring<8, 8, 2, 2, 128>(ctx, x, parts, M, K, ldo, alpha);
}

}  // namespace

int32_t launch_gemm_exact(pssa_b200_ctx* ctx, const float* x, const float* w, float* out, size_t M, size_t N, size_t K,
                          size_t ldo, int epi, float alpha) {
    if (K == 8 || K >= 16) {
        ExactParts parts{};
        parts.count = 1, parts.p[0] = {w, out, (int)N, 0, epi};
        return launch_parts(ctx, x, parts, M, K, ldo, alpha);
    }
    size_t bx = (M + 4 * RT - 1) / (4 * RT), by = (N + 2 * CT - 1) / (2 * CT);
    if (bx > 0x7fffffffull || by > 65535)
        return fail(ctx, PSSA_B200_ERR_SHAPE, "B200 GEMM grid (%zu, %zu) exceeds grid limits; refusing launch", bx, by);
    gemm_xwt_exact_kernel<<<dim3((unsigned)bx, (unsigned)by), 256, 0, ctx->stream>>>(x, w, out, M, (int)N, (int)K, ldo, epi,
                                                                                   alpha);
    return after_launch(ctx, "gemm_xwt_exact_kernel");
}

int32_t launch_gemm_exact_many(pssa_b200_ctx* ctx, const float* x, const ExactProduct* products, int count, size_t M, size_t K, size_t ldo) {
    if (count > kMaxParts || !(K == 8 || K >= 16)) {
        for (int i = 0; i < count; ++i) {
            const int32_t rc = launch_gemm_exact(ctx, x, products[i].w, products[i].out, M, products[i].n, K, ldo, products[i].epi, 1.0f);
            if (rc) return rc;
        }
        return PSSA_B200_OK;
    }
    ExactParts parts{};
    parts.count = count;
    for (int i = 0; i < count; ++i) parts.p[i] = {products[i].w, products[i].out, (int)products[i].n, 0, products[i].epi};
    return launch_parts(ctx, x, parts, M, K, ldo, 1.0f);
}

}  // namespace pssa
