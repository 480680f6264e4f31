// One decode step -- every lane advances by one token -- through all blocks and the vocabulary head in ONE launch.
//
// The block schedule of model_forward.cu is eight launches per block; with one row per stream each of them is a chain of
// launch, descriptor, pipeline-fill and drain latencies of about 11 us around a microsecond of work (98 launches, 0.84 ms per
// token of the 12-block model whose weights stream in 23 us). Here one CTA per SM stays for the whole step and the stages
// of a block are separated by grid barriers (a cooperative launch, every wait bounded):
//
//   1  x = RMSNorm(features), formed while it is loaded; delta | B | C | q_x | gate | adapter = epilogue(Wcat x)
//   2  SSM step on the carries (8 channels of a row per warp); the query's y part leaves as one partial per 8 channels,
//      so the query needs no product stage of its own
//   3  query = q_x + partials, projection into the ball, distances, softmax: a CTA per row
//   4  z' = gate * (VP w) + y / sqrt(s)          5  h = silu(W1 [z'; act])          6  features += scale * (W2 [h; act] + z')
//
// The products are m16n8k16 bf16 mma.sync, weights as the 16-row operand: at these sizes a product is the latency of its loads,
// not tensor throughput, and the tcgen05 path's fixed costs (descriptors, TMEM, an elected issuer) are what this kernel is
// there to avoid. With the 16 k of an mma permuted so that lane t of a quad owns k = 4t .. 4t + 3, every fragment is an 8-byte
// load of row-major memory. (An mma rounds once whatever the order of its 16 products, and as tcgen05.mma does: compared bit by
// bit, operands of one size and spread over 2^24. 16-byte loads, a k16 half in the lower and one in the upper 8 bytes, were 3 to
// 6 % faster up to 16 rows, but those are other sets of 16 than a tcgen05.mma's; exchanged by shuffles they were 10 % slower.)
//
// A stream's bits must not depend on how many others step with it, so every sum has one order for all row counts: K is cut
// into eight segments, each accumulated by one chain of mma, the segments added as ((s0+s1)+s2)+s3 + ((s4+s5)+s6)+s7. Here
// the eight warps of a CTA take a segment each of one 16-column tile, whose weights were requested before the barrier; above 32
// rows (step_schedule.cu) a segment is a TMEM accumulator.
#include <algorithm>
#include <cmath>

#include "step_stages.cuh"

namespace pssa {
namespace {

using namespace step;

constexpr int kMaxSegKb = 8;         // 32-wide k steps of a segment whose weights are requested ahead: K <= 2048
// Rows up to which one kernel is the faster way; step_schedule.cu above, with the same bits. Us per step, this and that one, at
// 32 rows: 1 block of d 192 41 and 58, 4 of d 384 128 and 230, 12 of d 768 525 and 840. (With 64-row mma.sync tiles this kernel took
// 72, 254 and 1000 at 33 rows, 79, 278 and 1119 at 128; the launches 63, 250 and 949.)
constexpr int kOneKernelRows = 32;
constexpr int kPitch = 20;           // floats per row of a partial tile: the fragment stores of a warp hit 32 banks

struct StepArgs : StepCommon {
    unsigned long long* barrier;
    StepBlock block[kMaxDepth];
};

__device__ __forceinline__ void mma_bf16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the two k16 halves of a 32-wide step: lo / hi are the lane's two 8-byte pieces of weight rows g and g + 8, b of activation row g
__device__ __forceinline__ void mma_step(float (&d)[4], const uint4& lo, const uint4& hi, const uint4& b) {
    mma_bf16(d, lo.x, hi.x, lo.y, hi.y, b.x, b.y);
    mma_bf16(d, lo.z, hi.z, lo.w, hi.w, b.z, b.w);
}

// ---- grid barrier on one 64-bit arrival count that is never reset: a launch finds it between k and k + 1 times the grid size
// (no CTA passes the first barrier before all have read it), so barrier i of the launch is over at (k + i + 1) * grid. One
// word to arrive at and to poll: 2430 cycles (1.3 us), 2950 with a store to publish, of which 820 are the release. A CTA that waits too long records the expiry and no
// longer waits.
struct Barrier {
    unsigned long long* count;
    int* status;
    unsigned long long target;
    bool dead;
    __device__ __forceinline__ static unsigned long long look(const unsigned long long* p) {
        unsigned long long v;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
        return v;
    }
    __device__ __forceinline__ void init() {
        if (threadIdx.x == 0) target = look(count) / gridDim.x * gridDim.x;
        dead = false;
    }
    // arrive, then what does not depend on the other CTAs (the next stage's weights), then wait
    __device__ __forceinline__ void arrive() {
        __syncthreads();
        if (threadIdx.x == 0) {
            target += gridDim.x;
            asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(count) : "memory");
        }
    }
    __device__ __forceinline__ void wait() {
        if (threadIdx.x == 0) {
            unsigned polls = 0;
            while (!dead && look(count) < target)
                if (++polls > (1u << 20)) atomicExch(status, PSSA_B200_ERR_TIMEOUT), dead = true;
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
        }
        __syncthreads();
    }
};

// ---- activation rows as B fragments: get(row, k) is the lane's share of row's 32-wide step at k, k + 4t .. and k + 16 + 4t ..
struct RowsBf16 {  // row-major bf16
    const __nv_bfloat16* x;
    size_t ld;
    __device__ __forceinline__ uint4 get(int row, int k) const {
        const __nv_bfloat16* e = x + (size_t)row * ld + k + 4 * (threadIdx.x & 3);
        const uint2 a = ld_u2(e), b = ld_u2(e + 16);
        return make_uint4(a.x, a.y, b.x, b.y);
    }
};
struct RowsF32 {  // row-major fp32, rounded to bf16
    const float* x;
    size_t ld;
    __device__ __forceinline__ uint4 get(int row, int k) const {
        const float* e = x + (size_t)row * ld + k + 4 * (threadIdx.x & 3);
        const float4 a = ld_f4(e), b = ld_f4(e + 16);
        return make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
    }
};
struct RowsNorm {  // RMSNorm of the features, rounded to bf16; inv[row - row0] in shared memory
    Features f;
    const float *gamma, *beta, *inv;
    int row0;
    __device__ __forceinline__ uint4 get(int row, int k) const {
        k += 4 * (threadIdx.x & 3);
        const float* e = f.row(row) + k;
        const float4 a = ld_f4(e), b = ld_f4(e + 16);
        const float4 ga = __ldg(reinterpret_cast<const float4*>(gamma + k)), gb = __ldg(reinterpret_cast<const float4*>(gamma + k + 16));
        const float4 ta = __ldg(reinterpret_cast<const float4*>(beta + k)), tb = __ldg(reinterpret_cast<const float4*>(beta + k + 16));
        const float s = inv[row - row0];
        return make_uint4(pack_bf16(norm1(a.x, s, ga.x, ta.x), norm1(a.y, s, ga.y, ta.y)), pack_bf16(norm1(a.z, s, ga.z, ta.z), norm1(a.w, s, ga.w, ta.w)),
                          pack_bf16(norm1(b.x, s, gb.x, tb.x), norm1(b.y, s, gb.y, tb.y)), pack_bf16(norm1(b.z, s, gb.z, tb.z), norm1(b.w, s, gb.w, tb.w)));
    }
};

struct Weights {
    const __nv_bfloat16* w;  // [n, ld] row-major, the first k columns are multiplied
    size_t ld;
    int n, k;
};

// ---- one 16-column tile per CTA, a warp per segment of K
__device__ __forceinline__ uint4 weight_pieces(const __nv_bfloat16* w) {
    const uint2 a = __ldg(reinterpret_cast<const uint2*>(w)), b = __ldg(reinterpret_cast<const uint2*>(w + 16));
    return make_uint4(a.x, a.y, b.x, b.y);
}
struct Ahead {
    uint4 a[kMaxSegKb][2];
};
__device__ __forceinline__ void request(const Weights& w, int tile, Ahead& r) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    int first, count;
    segment(w.k, threadIdx.x >> 5, first, count);
    const __nv_bfloat16* lo = w.w + (size_t)min(tile * 16 + g, w.n - 1) * w.ld + first * 32 + 4 * t;
    const __nv_bfloat16* hi = w.w + (size_t)min(tile * 16 + g + 8, w.n - 1) * w.ld + first * 32 + 4 * t;
#pragma unroll
    for (int kb = 0; kb < kMaxSegKb; ++kb)
        if (kb < count) {
            r.a[kb][0] = weight_pieces(lo + kb * 32);
            r.a[kb][1] = weight_pieces(hi + kb * 32);
        }
}
// epi(col, row, value): called once per output, sixteen columns of a row by neighbouring threads
template <int NT, class X, class Epi>
__device__ __forceinline__ void small_product(const Weights& w, const X& x, int rows, Ahead& ahead, float* part, Epi&& epi) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int tiles = (w.n + 15) / 16;
    int first, count;
    segment(w.k, warp, first, count);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.0f;
#pragma unroll
        for (int kb = 0; kb < kMaxSegKb; ++kb)
            if (kb < count) {
                uint4 b[NT];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) b[nt] = x.get(min(nt * 8 + g, rows - 1), (first + kb) * 32);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) mma_step(acc[nt], ahead.a[kb][0], ahead.a[kb][1], b[nt]);
            }
        if (tile + (int)gridDim.x < tiles) request(w, tile + gridDim.x, ahead);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            float* p0 = part + (warp * NT * 8 + nt * 8 + 2 * t) * kPitch + g;
            p0[0] = acc[nt][0], p0[kPitch] = acc[nt][1], p0[8] = acc[nt][2], p0[kPitch + 8] = acc[nt][3];
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < NT * 128; idx += kThreads) {
            const int row = idx >> 4, c = idx & 15;
            const float* p = part + row * kPitch + c;
            constexpr int S = NT * 8 * kPitch;
            const float v = (((p[0] + p[S]) + p[2 * S]) + p[3 * S]) + (((p[4 * S] + p[5 * S]) + p[6 * S]) + p[7 * S]);
            epi(tile * 16 + c, row, v);
        }
        __syncthreads();
    }
}

// 1 / rms of rows [r0, r0 + n) into inv_s, and into memory for the SSM stage
__device__ __forceinline__ void row_scales(const StepArgs& a, const Features& f, int r0, int n, float* inv_s, bool publish) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tiles = a.d / 16;
    for (int r = warp; r < n; r += kWarps) {
        float sum = 0.0f;
        if (f.ids) {
            const float* e = f.row(r0 + r);
            for (int i = lane * 4; i < a.d; i += 128) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(e + i));
                sum = fmaf(v.x, v.x, sum), sum = fmaf(v.y, v.y, sum), sum = fmaf(v.z, v.z, sum), sum = fmaf(v.w, v.w, sum);
            }
        } else {
            for (int i = lane; i < tiles; i += 32) sum += ld_f(a.ssq + (size_t)(r0 + r) * tiles + i);
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
        if (lane == 0) {
            const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)a.d), 1e-5f)));
            inv_s[r] = inv;
            if (publish) a.inv[r0 + r] = inv;
        }
    }
    __syncthreads();
}

// the next block's small vectors, on their way to L2 while this block is at work (its weights are asked for a stage ahead)
__device__ __forceinline__ void prefetch_vectors(const StepArgs& a, int l) {
    if (l >= a.depth || blockIdx.x != gridDim.x - 1) return;
    const StepBlock& b = a.block[l];
    for (int i = threadIdx.x * 32; i < a.d; i += kThreads * 32) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(b.gamma + i));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(b.beta + i));
    }
    for (int i = threadIdx.x * 32; i < a.cap; i += kThreads * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(b.norm_sq + i));
}

// NT 8-row tiles of rows: the stages are inlined, because the weights and carries that a stage asks for before
// the barrier in front of it stay in registers across it.
template <int NT, int NV, bool OWN>
__global__ void __launch_bounds__(kThreads, 1) step_kernel(const __grid_constant__ StepArgs a) {
    extern __shared__ __align__(128) float step_smem[];
    constexpr int kShared = NT * 64 * kPitch < 448 ? 448 : NT * 64 * kPitch;
    float *inv_s = step_smem, *sm = step_smem + 64;  // [64] row scales, then the stages' own
    float* keys_s = sm + kShared;
    Barrier bar{a.barrier, a.status, 0, false};
    bar.init();
    const int d = a.d, tiles = d / 16;
    Ahead ah;
    auto ahead = [&](const Weights& w) {
        if ((int)blockIdx.x * 16 < w.n) request(w, blockIdx.x, ah);
    };
    ahead({a.block[0].wcat, (size_t)d, a.nc, d});
    check_ids<OWN>(a);
    prefetch_vectors(a, 0);
    const float* in = nullptr;
    for (int l = 0; l < a.depth; ++l) {
        const StepBlock& b = a.block[l];
        float* out = in == a.feat_a ? a.feat_b : a.feat_a;
        const Features f{a.embed, l == 0 ? ids_of<OWN>(a) : nullptr, in, d, a.vocab};
        const Weights wcat{b.wcat, (size_t)d, a.nc, d}, vp{b.vp, (size_t)3 * a.cap, d, a.cap}, w1{b.w1, (size_t)d + 64, 2 * d, d + 64},
            w2{b.w2, (size_t)2 * d + 64, d, 2 * d + 64};
        row_scales(a, f, 0, a.rows, inv_s, blockIdx.x == 0);
        small_product<NT>(wcat, RowsNorm{f, b.gamma, b.beta, inv_s, 0}, a.rows, ah, sm, [&](int c, int r, float v) { store(PutXside{a}, c, r, v); });
        bar.arrive();
        SsmAhead<NV, 2> sa;
        ssm_request<OWN>(a, b, sa);
        const bool keys_here = request_keys(a, b, keys_s);
        bar.wait();
        ssm_stage<OWN>(a, f, sa, b.state);
        bar.arrive();
        ahead(vp);
        bar.wait();
        read_stage<1>(a, b, sm, keys_here ? keys_s : nullptr);
        bar.arrive();
        bar.wait();
        const RowsBf16 xw{a.w, (size_t)3 * a.cap}, xz{a.z, (size_t)d + 64}, xa{a.act, (size_t)2 * d + 64};
        small_product<NT>(vp, xw, a.rows, ah, sm, [&](int c, int r, float v) { store(PutGated{a}, c, r, v); });
        bar.arrive();
        ahead(w1);
        prefetch_vectors(a, l + 1);
        bar.wait();
        small_product<NT>(w1, xz, a.rows, ah, sm, [&](int c, int r, float v) { store(PutHidden{a}, c, r, v); });
        bar.arrive();
        ahead(w2);
        bar.wait();
        small_product<NT>(w2, xa, a.rows, ah, sm, [&](int c, int r, float v) {
            const float fv = new_feature(a, in, b.res_scale, c, r, v);
            if (r < a.rows) out[(size_t)r * d + c] = fv;
            const float q = squares16(fv);
            if (c % 16 == 0 && r < a.rows) a.ssq[(size_t)r * tiles + c / 16] = q;
        });
        in = out;
        bar.arrive();
        if (l + 1 < a.depth) ahead({a.block[l + 1].wcat, (size_t)d, a.nc, d});
        else if (a.logits) ahead({a.unembed, (size_t)d, (int)a.vocab, d});
        bar.wait();
    }
    if (!a.logits) return;
    small_product<NT>({a.unembed, (size_t)d, (int)a.vocab, d}, RowsF32{in, (size_t)d}, a.rows, ah, sm, [&](int c, int r, float v) { store(PutLogit{a}, c, r, v); });
}

template <int NT, int NV, bool OWN>
int32_t launch_one_kernel(pssa_b200_ctx* ctx, StepArgs& a) {
    constexpr size_t own = 64 * 4 + (size_t)(NT * 64 * kPitch < 448 ? 448 : NT * 64 * kPitch) * 4;
    auto kern = step_kernel<NT, NV, OWN>;
    static PerDeviceOnce attr;
    if (attr.need(ctx->device)) {
        PSSA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(own + kKeyQuads * 16)));
        attr.done(ctx->device);
    }
    void* args[] = {&a};
    // cooperative: the barriers need every CTA of the grid resident at once
    PSSA_CUDA(ctx, cudaLaunchCooperativeKernel((const void*)kern, dim3((unsigned)ctx->sm_count), dim3(kThreads), args,
                                               own + (size_t)std::min(a.k / 4 * a.cap, kKeyQuads) * 16, ctx->stream));
    return after_launch(ctx, "step_kernel");
}
template <int NV, bool OWN>
int32_t launch_rows(pssa_b200_ctx* ctx, StepArgs& a) {
    return a.rows <= 8 ? launch_one_kernel<1, NV, OWN>(ctx, a) : a.rows <= 16 ? launch_one_kernel<2, NV, OWN>(ctx, a) : launch_one_kernel<4, NV, OWN>(ctx, a);
}

// keys [cap, k] -> [k / 4][cap] quads: a warp's read of one quad of 32 slots is contiguous
__global__ void keys_by_quad_kernel(const float* __restrict__ keys, float* __restrict__ out, int cap, int k) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cap * (k / 4)) return;
    const int q = i / cap, s = i % cap;
    reinterpret_cast<float4*>(out)[i] = *reinterpret_cast<const float4*>(keys + (size_t)s * k + q * 4);
}

}  // namespace

int32_t launch_keys_by_quad(pssa_b200_ctx* ctx, const float* keys, float* out, int cap, int k) {
    const int n = cap * (k / 4);
    keys_by_quad_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(keys, out, cap, k);
    return after_launch(ctx, "keys_by_quad_kernel");
}

bool step_shape_ok(size_t depth, size_t d, size_t s, size_t k, size_t cap, size_t rank) {
    return depth <= kMaxDepth && d % 32 == 0 && 2 * d + 64 <= 8 * kMaxSegKb * 32 && (s == 16 || s == 32 || s == 64) && (k == 64 || k == 128) && cap % 64 == 0 &&
           cap <= 4 * kThreads && rank == 16;
}

static_assert(kOneKernelRows == kStepOwnRows, "a host call's rows travel with the one kernel's launch");

int32_t launch_decode_step(pssa_b200_ctx* ctx, const StepLaunch& p) {
    if (p.rows > kOneKernelRows) return launch_step_schedule(ctx, p);
    StepArgs a{};
    static_cast<StepCommon&>(a) = step_common(ctx, p);
    a.barrier = (unsigned long long*)p.barrier;
    for (size_t l = 0; l < p.depth; ++l) a.block[l] = step_block(p.blocks[l]);
    if (!p.ids) return p.s == 16 ? launch_rows<1, true>(ctx, a) : p.s == 32 ? launch_rows<2, true>(ctx, a) : launch_rows<4, true>(ctx, a);
    return p.s == 16 ? launch_rows<1, false>(ctx, a) : p.s == 32 ? launch_rows<2, false>(ctx, a) : launch_rows<4, false>(ctx, a);
}

}  // namespace pssa
