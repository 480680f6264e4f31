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
// there to avoid. With the 32 k of a step permuted so that lane t of a quad owns k = 8t .. 8t + 7, every fragment is one
// 16-byte load of row-major memory.
//
// A stream's bits must not depend on how many others step with it, so every sum has one order for all row counts: K is cut
// into eight segments, each accumulated by one chain of mma, the segments added as ((s0+s1)+s2)+s3 + ((s4+s5)+s6)+s7. Few rows:
// the eight warps of a CTA take a segment each of one 16-column tile, whose weights were requested before the barrier. More:
// the warps share out 64-row tiles and walk the segments one after another.
#include <cuda_bf16.h>
#include <math_constants.h>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "context.hpp"
#include "device_math.cuh"
#include "kernels.hpp"

namespace pssa {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = 8;
constexpr int kMaxSegKb = 8;         // 32-wide k steps of a segment whose weights are requested ahead: K <= 2048
constexpr int kMaxDepth = 32;        // blocks whose pointers fit in the kernel's parameters
constexpr int kSmallRows = 32;       // rows up to which a warp takes a segment of K
constexpr int kStepRows = 128;       // rows up to which this kernel is the faster way: 12 blocks, d 768, us per step at 1 / 32 / 128 rows
                                     // 840 -> 260 / 960 -> 540 / 1060 -> 1090; at 256 the separate kernels' tensor-core products win (1130, 1840)
constexpr int kKeyQuads = 8192;      // the bank's keys are staged in shared memory (128 KB) up to here
constexpr int kTileBytes = 212 * 1024;
constexpr int kPitch = 20;           // floats per row of a partial tile: the fragment stores of a warp hit 32 banks

__device__ __forceinline__ void mma_bf16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the two k16 halves of a 32-wide step: lo / hi are the lane's 16 bytes of weight rows g and g + 8, b of activation row g
__device__ __forceinline__ void mma_step(float (&d)[4], const uint4& lo, const uint4& hi, const uint4& b) {
    mma_bf16(d, lo.x, hi.x, lo.y, hi.y, b.x, b.y);
    mma_bf16(d, lo.z, hi.z, lo.w, hi.w, b.z, b.w);
}
__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<unsigned*>(&v);
}
// data written by other CTAs of this launch: not through the non-coherent path
__device__ __forceinline__ uint4 ld_u4(const void* p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_f4(const float* p) {
    float4 v;
    asm volatile("ld.global.cg.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_f(const float* p) {
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float softplus_fast(float x) {  // the tensor-core epilogue's formula
    const float e = __expf(x), mid = __logf(1.0f + e), low = e * fmaf(-0.5f, e, 1.0f);
    return x > 20.0f ? x : (x < -4.0f ? low : mid);
}

// ---- grid barrier on one 64-bit arrival count that is never reset: a launch finds it between k and k + 1 times the grid size
// (no CTA passes the first barrier before all have read it), so barrier i of the launch is over at (k + i + 1) * grid. One
// word to arrive at and to poll: 2400 cycles, 900 of them the release. A CTA that waits too long records the expiry and no
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

struct StepBlock {
    const __nv_bfloat16 *wcat, *wqh, *vp, *w1, *w2;
    const float *rates, *gamma, *beta, *keys_t, *norm_sq;
    float* state;  // carry of stream 0 of this block
    float res_scale;
    int count;
};
struct StepArgs {
    int rows, depth, d, s, k, cap, nc, off_b, off_q, off_gate, off_act;
    unsigned vocab;
    float ssm_scale, head_scale, tau;
    const float* embed;
    const unsigned *ids, *slots;
    const __nv_bfloat16* unembed;
    size_t carry_stride;
    float *feat_a, *feat_b, *proj, *y, *qpart, *ssq, *inv, *logits;
    __nv_bfloat16 *x, *w, *z, *act;  // x: the normalised rows, at the end the features (many-rows kernel)
    unsigned long long* barrier;
    int* status;
    StepBlock block[kMaxDepth];
};

// ---- activation rows as B fragments: lane (g, t) of row g takes k = 8t .. 8t + 7 of a 32-wide step
struct RowsBf16 {  // row-major bf16
    const __nv_bfloat16* x;
    size_t ld;
    __device__ __forceinline__ uint4 get(int row, int k) const { return ld_u4(x + (size_t)row * ld + k); }
};
struct RowsF32 {  // row-major fp32, rounded to bf16
    const float* x;
    size_t ld;
    __device__ __forceinline__ uint4 get(int row, int k) const {
        const float4 a = ld_f4(x + (size_t)row * ld + k), b = ld_f4(x + (size_t)row * ld + k + 4);
        return make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
    }
};
// the features of a row: embedding row of its id (first block) or the previous block's output
struct Features {
    const float* embed;
    const unsigned* ids;  // null: feats
    const float* feats;
    int d;
    unsigned vocab;
    __device__ __forceinline__ const float* row(int r) const {
        if (!ids) return feats + (size_t)r * d;
        const unsigned id = ids[r];
        return embed + (size_t)(id < vocab ? id : 0) * d;
    }
};
__device__ __forceinline__ float norm1(float e, float inv, float g, float b) { return __fadd_rn(__fmul_rn(g, __fmul_rn(e, inv)), b); }
struct RowsNorm {  // RMSNorm of the features, rounded to bf16; inv[row - row0] in shared memory
    Features f;
    const float *gamma, *beta, *inv;
    int row0;
    __device__ __forceinline__ uint4 get(int row, int k) const {
        const float* e = f.row(row) + k;
        const float4 a = ld_f4(e), b = ld_f4(e + 4);
        const float4 ga = __ldg(reinterpret_cast<const float4*>(gamma + k)), gb = __ldg(reinterpret_cast<const float4*>(gamma + k + 4));
        const float4 ta = __ldg(reinterpret_cast<const float4*>(beta + k)), tb = __ldg(reinterpret_cast<const float4*>(beta + k + 4));
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
// segment s of K: its first 32-wide step and the number of them
__device__ __forceinline__ void segment(int k, int s, int& first, int& count) {
    const int nkb = k >> 5, base = nkb >> 3, rem = nkb & 7;
    first = s * base + min(s, rem), count = base + (s < rem ? 1 : 0);
}

// ---- few rows: one 16-column tile per CTA, a warp per segment of K
struct Ahead {
    uint4 a[kMaxSegKb][2];
};
__device__ __forceinline__ void request(const Weights& w, int tile, Ahead& r) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    int first, count;
    segment(w.k, threadIdx.x >> 5, first, count);
    const __nv_bfloat16* lo = w.w + (size_t)min(tile * 16 + g, w.n - 1) * w.ld + first * 32 + 8 * t;
    const __nv_bfloat16* hi = w.w + (size_t)min(tile * 16 + g + 8, w.n - 1) * w.ld + first * 32 + 8 * t;
#pragma unroll
    for (int kb = 0; kb < kMaxSegKb; ++kb)
        if (kb < count) {
            r.a[kb][0] = __ldg(reinterpret_cast<const uint4*>(lo + kb * 32));
            r.a[kb][1] = __ldg(reinterpret_cast<const uint4*>(hi + kb * 32));
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
                for (int nt = 0; nt < NT; ++nt) b[nt] = x.get(min(nt * 8 + g, rows - 1), (first + kb) * 32 + 8 * t);
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

// ---- more rows: tiles of 64 rows x (WC * MT * 16) columns, the warps WC x (8 / WC) over columns and rows. Both operands come into
// shared memory a segment of K at a time; the segments of a CTA's tiles form one stream, as much of it in flight as fits (a
// segment arrives from L2 in about a microsecond and is used up in a quarter of one), so a tile's first segments are on
// their way during the epilogue before it. A row pitch that is an odd multiple of 64 bytes keeps the 16-byte fragment reads
// conflict free.
__device__ __forceinline__ void cp16(char* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void wait_pending(int n) {  // at most n copy groups still in flight
    switch (n) {
        case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
        case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
        case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
        case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
        case 5: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
        case 6: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
        default: asm volatile("cp.async.wait_group 7;" ::: "memory"); break;
    }
}
template <int WC, int MT, class Epi>
__device__ __forceinline__ void large_product(const Weights& w, const RowsBf16& x, int rows, char* sm, Epi&& epi) {
    constexpr int WR = kWarps / WC, NT = 8 / WR, COLS = WC * MT * 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int wr = warp % WR, wc = warp / WR;
    const int ct = (w.n + COLS - 1) / COLS, rt = (rows + 63) / 64;
    const int pitch = (((w.k >> 5) + 7) / 8 | 1) * 64, buf = (64 + COLS) * pitch, nbuf = min(8, kTileBytes / buf);
    // a CTA's tiles lie one after another on the same rows as far as there are columns
    const int per = (ct * rt + gridDim.x - 1) / gridDim.x, task0 = blockIdx.x * per, tasks = min(ct * rt, task0 + per) - task0;
    if (tasks <= 0) return;
    const int stream = tasks * 8;
    auto load = [&](int j) {
        if (j < stream) {
            const int task = task0 + (j >> 3), r0 = task / ct * 64, c0 = task % ct * COLS;
            int first, count;
            segment(w.k, j & 7, first, count);
            char* const dst = sm + j % nbuf * buf;
            // eight lanes take the 16-byte pieces of a row (a piece of up to 8 x 64 bytes), four rows to a warp
            for (int c = lane & 7; c < count * 4; c += 8) {
                const __nv_bfloat16* ws = w.w + first * 32 + c * 8;
                const __nv_bfloat16* xs = x.x + first * 32 + c * 8;
                char* const to = dst + c * 16;
#pragma unroll
                for (int i = 0; i < 64 / 32; ++i) {
                    const int r = i * 32 + warp * 4 + (lane >> 3);
                    cp16(to + r * pitch, xs + (size_t)min(r0 + r, rows - 1) * x.ld);
                }
#pragma unroll
                for (int i = 0; i < COLS / 32; ++i) {
                    const int r = i * 32 + warp * 4 + (lane >> 3);
                    cp16(to + (64 + r) * pitch, ws + (size_t)min(c0 + r, w.n - 1) * w.ld);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int j = 0; j < nbuf - 1; ++j) load(j);
    float tot[2][MT][NT][4];
    for (int task = task0; task < task0 + tasks; ++task) {
        const int j0 = (task - task0) * 8;
#pragma unroll
        for (int sg = 0; sg < 8; ++sg) {
            wait_pending(nbuf - 2);
            __syncthreads();  // segment j0 + sg has landed; every warp is done with the one before, whose buffer comes next
            load(j0 + sg + nbuf - 1);
            const char* src = sm + (j0 + sg) % nbuf * buf;
            const char* xb = src + (wr * NT * 8 + g) * pitch + t * 16;
            const char* wb = src + (64 + wc * MT * 16 + g) * pitch + t * 16;
            float acc[MT][NT][4];
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) acc[m][nt][0] = acc[m][nt][1] = acc[m][nt][2] = acc[m][nt][3] = 0.0f;
            int first, count;
            segment(w.k, sg, first, count);
#pragma unroll 2
            for (int kb = 0; kb < count; ++kb) {
                uint4 a[MT][2], b[NT];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    a[m][0] = *reinterpret_cast<const uint4*>(wb + m * 16 * pitch + kb * 64);
                    a[m][1] = *reinterpret_cast<const uint4*>(wb + (m * 16 + 8) * pitch + kb * 64);
                }
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) b[nt] = *reinterpret_cast<const uint4*>(xb + nt * 8 * pitch + kb * 64);
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) mma_step(acc[m][nt], a[m][0], a[m][1], b[nt]);
            }
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        tot[sg >> 2][m][nt][e] = (sg & 3) == 0 ? acc[m][nt][e] : tot[sg >> 2][m][nt][e] + acc[m][nt][e];
        }
        const int r0 = task / ct * 64, c0 = task % ct * COLS;
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int c = c0 + wc * MT * 16 + m * 16 + g, r = r0 + (wr * NT + nt) * 8 + 2 * t;
                float v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = tot[0][m][nt][e] + tot[1][m][nt][e];
                epi(c, r, v[0], v[2]);      // columns c and c + 8 of row r
                epi(c, r + 1, v[1], v[3]);  // and of row r + 1
            }
    }
    wait_pending(0);
    __syncthreads();
}
// fewer than a tile per SM: tiles of 32 columns, otherwise 64
template <class Epi>
__device__ __forceinline__ void large_product(const Weights& w, const RowsBf16& x, int rows, char* sm, bool narrow, Epi&& epi) {
    if (narrow) large_product<1, 2>(w, x, rows, sm, epi);
    else large_product<2, 2>(w, x, rows, sm, epi);
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

// SSM step: a warp owns 8 adjacent channels (four lanes to a channel) of some of the rows, so rates, norm and query weights stay in
// registers; the carries of RING rows and the operands of the next ones are in flight (at hundreds of rows the stage is
// the carries' trip through HBM). What does not depend on this step's products is asked for before the barrier.
template <int NV, int RING>  // states per channel / 16; rows whose carries are in flight
struct SsmAhead {
    float4 rates[NV], h[RING][NV];
    uint4 wq[4];
    float gamma, beta;
    float* carry[RING];
    int r0, r1, group;
};
template <int NV, int RING>
__device__ __forceinline__ void ssm_request(const StepArgs& a, const StepBlock& b, SsmAhead<NV, RING>& q) {
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, groups = a.d / 8;
    const int chunks = min(a.rows, (int)gridDim.x * kWarps / groups), chunk = w / groups;
    q.group = w % groups;
    q.r0 = chunk < chunks ? (int)((long long)a.rows * chunk / chunks) : 0, q.r1 = chunk < chunks ? (int)((long long)a.rows * (chunk + 1) / chunks) : 0;
    if (q.r0 >= q.r1) return;
    const int i = q.group * 8 + (lane >> 2);
#pragma unroll
    for (int u = 0; u < RING; ++u)
        if (q.r0 + u < q.r1) {
            const float* c = q.carry[u] = b.state + (size_t)a.slots[q.r0 + u] * a.carry_stride + (size_t)i * (NV * 16) + (lane & 3) * 4;
#pragma unroll
            for (int v = 0; v < NV; ++v) q.h[u][v] = *reinterpret_cast<const float4*>(c + v * 16);
        }
#pragma unroll
    for (int v = 0; v < NV; ++v) q.rates[v] = __ldg(reinterpret_cast<const float4*>(b.rates + (size_t)i * (NV * 16) + v * 16 + (lane & 3) * 4));
#pragma unroll
    for (int v = 0; v < 4; ++v)
        if (v * 32 < a.k) q.wq[v] = __ldg(reinterpret_cast<const uint4*>(b.wqh + (size_t)(v * 32 + lane) * a.d + q.group * 8));
    q.gamma = __ldg(b.gamma + i), q.beta = __ldg(b.beta + i);
}
template <int NV, int RING>
__device__ __forceinline__ void ssm_stage(const StepArgs& a, const Features& f, SsmAhead<NV, RING>& s, float* state) {
    if (s.r0 >= s.r1) return;
    constexpr int LEAD = RING > 2 ? 2 : 1;  // rows whose operands are asked for ahead
    const int lane = threadIdx.x & 31, q = lane & 3, groups = a.d / 8, i = s.group * 8 + (lane >> 2);
    struct Row {
        float dl, e, inv;
        float4 b[NV], c[NV];
    } in[RING];
    auto fetch = [&](int r, Row& o) {
        const float* pr = a.proj + (size_t)r * a.nc;
        o.dl = ld_f(pr + i), o.e = ld_f(f.row(r) + i), o.inv = ld_f(a.inv + r);
#pragma unroll
        for (int v = 0; v < NV; ++v) o.b[v] = ld_f4(pr + a.off_b + v * 16 + q * 4), o.c[v] = ld_f4(pr + a.off_b + NV * 16 + v * 16 + q * 4);
    };
    fetch(s.r0, in[0]);
    if (LEAD > 1 && s.r0 + 1 < s.r1) fetch(s.r0 + 1, in[1]);
    unsigned slot = s.r0 + RING < s.r1 ? a.slots[s.r0 + RING] : 0;  // of the row whose carry is asked for next
    for (int rb = s.r0; rb < s.r1; rb += RING) {
#pragma unroll
        for (int u = 0; u < RING; ++u) {
            const int r = rb + u;
            if (r >= s.r1) break;
            if (r + LEAD < s.r1) fetch(r + LEAD, in[(u + LEAD) % RING]);
            const Row& now = in[u];
            const float x = norm1(now.e, now.inv, s.gamma, s.beta);
            const float w = now.dl * x, kf = now.dl * 1.4426950408889634f;
            float* carry = s.carry[u];
            float y = 0.0f;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const float4 r4 = s.rates[v], h4 = s.h[u][v], b4 = now.b[v], c4 = now.c[v];
                float4 h;
                h.x = fmaf(ex2(kf * r4.x), h4.x, w * b4.x), h.y = fmaf(ex2(kf * r4.y), h4.y, w * b4.y);
                h.z = fmaf(ex2(kf * r4.z), h4.z, w * b4.z), h.w = fmaf(ex2(kf * r4.w), h4.w, w * b4.w);
                y += fmaf(h.x, c4.x, fmaf(h.y, c4.y, fmaf(h.z, c4.z, h.w * c4.w)));
                *reinterpret_cast<float4*>(carry + v * 16) = h;
            }
            if (r + RING < s.r1) {
                const float* c = s.carry[u] = state + (size_t)slot * a.carry_stride + (size_t)i * (NV * 16) + q * 4;
                if (r + RING + 1 < s.r1) slot = a.slots[r + RING + 1];
#pragma unroll
                for (int v = 0; v < NV; ++v) s.h[u][v] = *reinterpret_cast<const float4*>(c + v * 16);
            }
            y += __shfl_xor_sync(0xffffffffu, y, 1);
            y += __shfl_xor_sync(0xffffffffu, y, 2);
            if (q == 0) a.y[(size_t)r * a.d + i] = y;
            float yc[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) yc[c] = __shfl_sync(0xffffffffu, y, c * 4);
#pragma unroll
            for (int v = 0; v < 4; ++v)
                if (v * 32 < a.k) {
                    const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&s.wq[v]);
                    float acc = 0.0f;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float2 wf = __bfloat1622float2(w2[c]);
                        acc = fmaf(wf.x, yc[2 * c], acc), acc = fmaf(wf.y, yc[2 * c + 1], acc);
                    }
                    a.qpart[((size_t)r * groups + s.group) * a.k + v * 32 + lane] = acc;
                }
        }
    }
}

// Memory read of a row by one CTA: the formulas of retrieve_small_rows_kernel (projection in f64, squared differences in fp32,
// hardware-approximation distance, ex2.approx weights, one reciprocal per row). The keys (a hundred KB, the same for every
// row) are asked for before the barrier the query waits at.
__device__ __forceinline__ bool request_keys(const StepArgs& a, const StepBlock& b, float* dst) {
    const int n = a.k / 4 * a.cap;
    if ((int)blockIdx.x >= a.rows || n > kKeyQuads) return false;
    for (int i = threadIdx.x; i < n; i += kThreads) cp16(reinterpret_cast<char*>(dst) + i * 16, b.keys_t + (size_t)i * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
    return true;
}
template <int K>
__device__ __forceinline__ void read_rows(const StepArgs& a, const StepBlock& b, float* sm, const float* keys) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, groups = a.d / 8;
    float* pt = sm;               // [K] query, then the projected point
    float* qp = sm + 128;         // [256] partial sums of the query
    float* red = sm + 128 + 256;  // [8]
    float* misc = red + 8;        // 1 / (1 - |p|^2)
    constexpr int parts = kThreads / K;
    const int part = tid / K, kk = tid % K;
    const float scale2 = (1.0f / a.tau) * 1.4426950408889634f;
    if (keys) asm volatile("cp.async.wait_group 0;" ::: "memory");  // seen by all behind the next __syncthreads
    for (int r = blockIdx.x; r < a.rows; r += gridDim.x) {
        {
            float acc = 0.0f;
            const float* src = a.qpart + (size_t)r * groups * K + kk;
            const int g0 = groups * part / parts, g1 = groups * (part + 1) / parts;
#pragma unroll 24
            for (int gq = g0; gq < g1; ++gq) acc += ld_f(src + (size_t)gq * K);
            qp[tid] = acc;
        }
        __syncthreads();
        if (tid < K) {
            float v = ld_f(a.proj + (size_t)r * a.nc + a.off_q + tid);
#pragma unroll
            for (int p = 0; p < parts; ++p) v += qp[p * K + tid];
            pt[tid] = v;
        }
        __syncthreads();
        if (warp == 0) {
            double r2 = 0.0;
#pragma unroll
            for (int i = lane; i < K; i += 32) r2 += (double)pt[i] * (double)pt[i];
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) r2 += __shfl_xor_sync(0xffffffffu, r2, m);
            const double rad = sqrt(r2), max_radius = 1.0 - 8.0 * (double)FLT_EPSILON;
            // min(rad / (1 + rad), max_radius) / rad with one division
            const double scale = rad * (1.0 - max_radius) < max_radius ? 1.0 / (1.0 + rad) : max_radius / rad;
            double n2 = 0.0;
#pragma unroll
            for (int i = lane; i < K; i += 32) {
                const float pv = (float)((double)pt[i] * scale);
                pt[i] = pv;
                n2 += (double)pv * (double)pv;
            }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, m);
            if (lane == 0) {
                const float qs = (n2 < 1.0 && (float)n2 == 1.0f) ? __uint_as_float(0x3f7fffffu) : (float)n2;
                misc[0] = (float)(1.0 / (1.0 - (double)qs));
            }
        }
        __syncthreads();
        float dist[4], mn = FLT_MAX;
        const float row_inv = misc[0];
        // slots past `count` hold nothing: weight zero. Two slots at a time share the point's reads
        const float4* const kq = reinterpret_cast<const float4*>(keys ? keys : b.keys_t);
#pragma unroll
        for (int u = 0; u < 4; u += 2) {
            dist[u] = dist[u + 1] = CUDART_INF_F;
            const int s0 = tid + u * kThreads, s1 = s0 + kThreads;
            if (u * kThreads >= a.cap) continue;
            const float4 *p0 = kq + min(s0, a.cap - 1), *p1 = kq + min(s1, a.cap - 1);
            const float n0 = __ldg(b.norm_sq + min(s0, a.cap - 1)), n1 = __ldg(b.norm_sq + min(s1, a.cap - 1));
            float q0 = 0.0f, q1 = 0.0f;
#pragma unroll 8
            for (int i = 0; i < K / 4; ++i) {
                const float4 pv = *reinterpret_cast<const float4*>(pt + i * 4), v0 = p0[i * a.cap], v1 = p1[i * a.cap];
                float x = pv.x - v0.x, y = pv.y - v0.y, z = pv.z - v0.z, w = pv.w - v0.w;
                q0 = fmaf(x, x, q0), q0 = fmaf(y, y, q0), q0 = fmaf(z, z, q0), q0 = fmaf(w, w, q0);
                x = pv.x - v1.x, y = pv.y - v1.y, z = pv.z - v1.z, w = pv.w - v1.w;
                q1 = fmaf(x, x, q1), q1 = fmaf(y, y, q1), q1 = fmaf(z, z, q1), q1 = fmaf(w, w, q1);
            }
            if (s0 < b.count) dist[u] = fast_poincare_distance(q0 * (row_inv * __fdividef(1.0f, 1.0f - n0))), mn = fminf(mn, dist[u]);
            if (s1 < b.count) dist[u + 1] = fast_poincare_distance(q1 * (row_inv * __fdividef(1.0f, 1.0f - n1))), mn = fminf(mn, dist[u + 1]);
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, m));
        if (lane == 0) red[warp] = mn;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < 8; ++w) mn = fminf(mn, red[w]);
        __syncthreads();
        float sum = 0.0f;
#pragma unroll
        for (int u = 0; u < 4; ++u) dist[u] = ex2((mn - dist[u]) * scale2), sum += dist[u];
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
        if (lane == 0) red[warp] = sum;
        __syncthreads();
        const float total = ((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]));
        const float inv_sum = __fdiv_rn(1.0f, total);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int s = tid + u * kThreads;
            if (s < a.cap) a.w[(size_t)r * 3 * a.cap + s] = __float2bfloat16_rn(dist[u] * inv_sum);
        }
        __syncthreads();
    }
}
__device__ __forceinline__ void read_stage(const StepArgs& a, const StepBlock& b, float* sm, const float* keys) {
    if (a.k == 64) read_rows<64>(a, b, sm, keys);
    else read_rows<128>(a, b, sm, keys);
}

// ---- epilogues: one output each, the same instructions whichever product calls them
__device__ __forceinline__ void store_xside(const StepArgs& a, int col, int row, float v) {
    if (col >= a.nc || row >= a.rows) return;
    if (col >= a.off_act) {  // adapter activations: the extra K block of both MLP operands
        const __nv_bfloat16 h = __float2bfloat16_rn(v / (1.0f + __expf(-v)));
        a.z[(size_t)row * (a.d + 64) + a.d + col - a.off_act] = h;
        a.act[(size_t)row * (2 * a.d + 64) + 2 * a.d + col - a.off_act] = h;
        return;
    }
    a.proj[(size_t)row * a.nc + col] = col < a.off_b ? softplus_fast(v) : col < a.off_gate ? v : 1.0f / (1.0f + __expf(-v));
}
__device__ __forceinline__ void store_gated(const StepArgs& a, int col, int row, float v) {
    if (col >= a.d || row >= a.rows) return;
    const float g = ld_f(a.proj + (size_t)row * a.nc + a.off_gate + col), y = ld_f(a.y + (size_t)row * a.d + col);
    a.z[(size_t)row * (a.d + 64) + col] = __float2bfloat16_rn(fmaf(g, v, __fmul_rn(a.ssm_scale, y)));
}
__device__ __forceinline__ void store_hidden(const StepArgs& a, int col, int row, float v) {
    if (col >= 2 * a.d || row >= a.rows) return;
    a.act[(size_t)row * (2 * a.d + 64) + col] = __float2bfloat16_rn(v / (1.0f + __expf(-v)));
}
__device__ __forceinline__ float new_feature(const StepArgs& a, const float* in, float scale, int col, int row, float v) {
    if (col >= a.d || row >= a.rows) return 0.0f;
    const unsigned short zb = __ldcg(reinterpret_cast<const unsigned short*>(a.z + (size_t)row * (a.d + 64) + col));
    const float f = __fadd_rn(v, __bfloat162float(__ushort_as_bfloat16(zb)));
    return in ? fmaf(scale, f, ld_f(in + (size_t)row * a.d + col)) : f;
}
__device__ __forceinline__ void store_logit(const StepArgs& a, int col, int row, float v) {
    if (col < (int)a.vocab && row < a.rows) a.logits[(size_t)row * a.vocab + col] = __fmul_rn(v, a.head_scale);
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
// device-resident ids cannot be checked on the host: row 0 is read and the status word raised
__device__ __forceinline__ void check_ids(const StepArgs& a) {
    if (blockIdx.x == 0)
        for (int r = threadIdx.x; r < a.rows; r += kThreads)
            if (a.ids[r] >= a.vocab) atomicExch(a.status, PSSA_B200_ERR_TOKEN);
}

// ---- many rows: the same stages with 64-row tiles, and the normalised rows formed once, in a stage of their own
__device__ __forceinline__ void norm_stage(const StepArgs& a, const StepBlock& b, const Features& f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tiles = a.d / 16;
    for (int r = warp * gridDim.x + blockIdx.x; r < a.rows; r += gridDim.x * kWarps) {
        const float* e = f.row(r);
        float sum = 0.0f;
        if (f.ids) {
            for (int i = lane * 4; i < a.d; i += 128) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(e + i));
                sum = fmaf(v.x, v.x, sum), sum = fmaf(v.y, v.y, sum), sum = fmaf(v.z, v.z, sum), sum = fmaf(v.w, v.w, sum);
            }
        } else {
            for (int i = lane; i < tiles; i += 32) sum += ld_f(a.ssq + (size_t)r * tiles + i);
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
        const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum, (float)a.d), 1e-5f)));
        if (lane == 0) a.inv[r] = inv;
#pragma unroll 2
        for (int i = lane * 8; i < a.d; i += 256) {
            const float4 u = ld_f4(e + i), v = ld_f4(e + i + 4);
            const float4 gu = __ldg(reinterpret_cast<const float4*>(b.gamma + i)), gv = __ldg(reinterpret_cast<const float4*>(b.gamma + i + 4));
            const float4 tu = __ldg(reinterpret_cast<const float4*>(b.beta + i)), tv = __ldg(reinterpret_cast<const float4*>(b.beta + i + 4));
            *reinterpret_cast<uint4*>(a.x + (size_t)r * a.d + i) =
                make_uint4(pack_bf16(norm1(u.x, inv, gu.x, tu.x), norm1(u.y, inv, gu.y, tu.y)), pack_bf16(norm1(u.z, inv, gu.z, tu.z), norm1(u.w, inv, gu.w, tu.w)),
                           pack_bf16(norm1(v.x, inv, gv.x, tv.x), norm1(v.y, inv, gv.y, tv.y)), pack_bf16(norm1(v.z, inv, gv.z, tv.z), norm1(v.w, inv, gv.w, tv.w)));
        }
    }
}
// Weights of this block's later products and the next block's first one, on their way to L2 during the SSM stage: a product's
// tiles are few and would wait for HBM otherwise
__device__ __forceinline__ void prefetch_weights(const StepArgs& a, int l) {
    const size_t d = a.d;
    const int thread = blockIdx.x * kThreads + threadIdx.x, threads = gridDim.x * kThreads;
    auto lines = [&](const __nv_bfloat16* w, size_t n) {
        for (size_t i = (size_t)thread * 64; i < n; i += (size_t)threads * 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(w + i));
    };
    const StepBlock& b = a.block[l];
    lines(b.w1, 2 * d * (d + 64));
    lines(b.w2, d * (2 * d + 64));
    for (int i = thread; i < a.d * (a.cap / 64); i += threads)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(b.vp + (size_t)(i / (a.cap / 64)) * 3 * a.cap + i % (a.cap / 64) * 64));
    if (l + 1 < a.depth) lines(a.block[l + 1].wcat, (size_t)a.nc * d);
}

template <int NV>
__global__ void __launch_bounds__(kThreads, 1) step_large_kernel(const __grid_constant__ StepArgs a) {
    extern __shared__ __align__(128) float step_smem[];
    char* sm = reinterpret_cast<char*>(step_smem);
    Barrier bar{a.barrier, a.status, 0, false};
    bar.init();
    check_ids(a);
    prefetch_vectors(a, 0);
    const int d = a.d, tiles = d / 16, rt = (a.rows + 63) / 64;
    const bool narrow = (d / 32) * rt <= (int)gridDim.x;  // tiles of 64 columns would leave half of the SMs without one
    const float* in = nullptr;
    for (int l = 0; l < a.depth; ++l) {
        const StepBlock& b = a.block[l];
        float* out = in == a.feat_a ? a.feat_b : a.feat_a;
        const Features f{a.embed, l == 0 ? a.ids : nullptr, in, d, a.vocab};
        norm_stage(a, b, f);
        bar.arrive();
        bar.wait();
        large_product({b.wcat, (size_t)d, a.nc, d}, RowsBf16{a.x, (size_t)d}, a.rows, sm, narrow,
                      [&](int c, int r, float v0, float v1) { store_xside(a, c, r, v0), store_xside(a, c + 8, r, v1); });
        bar.arrive();
        bar.wait();
        prefetch_weights(a, l);
        {
            SsmAhead<NV, 3> sa;
            ssm_request(a, b, sa);
            ssm_stage(a, f, sa, b.state);
        }
        bar.arrive();
        bar.wait();
        {
            float* const keys = reinterpret_cast<float*>(sm) + 448;
            const bool staged = request_keys(a, b, keys);
            read_stage(a, b, reinterpret_cast<float*>(sm), staged ? keys : nullptr);
        }
        bar.arrive();
        bar.wait();
        large_product({b.vp, (size_t)3 * a.cap, d, a.cap}, RowsBf16{a.w, (size_t)3 * a.cap}, a.rows, sm, narrow,
                      [&](int c, int r, float v0, float v1) { store_gated(a, c, r, v0), store_gated(a, c + 8, r, v1); });
        prefetch_vectors(a, l + 1);
        bar.arrive();
        bar.wait();
        large_product({b.w1, (size_t)d + 64, 2 * d, d + 64}, RowsBf16{a.z, (size_t)d + 64}, a.rows, sm, narrow,
                      [&](int c, int r, float v0, float v1) { store_hidden(a, c, r, v0), store_hidden(a, c + 8, r, v1); });
        bar.arrive();
        bar.wait();
        large_product({b.w2, (size_t)2 * d + 64, d, 2 * d + 64}, RowsBf16{a.act, (size_t)2 * d + 64}, a.rows, sm, narrow,
                      [&](int c, int r, float v0, float v1) {
            // and the sum of squares of each 16 of them: pair c, c + 8 first, then over the eight c
            const float f0 = new_feature(a, in, b.res_scale, c, r, v0), f1 = new_feature(a, in, b.res_scale, c + 8, r, v1);
            const bool live = r < a.rows && c < d;
            if (live) {
                out[(size_t)r * d + c] = f0, out[(size_t)r * d + c + 8] = f1;
                if (l + 1 == a.depth) a.x[(size_t)r * d + c] = __float2bfloat16_rn(f0), a.x[(size_t)r * d + c + 8] = __float2bfloat16_rn(f1);
            }
            float q = __fadd_rn(__fmul_rn(f0, f0), __fmul_rn(f1, f1));
            q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 4));
            q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 8));
            q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 16));
            if ((threadIdx.x & 31) < 4 && live) a.ssq[(size_t)r * tiles + c / 16] = q;
        });
        in = out;
        bar.arrive();
        bar.wait();
    }
    if (a.logits)
        large_product<2, 2>({a.unembed, (size_t)d, (int)a.vocab, d}, RowsBf16{a.x, (size_t)d}, a.rows, sm,
                            [&](int c, int r, float v0, float v1) { store_logit(a, c, r, v0), store_logit(a, c + 8, r, v1); });
}

// Up to kSmallRows rows, NT 8-row tiles of them: the stages are inlined, because the weights and carries that a stage asks for before
// the barrier in front of it stay in registers across it.
template <int NT, int NV>
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
    check_ids(a);
    prefetch_vectors(a, 0);
    const float* in = nullptr;
    for (int l = 0; l < a.depth; ++l) {
        const StepBlock& b = a.block[l];
        float* out = in == a.feat_a ? a.feat_b : a.feat_a;
        const Features f{a.embed, l == 0 ? a.ids : nullptr, in, d, a.vocab};
        const Weights wcat{b.wcat, (size_t)d, a.nc, d}, vp{b.vp, (size_t)3 * a.cap, d, a.cap}, w1{b.w1, (size_t)d + 64, 2 * d, d + 64},
            w2{b.w2, (size_t)2 * d + 64, d, 2 * d + 64};
        row_scales(a, f, 0, a.rows, inv_s, blockIdx.x == 0);
        small_product<NT>(wcat, RowsNorm{f, b.gamma, b.beta, inv_s, 0}, a.rows, ah, sm, [&](int c, int r, float v) { store_xside(a, c, r, v); });
        bar.arrive();
        SsmAhead<NV, 2> sa;
        ssm_request(a, b, sa);
        const bool keys_here = request_keys(a, b, keys_s);
        bar.wait();
        ssm_stage(a, f, sa, b.state);
        bar.arrive();
        ahead(vp);
        bar.wait();
        read_stage(a, b, sm, keys_here ? keys_s : nullptr);
        bar.arrive();
        bar.wait();
        const RowsBf16 xw{a.w, (size_t)3 * a.cap}, xz{a.z, (size_t)d + 64}, xa{a.act, (size_t)2 * d + 64};
        small_product<NT>(vp, xw, a.rows, ah, sm, [&](int c, int r, float v) { store_gated(a, c, r, v); });
        bar.arrive();
        ahead(w1);
        prefetch_vectors(a, l + 1);
        bar.wait();
        small_product<NT>(w1, xz, a.rows, ah, sm, [&](int c, int r, float v) { store_hidden(a, c, r, v); });
        bar.arrive();
        ahead(w2);
        bar.wait();
        small_product<NT>(w2, xa, a.rows, ah, sm, [&](int c, int r, float v) {
            const float fv = new_feature(a, in, b.res_scale, c, r, v);
            if (r < a.rows) out[(size_t)r * d + c] = fv;
            float q = __fmul_rn(fv, fv);
            q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 8));
            q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 1));
            q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 2));
            q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 4));
            if (c % 16 == 0 && r < a.rows) a.ssq[(size_t)r * tiles + c / 16] = q;
        });
        in = out;
        bar.arrive();
        if (l + 1 < a.depth) ahead({a.block[l + 1].wcat, (size_t)d, a.nc, d});
        else if (a.logits) ahead({a.unembed, (size_t)d, (int)a.vocab, d});
        bar.wait();
    }
    if (!a.logits) return;
    small_product<NT>({a.unembed, (size_t)d, (int)a.vocab, d}, RowsF32{in, (size_t)d}, a.rows, ah, sm, [&](int c, int r, float v) { store_logit(a, c, r, v); });
}

template <int NV>
void* kernel_of(int nt) {
    return nt == 1 ? (void*)step_kernel<1, NV> : nt == 2 ? (void*)step_kernel<2, NV> : nt == 4 ? (void*)step_kernel<4, NV> : (void*)step_large_kernel<NV>;
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

bool step_rows_ok(size_t rows) { return rows <= kStepRows; }

bool step_shape_ok(size_t depth, size_t d, size_t s, size_t k, size_t cap, size_t rank) {
    return depth <= kMaxDepth && d % 32 == 0 && 2 * d + 64 <= 1664 && (s == 16 || s == 32 || s == 64) && (k == 64 || k == 128) && cap % 64 == 0 &&
           cap <= 4 * kThreads && rank == 16;
}

int32_t launch_decode_step(pssa_b200_ctx* ctx, const StepLaunch& p) {
    StepArgs a{};
    a.rows = p.rows, a.depth = (int)p.depth, a.d = p.d, a.s = p.s, a.k = p.k, a.cap = p.cap, a.nc = p.nc;
    a.off_b = p.off_b, a.off_q = p.off_q, a.off_gate = p.off_gate, a.off_act = p.off_act, a.vocab = p.vocab;
    a.ssm_scale = p.ssm_scale, a.head_scale = p.head_scale, a.tau = p.tau;
    a.embed = p.embed, a.ids = p.ids, a.slots = p.slots, a.unembed = (const __nv_bfloat16*)p.unembed, a.carry_stride = p.carry_stride;
    a.feat_a = p.feat_a, a.feat_b = p.feat_b, a.proj = p.proj, a.y = p.y, a.qpart = p.qpart, a.ssq = p.ssq, a.inv = p.inv, a.logits = p.logits;
    a.x = (__nv_bfloat16*)p.x, a.w = (__nv_bfloat16*)p.w, a.z = (__nv_bfloat16*)p.z, a.act = (__nv_bfloat16*)p.act, a.barrier = (unsigned long long*)p.barrier;
    a.status = ctx->status_dev;
    for (size_t l = 0; l < p.depth; ++l) {
        const StepLaunch::Block& s = p.blocks[l];
        a.block[l] = {(const __nv_bfloat16*)s.wcat, (const __nv_bfloat16*)s.wqh, (const __nv_bfloat16*)s.vp, (const __nv_bfloat16*)s.w1,
                      (const __nv_bfloat16*)s.w2,   s.rates, s.gamma, s.beta, s.keys_t, s.norm_sq, s.state, s.res_scale, s.count};
    }
    const int nt = p.rows <= 8 ? 1 : p.rows <= 16 ? 2 : p.rows <= kSmallRows ? 4 : 0;
    const size_t key_bytes = (size_t)std::min(p.k / 4 * p.cap, kKeyQuads) * 16;
    const size_t smem = 64 * 4 + (nt ? std::max(448, nt * 64 * kPitch) * 4 + key_bytes : std::max<size_t>(448 * 4 + key_bytes, kTileBytes));
    void* kern = p.s == 16 ? kernel_of<1>(nt) : p.s == 32 ? kernel_of<2>(nt) : kernel_of<4>(nt);
    PSSA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    void* args[] = {&a};
    // cooperative: the barriers need every CTA of the grid resident at once
    PSSA_CUDA(ctx, cudaLaunchCooperativeKernel(kern, dim3((unsigned)ctx->sm_count), dim3(kThreads), args, smem, ctx->stream));
    return after_launch(ctx, "step_kernel");
}

}  // namespace pssa
