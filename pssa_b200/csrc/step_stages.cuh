// Stages of a decode step (one token per row, bf16 mode) that its two forms share: one cooperative kernel for the whole step
// (step_decode.cu) and, for many rows, a launch per stage (step_schedule.cu). The choice between them must not show in a
// stream's bits, so everything that rounds is written once, here.
#pragma once
#include <cuda_bf16.h>
#include <math_constants.h>

#include <cfloat>

#include "context.hpp"
#include "device_math.cuh"
#include "kernels.hpp"

namespace pssa {
namespace step {

constexpr int kThreads = 256;
constexpr int kWarps = 8;
constexpr int kMaxDepth = 32;     // blocks whose pointers fit in the kernel's parameters
constexpr int kKeyQuads = 8192;   // the bank's keys are staged in shared memory (128 KB) up to here

__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<unsigned*>(&v);
}
// data written by other CTAs of this launch: not through the non-coherent path
__device__ __forceinline__ uint2 ld_u2(const void* p) {
    uint2 v;
    asm volatile("ld.global.cg.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
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
__device__ __forceinline__ void cp16(char* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
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


struct StepBlock {
    const __nv_bfloat16 *wcat, *wqh, *vp, *w1, *w2;
    const float *rates, *gamma, *beta, *keys_t, *norm_sq;
    float* state;  // carry of stream 0 of this block
    float res_scale;
    int count;
};
struct StepCommon {
    int rows, depth, d, k, cap, nc, off_b, off_q, off_gate, off_act;
    unsigned vocab;
    float ssm_scale, head_scale, tau;
    const float* embed;
    const unsigned *ids, *slots;  // [rows]; a host call's few rows have theirs in own_ids, own_slots
    const __nv_bfloat16* unembed;
    size_t carry_stride;
    float *feat_a, *feat_b, *proj, *y, *qpart, *ssq, *inv, *logits;
    __nv_bfloat16 *x, *w, *z, *act;  // x: the normalised rows, at the end the features (where rows have a norm stage)
    int* status;
    unsigned own_ids[kStepOwnRows], own_slots[kStepOwnRows];  // of a host call's few rows: no copy in front of the launch
};
// (OWN, known at compile time: a choice at run time costs the SSM stage registers it does not have, 270 -> 278 us a step)
template <bool OWN>
__device__ __forceinline__ const unsigned* ids_of(const StepCommon& a) { return OWN ? a.own_ids : a.ids; }
template <bool OWN>
__device__ __forceinline__ unsigned slot_of(const StepCommon& a, int r) { return OWN ? a.own_slots[r] : a.slots[r]; }

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

// segment s of K: its first 32-wide step and the number of them
__device__ __forceinline__ void segment(int k, int s, int& first, int& count) {
    const int nkb = k >> 5, base = nkb >> 3, rem = nkb & 7;
    first = s * base + min(s, rem), count = base + (s < rem ? 1 : 0);
}

// many rows: the normalised rows formed once, in a stage of their own
__device__ __forceinline__ void norm_stage(const StepCommon& a, const StepBlock& b, const Features& f) {
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
template <bool OWN = false, int NV, int RING>
__device__ __forceinline__ void ssm_request(const StepCommon& a, const StepBlock& b, SsmAhead<NV, RING>& q) {
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, groups = a.d / 8;
    const int chunks = min(a.rows, (int)gridDim.x * kWarps / groups), chunk = w / groups;
    q.group = w % groups;
    q.r0 = chunk < chunks ? (int)((long long)a.rows * chunk / chunks) : 0, q.r1 = chunk < chunks ? (int)((long long)a.rows * (chunk + 1) / chunks) : 0;
    if (q.r0 >= q.r1) return;
    const int i = q.group * 8 + (lane >> 2);
#pragma unroll
    for (int u = 0; u < RING; ++u)
        if (q.r0 + u < q.r1) {
            const float* c = q.carry[u] = b.state + (size_t)slot_of<OWN>(a, q.r0 + u) * a.carry_stride + (size_t)i * (NV * 16) + (lane & 3) * 4;
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
template <bool OWN = false, int NV, int RING>
__device__ __forceinline__ void ssm_stage(const StepCommon& a, const Features& f, SsmAhead<NV, RING>& s, float* state) {
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
    unsigned slot = s.r0 + RING < s.r1 ? slot_of<OWN>(a, s.r0 + RING) : 0;  // of the row whose carry is asked for next
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
                if (r + RING + 1 < s.r1) slot = slot_of<OWN>(a, r + RING + 1);
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
__device__ __forceinline__ bool request_keys(const StepCommon& a, const StepBlock& b, float* dst) {
    const int n = a.k / 4 * a.cap;
    if ((int)blockIdx.x >= a.rows || n > kKeyQuads) return false;
    for (int i = threadIdx.x; i < n; i += kThreads) cp16(reinterpret_cast<char*>(dst) + i * 16, b.keys_t + (size_t)i * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
    return true;
}
// R rows at a time share the keys' reads; a row's bits do not depend on R. `sm`: read_floats(R) floats.
constexpr int read_floats(int r) { return r * (128 + 256 + 8) + (r + 3) / 4 * 4; }
template <int K, int R>
__device__ __forceinline__ void read_rows(const StepCommon& a, const StepBlock& b, float* sm, const float* keys) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, groups = a.d / 8;
    float* pt = sm;              // [R][128] queries, then the projected points
    float* qp = pt + R * 128;    // [R][256] partial sums of the queries
    float* red = qp + R * 256;   // [R][8]
    float* misc = red + R * 8;   // [R] 1 / (1 - |p|^2)
    constexpr int parts = kThreads / K;
    const int part = tid / K, kk = tid % K;
    const float scale2 = (1.0f / a.tau) * 1.4426950408889634f;
    if (keys) asm volatile("cp.async.wait_group 0;" ::: "memory");  // seen by all behind the next __syncthreads
    for (int r0 = blockIdx.x * R; r0 < a.rows; r0 += gridDim.x * R) {
#pragma unroll
        for (int u = 0; u < R; ++u) {
            float acc = 0.0f;
            const float* src = a.qpart + (size_t)min(r0 + u, a.rows - 1) * groups * K + kk;
            const int g0 = groups * part / parts, g1 = groups * (part + 1) / parts;
            // 24 at a time whatever their number: in a loop's remainder each would be a trip to L2 of its own
            for (int gq = g0; gq < g1; gq += 24) {
                float t[24];
#pragma unroll
                for (int i = 0; i < 24; ++i) t[i] = gq + i < g1 ? ld_f(src + (size_t)(gq + i) * K) : 0.0f;
#pragma unroll
                for (int i = 0; i < 24; ++i) acc += t[i];
            }
            qp[u * 256 + tid] = acc;
        }
        __syncthreads();
        if (tid < K) {
#pragma unroll
            for (int u = 0; u < R; ++u) {
                float v = ld_f(a.proj + (size_t)min(r0 + u, a.rows - 1) * a.nc + a.off_q + tid);
#pragma unroll
                for (int p = 0; p < parts; ++p) v += qp[u * 256 + p * K + tid];
                pt[u * 128 + tid] = v;
            }
        }
        __syncthreads();
        if (warp < R) {
            float* const q = pt + warp * 128;
            double r2 = 0.0;
#pragma unroll
            for (int i = lane; i < K; i += 32) r2 += (double)q[i] * (double)q[i];
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) r2 += __shfl_xor_sync(0xffffffffu, r2, m);
            const double rad = sqrt(r2), max_radius = 1.0 - 8.0 * (double)FLT_EPSILON;
            // min(rad / (1 + rad), max_radius) / rad with one division
            const double scale = rad * (1.0 - max_radius) < max_radius ? 1.0 / (1.0 + rad) : max_radius / rad;
            double n2 = 0.0;
#pragma unroll
            for (int i = lane; i < K; i += 32) {
                const float pv = (float)((double)q[i] * scale);
                q[i] = pv;
                n2 += (double)pv * (double)pv;
            }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, m);
            if (lane == 0) {
                const float qs = (n2 < 1.0 && (float)n2 == 1.0f) ? __uint_as_float(0x3f7fffffu) : (float)n2;
                misc[warp] = (float)(1.0 / (1.0 - (double)qs));
            }
        }
        __syncthreads();
        float dist[R][4], mn[R];
#pragma unroll
        for (int u = 0; u < R; ++u) mn[u] = FLT_MAX;
        // slots past `count` hold nothing: weight zero. Two slots at a time share the points' reads
        const float4* const kq = reinterpret_cast<const float4*>(keys ? keys : b.keys_t);
#pragma unroll
        for (int v = 0; v < 4; v += 2) {
#pragma unroll
            for (int u = 0; u < R; ++u) dist[u][v] = dist[u][v + 1] = CUDART_INF_F;
            const int s0 = tid + v * kThreads, s1 = s0 + kThreads;
            if (v * kThreads >= a.cap) continue;
            const float4 *p0 = kq + min(s0, a.cap - 1), *p1 = kq + min(s1, a.cap - 1);
            const float n0 = __ldg(b.norm_sq + min(s0, a.cap - 1)), n1 = __ldg(b.norm_sq + min(s1, a.cap - 1));
            float q0[R], q1[R];
#pragma unroll
            for (int u = 0; u < R; ++u) q0[u] = q1[u] = 0.0f;
#pragma unroll 8
            for (int i = 0; i < K / 4; ++i) {
                const float4 v0 = p0[i * a.cap], v1 = p1[i * a.cap];
#pragma unroll
                for (int u = 0; u < R; ++u) {
                    const float4 pv = *reinterpret_cast<const float4*>(pt + u * 128 + i * 4);
                    float x = pv.x - v0.x, y = pv.y - v0.y, z = pv.z - v0.z, w = pv.w - v0.w;
                    q0[u] = fmaf(x, x, q0[u]), q0[u] = fmaf(y, y, q0[u]), q0[u] = fmaf(z, z, q0[u]), q0[u] = fmaf(w, w, q0[u]);
                    x = pv.x - v1.x, y = pv.y - v1.y, z = pv.z - v1.z, w = pv.w - v1.w;
                    q1[u] = fmaf(x, x, q1[u]), q1[u] = fmaf(y, y, q1[u]), q1[u] = fmaf(z, z, q1[u]), q1[u] = fmaf(w, w, q1[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const float row_inv = misc[u];
                if (s0 < b.count)
                    dist[u][v] = fast_poincare_distance(q0[u] * (row_inv * __fdividef(1.0f, 1.0f - n0))), mn[u] = fminf(mn[u], dist[u][v]);
                if (s1 < b.count)
                    dist[u][v + 1] = fast_poincare_distance(q1[u] * (row_inv * __fdividef(1.0f, 1.0f - n1))), mn[u] = fminf(mn[u], dist[u][v + 1]);
            }
        }
#pragma unroll
        for (int u = 0; u < R; ++u) {
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) mn[u] = fminf(mn[u], __shfl_xor_sync(0xffffffffu, mn[u], m));
            if (lane == 0) red[u * 8 + warp] = mn[u];
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < R; ++u)
#pragma unroll
            for (int w = 0; w < 8; ++w) mn[u] = fminf(mn[u], red[u * 8 + w]);
        __syncthreads();
#pragma unroll
        for (int u = 0; u < R; ++u) {
            float sum = 0.0f;
#pragma unroll
            for (int v = 0; v < 4; ++v) dist[u][v] = ex2((mn[u] - dist[u][v]) * scale2), sum += dist[u][v];
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
            if (lane == 0) red[u * 8 + warp] = sum;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const float* t = red + u * 8;
            const float total = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
            const float inv_sum = __fdiv_rn(1.0f, total);
            if (r0 + u < a.rows)
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const int s = tid + v * kThreads;
                    if (s < a.cap) a.w[(size_t)(r0 + u) * 3 * a.cap + s] = __float2bfloat16_rn(dist[u][v] * inv_sum);
                }
        }
        __syncthreads();
    }
}
template <int R>
__device__ __forceinline__ void read_stage(const StepCommon& a, const StepBlock& b, float* sm, const float* keys) {
    if (a.k == 64) read_rows<64, R>(a, b, sm, keys);
    else read_rows<128, R>(a, b, sm, keys);
}

// ---- epilogues, one output each: what it reads besides the product (fetch: of an output inside the matrix), its value, its place
// Where nothing is read, eight outputs of a column at once too (values): their chains side by side, no branch between them.
struct Pre {
    float a, b;
};
__device__ __forceinline__ void logistic(float (&f)[8], bool sigmoid) {  // sigmoid, or SiLU
    float e[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] = 1.0f + __expf(-f[i]);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = (sigmoid ? 1.0f : f[i]) / e[i];
}
struct PutXside {  // x-side products: softplus | B, C, q_x | gate | adapter
    static constexpr bool kReads = false;
    const StepCommon& a;
    __device__ __forceinline__ int cols() const { return a.nc; }
    __device__ __forceinline__ Pre fetch(int, int) const { return {0.0f, 0.0f}; }
    __device__ __forceinline__ float value(int col, float v, Pre) const {
        if (col < a.off_b) return softplus_fast(v);
        if (col < a.off_gate) return v;
        return (col < a.off_act ? 1.0f : v) / (1.0f + __expf(-v));
    }
    __device__ __forceinline__ void values(int col, float (&f)[8]) const {
        if (col < a.off_b) {
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = softplus_fast(f[i]);
        } else if (col >= a.off_gate) {
            logistic(f, col < a.off_act);
        }
    }
    __device__ __forceinline__ void store(int col, int row, float f) const {
        if (col >= a.off_act) {  // adapter activations: the extra K block of both MLP operands
            const __nv_bfloat16 h = __float2bfloat16_rn(f);
            a.z[(size_t)row * (a.d + 64) + a.d + col - a.off_act] = h;
            a.act[(size_t)row * (2 * a.d + 64) + 2 * a.d + col - a.off_act] = h;
        } else {
            a.proj[(size_t)row * a.nc + col] = f;
        }
    }
};
struct PutGated {  // z' = gate * v + y / sqrt(s)
    static constexpr bool kReads = true;
    const StepCommon& a;
    __device__ __forceinline__ int cols() const { return a.d; }
    __device__ __forceinline__ Pre fetch(int col, int row) const {
        return {ld_f(a.proj + (size_t)row * a.nc + a.off_gate + col), ld_f(a.y + (size_t)row * a.d + col)};
    }
    __device__ __forceinline__ float value(int, float v, Pre p) const { return fmaf(p.a, v, __fmul_rn(a.ssm_scale, p.b)); }
    __device__ __forceinline__ void store(int col, int row, float f) const { a.z[(size_t)row * (a.d + 64) + col] = __float2bfloat16_rn(f); }
};
struct PutHidden {
    static constexpr bool kReads = false;
    const StepCommon& a;
    __device__ __forceinline__ int cols() const { return 2 * a.d; }
    __device__ __forceinline__ Pre fetch(int, int) const { return {0.0f, 0.0f}; }
    __device__ __forceinline__ float value(int, float v, Pre) const { return v / (1.0f + __expf(-v)); }
    __device__ __forceinline__ void values(int, float (&f)[8]) const { logistic(f, false); }
    __device__ __forceinline__ void store(int col, int row, float f) const { a.act[(size_t)row * (2 * a.d + 64) + col] = __float2bfloat16_rn(f); }
};
struct PutLogit {
    static constexpr bool kReads = false;
    const StepCommon& a;
    __device__ __forceinline__ int cols() const { return (int)a.vocab; }
    __device__ __forceinline__ Pre fetch(int, int) const { return {0.0f, 0.0f}; }
    __device__ __forceinline__ float value(int, float v, Pre) const { return __fmul_rn(v, a.head_scale); }
    __device__ __forceinline__ void values(int, float (&f)[8]) const {
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = __fmul_rn(f[i], a.head_scale);
    }
    __device__ __forceinline__ void store(int col, int row, float f) const { a.logits[(size_t)row * a.vocab + col] = f; }
};
template <class Put>
__device__ __forceinline__ void store(const Put& p, int col, int row, float v) {
    if (col < p.cols() && row < p.a.rows) p.store(col, row, p.value(col, v, p.fetch(col, row)));
}
// the block's output: features + scale * (W2 h + z'), or W2 h + z' in the first block
__device__ __forceinline__ Pre feature_fetch(const StepCommon& a, const float* in, int col, int row) {
    const unsigned short zb = __ldcg(reinterpret_cast<const unsigned short*>(a.z + (size_t)row * (a.d + 64) + col));
    return {__bfloat162float(__ushort_as_bfloat16(zb)), in ? ld_f(in + (size_t)row * a.d + col) : 0.0f};
}
__device__ __forceinline__ float feature_value(Pre p, bool residual, float scale, float v) {
    const float f = __fadd_rn(v, p.a);
    return residual ? fmaf(scale, f, p.b) : f;
}
// sum of squares of the 16 columns that 16 neighbouring lanes hold: the pair c, c + 8 first, then over the eight c
__device__ __forceinline__ float squares16(float f) {
    float q = __fmul_rn(f, f);
    q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 8));
    q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 1));
    q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 2));
    return __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, 4));
}
__device__ __forceinline__ float new_feature(const StepCommon& a, const float* in, float scale, int col, int row, float v) {
    if (col >= a.d || row >= a.rows) return 0.0f;
    return feature_value(feature_fetch(a, in, col, row), in != nullptr, scale, v);
}

// device-resident ids cannot be checked on the host: row 0 is read and the status word raised
template <bool OWN = false>
__device__ __forceinline__ void check_ids(const StepCommon& a) {
    if (blockIdx.x == 0)
        for (int r = threadIdx.x; r < a.rows; r += kThreads)
            if (ids_of<OWN>(a)[r] >= a.vocab) atomicExch(a.status, PSSA_B200_ERR_TOKEN);
}

// ---- host side
inline StepCommon step_common(const pssa_b200_ctx* ctx, const StepLaunch& p) {
    StepCommon a{};
    a.rows = p.rows, a.depth = (int)p.depth, a.d = p.d, a.k = p.k, a.cap = p.cap, a.nc = p.nc;
    a.off_b = p.off_b, a.off_q = p.off_q, a.off_gate = p.off_gate, a.off_act = p.off_act, a.vocab = p.vocab;
    a.ssm_scale = p.ssm_scale, a.head_scale = p.head_scale, a.tau = p.tau;
    a.embed = p.embed, a.ids = p.ids, a.slots = p.slots, a.unembed = (const __nv_bfloat16*)p.unembed, a.carry_stride = p.carry_stride;
    a.feat_a = p.feat_a, a.feat_b = p.feat_b, a.proj = p.proj, a.y = p.y, a.qpart = p.qpart, a.ssq = p.ssq, a.inv = p.inv, a.logits = p.logits;
    a.x = (__nv_bfloat16*)p.x, a.w = (__nv_bfloat16*)p.w, a.z = (__nv_bfloat16*)p.z, a.act = (__nv_bfloat16*)p.act;
    a.status = ctx->status_dev;
    if (!p.ids)
        for (int r = 0; r < p.rows && r < kStepOwnRows; ++r) a.own_ids[r] = p.host_ids[r], a.own_slots[r] = p.host_slots[r];
    return a;
}
inline StepBlock step_block(const StepLaunch::Block& s) {
    return {(const __nv_bfloat16*)s.wcat, (const __nv_bfloat16*)s.wqh, (const __nv_bfloat16*)s.vp, (const __nv_bfloat16*)s.w1,
            (const __nv_bfloat16*)s.w2,   s.rates, s.gamma, s.beta, s.keys_t, s.norm_sq, s.state, s.res_scale, s.count};
}

}  // namespace step
}  // namespace pssa
