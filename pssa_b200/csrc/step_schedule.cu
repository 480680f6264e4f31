// A decode step of many rows: the stages of step_decode.cu's kernel as a launch each, with the products on the tcgen05 path.
//
// Above a hundred rows or so a product is no longer the latency of its loads and the one kernel's mma.sync tiles fall behind
// the tensor cores; the stages between the products are the same device functions (step_stages.cuh). A stream's bits must be
// the same here and there, so the products keep the one kernel's order of every sum: K in eight segments, a chain of k = 16
// steps each, the segments added as ((s0+s1)+s2)+s3 + ((s4+s5)+s6)+s7. A segment is a TMEM accumulator of its own (eight of
// them are 256 columns with 32-wide tiles, all 512 with 64-wide ones), the epilogue adds them up; tcgen05.mma and mma.sync
// round a k = 16 step alike.
#include <cuda.h>
#include <cuda_bf16.h>

#include <type_traits>

#include "step_stages.cuh"
#include "tcgen05.cuh"

namespace pssa {
namespace {

using namespace step;
using namespace tc;

constexpr int kEpiWarps = 16;  // four per TMEM lane quadrant
constexpr int kReadRows = 4;  // rows of a CTA of the memory read: a key is loaded once for them

// A block of the 12-block, d 768 model at 256 streams, us a launch under a profiler: norm 7, x-side 13, SSM 25 (100 MB of carries, 16 at
// the copy rate), read 14, gated value read 10, MLP up 12, MLP down 16; the step 1107, as the block schedule that it replaces above
// 128 streams (1124), and 864 / 935 at 64 / 128 streams where the one kernel's 64-row mma.sync tiles took 959 / 1088. A launch of a
// few hundred rows is prologue, first trip to memory and epilogue: nothing is busy.

// The block's output rows; q sums of squares of 16 columns go to the next norm, at the last block the bf16 rows to the head.
struct PutFeature {
    static constexpr bool kReads = true;
    const StepCommon& a;
    const float* in;
    float* out;
    float scale;
    bool last;
    __device__ __forceinline__ int cols() const { return a.d; }
    __device__ __forceinline__ Pre fetch(int col, int row) const { return feature_fetch(a, in, col, row); }
    __device__ __forceinline__ float value(int, float v, Pre p) const { return feature_value(p, in != nullptr, scale, v); }
    __device__ __forceinline__ void store(int col, int row, float f) const {
        out[(size_t)row * a.d + col] = f;
        if (last) a.x[(size_t)row * a.d + col] = __float2bfloat16_rn(f);
    }
    __device__ __forceinline__ void store_squares(int col, int row, float q) const {
        if ((col & 15) == 0) a.ssq[(size_t)row * (a.d / 16) + col / 16] = q;
    }
};

// one lane of the warp, in a form the compiler knows to be one: behind `lane == 0` an MMA took 82 cycles to issue, behind this 52
__device__ __forceinline__ bool elected() {
    int r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void quad_sync(int quad) { asm volatile("bar.sync %0, 128;" ::"r"(quad + 1) : "memory"); }
// the same barrier, true where all four warps bring true: they go on, or leave, together
__device__ __forceinline__ bool quad_all(int quad, bool ok) {
    int all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %2, 0;\n\t"
        "bar.red.and.pred q, %1, 128, p;\n\t"
        "selp.b32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"(quad + 1), "r"((int)ok)
        : "memory");
    return all != 0;
}
// 32 lanes x 16 columns; the registers are valid after tcgen05.wait::ld
__device__ __forceinline__ void ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void wait_ld(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

template <int BN, int STAGES>
constexpr size_t product_smem() {
    return 1024 + (size_t)STAGES * (BM + BN) * BK * 2 + (2 * STAGES + 1) * 8 + 16 + 4 * 2 * 32 * 33 * 4;
}

// K in four runs of two segments; a box of operands is 64 wide, a run starts one of its own
constexpr int kRuns = 4;
struct Run {
    int first, boxes, seg0, seg1;  // first k; boxes; 32-wide steps of its two segments
};
__device__ __forceinline__ Run run_of(int k, int r) {
    int f0, c0, f1, c1;
    segment(k, 2 * r, f0, c0), segment(k, 2 * r + 1, f1, c1);
    return {f0 * 32, (c0 + c1 + 1) / 2, c0, c1};
}

// One 128 x BN tile per CTA: x [rows, .] times w [n, .]^T over the first k of K. Warp 0 loads, warp 1 issues: the four runs of K take
// turns, so that MMAs next to each other go to different accumulators (cycles for four boxes of 64, stamps in the issuing warp: 3800
// in K order, 2850 in turns, 2115 with an elected lane; the arrival of the boxes from L2, 38 B a cycle, is what is left). Warps 2 to 17: of a quadrant's four, two add up half of the segments for half of the columns each way,
// then each stores a quarter of the rows. What is read for an output is requested before the accumulators are waited for.
template <int BN, int STAGES, class Put>
__device__ __forceinline__ void product_tile(const CUtensorMap& map_x, const CUtensorMap& map_w, int n, int k, const Put& put) {
    constexpr uint32_t A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, TMEM_COLS = 8 * BN;
    static_assert(STAGES >= kRuns, "the boxes of a turn are waited for together");
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* const smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char *const smem_a = smem, *const smem_b = smem + STAGES * A_BYTES;
    uint64_t* const full_bar = reinterpret_cast<uint64_t*>(smem_b + STAGES * B_BYTES);
    uint64_t* const empty_bar = full_bar + STAGES;
    uint64_t* const acc_full = empty_bar + STAGES;
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    float* const stage = reinterpret_cast<float*>(tmem_slot + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = (n + BN - 1) / BN;
    const int m0 = (int)(blockIdx.x / n_tiles) * BM, n0 = (int)(blockIdx.x % n_tiles) * BN;
    const int rows = put.a.rows;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) mbar_init(&full_bar[s], 1), mbar_init(&empty_bar[s], 1);
        mbar_init(acc_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();
    pdl_wait();

    if (warp <= 1) {
        Run run[kRuns];
        int turns = 0;
#pragma unroll
        for (int r = 0; r < kRuns; ++r) run[r] = run_of(k, r), turns = max(turns, run[r].boxes);
        if (warp == 0 && elected()) {
            bool ok = true;
            int it = 0;
            for (int b = 0; b < turns; ++b)
#pragma unroll
                for (int r = 0; r < kRuns; ++r) {
                    if (b >= run[r].boxes || !ok) continue;
                    const int s = it % STAGES;
                    if (it >= STAGES && !mbar_wait(&empty_bar[s], (it / STAGES - 1) & 1)) {
                        atomicExch(put.a.status, PSSA_B200_ERR_TIMEOUT);
                        ok = false;
                        continue;
                    }
                    mbar_expect_tx(&full_bar[s], A_BYTES + B_BYTES);
                    tma_load_2d(smem_a + s * A_BYTES, &map_x, &full_bar[s], run[r].first + b * BK, m0);
                    tma_load_2d(smem_b + s * B_BYTES, &map_w, &full_bar[s], run[r].first + b * BK, n0);
                    ++it;
                }
        } else if (warp == 1 && elected()) {
            constexpr uint32_t idesc = umma_idesc_bf16(BM, BN);
            bool ok = true;
            int it = 0;
            for (int b = 0; b < turns && ok; ++b) {
                uint64_t da[kRuns], db[kRuns];
                const int it0 = it;
#pragma unroll
                for (int r = 0; r < kRuns; ++r) {
                    if (b >= run[r].boxes || !ok) continue;
                    const int s = it % STAGES;
                    ok = mbar_wait(&full_bar[s], (it / STAGES) & 1);
                    da[r] = umma_desc_sw128(smem_u32(smem_a + s * A_BYTES)), db[r] = umma_desc_sw128(smem_u32(smem_b + s * B_BYTES));
                    ++it;
                }
                if (!ok) {
                    atomicExch(put.a.status, PSSA_B200_ERR_TIMEOUT);
                    break;
                }
                tcgen05_fence_after();
#pragma unroll
                for (int j = 0; j < BK / UMMA_K; ++j)
#pragma unroll
                    for (int r = 0; r < kRuns; ++r) {
                        // step `at` of the run, in k = 16 steps: of its first segment or its second one
                        const int at = b * 4 + j, second = 2 * run[r].seg0;
                        if (at >= second + 2 * run[r].seg1) continue;
                        tcgen05_mma_bf16(tmem_base + (2 * r + (at >= second)) * BN, da[r] + (uint64_t)(j * 2), db[r] + (uint64_t)(j * 2), idesc,
                                         at != 0 && at != second);
                    }
                for (int i = it0; i < it; ++i) tcgen05_commit(&empty_bar[i % STAGES]);
            }
            tcgen05_commit(acc_full);
        }
    } else {
        const int quad = warp & 3, part = (warp - 2) >> 2, half = part & 1, c16 = (part >> 1) * 16, rbase = m0 + quad * 32;
        const bool live = rbase < rows;
        float* const stg = stage + quad * (2 * 32 * 33);
        bool ready = false;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
            const int col = n0 + c0 + lane, first = rbase + part * 8;
            const bool in = col < put.cols();
            Pre pre[Put::kReads ? 8 : 1];
            if constexpr (Put::kReads) {
#pragma unroll
                for (int i = 0; i < 8; ++i) pre[i] = put.fetch(min(col, put.cols() - 1), min(first + i, rows - 1));
            }
            if (!ready && !quad_all(quad, mbar_wait(acc_full, 0))) {
                if (lane == 0) atomicExch(put.a.status, PSSA_B200_ERR_TIMEOUT);
                break;
            }
            ready = true;
            if (!live) break;
            tcgen05_fence_after();
            uint32_t v[4][16];
#pragma unroll
            for (int u = 0; u < 4; ++u) ld_32x16(tmem_base + (half * 4 + u) * BN + c0 + c16 + ((uint32_t)(quad * 32) << 16), v[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u) wait_ld(v[u]);
            float sum[16];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                int at, count;
                segment(k, half * 4 + u, at, count);  // an empty segment's accumulator was never written
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float x = count > 0 ? __uint_as_float(v[u][j]) : 0.0f;
                    sum[j] = u == 0 ? x : sum[j] + x;
                }
            }
            // a thread has a row of 16 columns: transposed, so that a warp's loads and stores are whole lines
#pragma unroll
            for (int j = 0; j < 16; ++j) stg[(half * 32 + lane) * 33 + c16 + j] = sum[j];
            quad_sync(quad);
            const float* const mine = stg + part * 8 * 33 + lane;
            float f[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = mine[i * 33] + mine[(32 + i) * 33];
            if constexpr (Put::kReads) {
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = put.value(col, f[i], pre[i]);
            } else {
                put.values(col, f);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (first + i < rows && in) put.store(col, first + i, f[i]);
            if constexpr (std::is_same<Put, PutFeature>::value) {
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = squares16(f[i]);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (first + i < rows && in) put.store_squares(col, first + i, f[i]);
            }
            if (c0 + 32 < BN) quad_sync(quad);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

template <int BN, int STAGES, class Put>
__global__ void __launch_bounds__(64 + 32 * kEpiWarps, 1) step_product_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                              const __grid_constant__ CUtensorMap map_w,
                                                                              const __grid_constant__ StepCommon a, int n, int k) {
    product_tile<BN, STAGES>(map_x, map_w, n, k, Put{a});
}
template <int BN, int STAGES>
__global__ void __launch_bounds__(64 + 32 * kEpiWarps, 1) step_feature_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                              const __grid_constant__ CUtensorMap map_w,
                                                                              const __grid_constant__ StepCommon a, int k, const float* in,
                                                                              float* out, float scale, bool last) {
    product_tile<BN, STAGES>(map_x, map_w, a.d, k, PutFeature{a, in, out, scale, last});
}

__global__ void __launch_bounds__(kThreads) step_norm_kernel(const __grid_constant__ StepCommon a, const __grid_constant__ StepBlock b,
                                                             const unsigned* ids, const float* in) {
    pdl_trigger();
    pdl_wait();
    if (ids) check_ids(a);
    norm_stage(a, b, Features{a.embed, ids, in, a.d, a.vocab});
}
// CTAs to an SM: with few states two of 128 registers instead of one with three rows in flight a warp (32 states, 4 blocks of d 384,
// 256 / 512 streams: 256 -> 247, 305 -> 284 us a step), with 64 the rows' carries need the registers
constexpr int ssm_ctas(int nv) { return nv > 2 ? 1 : 2; }
template <int NV>
__global__ void __launch_bounds__(kThreads, ssm_ctas(NV)) step_ssm_kernel(const __grid_constant__ StepCommon a, const __grid_constant__ StepBlock b,
                                                               const unsigned* ids, const float* in) {
    pdl_trigger();
    pdl_wait();
    SsmAhead<NV, (NV > 2 ? 3 : 2)> sa;
    ssm_request(a, b, sa);
    ssm_stage(a, Features{a.embed, ids, in, a.d, a.vocab}, sa, b.state);
}
__global__ void __launch_bounds__(kThreads) step_read_kernel(const __grid_constant__ StepCommon a, const __grid_constant__ StepBlock b) {
    __shared__ __align__(16) float sm[read_floats(kReadRows)];
    pdl_trigger();
    pdl_wait();
    read_stage<kReadRows>(a, b, sm, nullptr);
}

// x [rows, ldx] times w [n, ldw]^T over the first k columns
template <int BN, int STAGES, class Launch>
int32_t with_maps(pssa_b200_ctx* ctx, const void* x, size_t ldx, const void* w, size_t ldw, int rows, int n, const void* kern, PerDeviceOnce& attr,
                  const char* name, Launch&& launch) {
    CUtensorMap map_x, map_w;
    int32_t rc;
    if ((rc = make_map(ctx, &map_x, x, (size_t)rows, ldx, BM)) || (rc = make_map(ctx, &map_w, w, (size_t)n, ldw, BN))) return rc;
    if (attr.need(ctx->device)) {
        PSSA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)product_smem<BN, STAGES>()));
        attr.done(ctx->device);
    }
    const unsigned grid = (unsigned)(((rows + BM - 1) / BM) * ((n + BN - 1) / BN));
    PSSA_CUDA(ctx, launch(dim3(grid), map_x, map_w));
    return after_launch(ctx, name);
}
template <int BN, int STAGES, class Put>
int32_t product(pssa_b200_ctx* ctx, const StepCommon& a, const void* x, size_t ldx, const void* w, size_t ldw, int n, int k, const char* name) {
    static PerDeviceOnce attr;
    auto kern = step_product_kernel<BN, STAGES, Put>;
    return with_maps<BN, STAGES>(ctx, x, ldx, w, ldw, a.rows, n, (const void*)kern, attr, name, [&](dim3 grid, const CUtensorMap& mx, const CUtensorMap& mw) {
        return launch_dependent(kern, grid, dim3(64 + 32 * kEpiWarps), product_smem<BN, STAGES>(), ctx->stream, mx, mw, a, n, k);
    });
}
template <int BN, int STAGES>
int32_t feature_product(pssa_b200_ctx* ctx, const StepCommon& a, const void* x, size_t ldx, const void* w, size_t ldw, int k, const float* in, float* out,
                        float scale, bool last) {
    static PerDeviceOnce attr;
    auto kern = step_feature_kernel<BN, STAGES>;
    return with_maps<BN, STAGES>(ctx, x, ldx, w, ldw, a.rows, a.d, (const void*)kern, attr, "step_product_kernel[MLP down + residuals]",
                                 [&](dim3 grid, const CUtensorMap& mx, const CUtensorMap& mw) {
        return launch_dependent(kern, grid, dim3(64 + 32 * kEpiWarps), product_smem<BN, STAGES>(), ctx->stream, mx, mw, a, k, in, out, scale, last);
    });
}
// 32-wide tiles while they fit in one wave, 64-wide ones beyond
bool narrow(const pssa_b200_ctx* ctx, const StepCommon& a, int n) { return ((a.rows + BM - 1) / BM) * ((n + 31) / 32) <= ctx->sm_count; }

}  // namespace

int32_t launch_step_schedule(pssa_b200_ctx* ctx, const StepLaunch& p) {
    const StepCommon a = step_common(ctx, p);
    const int d = a.d, s = p.s;
    const unsigned sms = (unsigned)ctx->sm_count;
    const size_t ldw = 3 * (size_t)a.cap, ldz = (size_t)d + 64, lda = 2 * (size_t)d + 64;
    const float* in = nullptr;
    int32_t rc;
    for (size_t l = 0; l < p.depth; ++l) {
        const StepBlock b = step_block(p.blocks[l]);
        float* const out = in == a.feat_a ? a.feat_b : a.feat_a;
        const unsigned* const ids = l == 0 ? a.ids : nullptr;
        // Started early its few CTAs crowd on the SMs that the product before leaves first, at every width and number of rows: us a step as a
        // graph, early -> in order, 4 blocks: d 64 x 256 rows 193 -> 177, d 192 x 200 219 -> 204, d 384 x 512 345 -> 331, d 768 x 256 374 -> 356,
        // x 2048 988 -> 968. The first block's follows another call: early saves 2 us of an eager step of 200 to 512 rows and costs 1 to 3
        // with fewer rows or as a graph; of 1024 rows and more of wide models it costs 3 to 7.
        const dim3 norm_grid(((unsigned)a.rows + kWarps - 1) / kWarps);
        if (l > 0 || d > 256) step_norm_kernel<<<norm_grid, kThreads, 0, ctx->stream>>>(a, b, ids, in);
        else PSSA_CUDA(ctx, launch_dependent(step_norm_kernel, norm_grid, dim3(kThreads), 0, ctx->stream, a, b, ids, in));
        if ((rc = after_launch(ctx, "step_norm_kernel"))) return rc;
        if ((rc = narrow(ctx, a, a.nc) ? product<32, 9, PutXside>(ctx, a, a.x, d, b.wcat, d, a.nc, d, "step_product_kernel[x-side]")
                                       : product<64, 7, PutXside>(ctx, a, a.x, d, b.wcat, d, a.nc, d, "step_product_kernel[x-side]")))
            return rc;
        auto ssm = s == 16 ? step_ssm_kernel<1> : s == 32 ? step_ssm_kernel<2> : step_ssm_kernel<4>;
        PSSA_CUDA(ctx, launch_dependent(ssm, dim3(sms * ssm_ctas(s / 16)), dim3(kThreads), 0, ctx->stream, a, b, ids, in));
        if ((rc = after_launch(ctx, "step_ssm_kernel"))) return rc;
        PSSA_CUDA(ctx, launch_dependent(step_read_kernel, dim3(((unsigned)a.rows + kReadRows - 1) / kReadRows), dim3(kThreads), 0, ctx->stream, a, b));
        if ((rc = after_launch(ctx, "step_read_kernel"))) return rc;
        if ((rc = narrow(ctx, a, d) ? product<32, 9, PutGated>(ctx, a, a.w, ldw, b.vp, ldw, d, a.cap, "step_product_kernel[gated value read]")
                                    : product<64, 7, PutGated>(ctx, a, a.w, ldw, b.vp, ldw, d, a.cap, "step_product_kernel[gated value read]")))
            return rc;
        if ((rc = narrow(ctx, a, 2 * d) ? product<32, 9, PutHidden>(ctx, a, a.z, ldz, b.w1, ldz, 2 * d, (int)ldz, "step_product_kernel[MLP up]")
                                        : product<64, 7, PutHidden>(ctx, a, a.z, ldz, b.w1, ldz, 2 * d, (int)ldz, "step_product_kernel[MLP up]")))
            return rc;
        const bool last = l + 1 == p.depth;
        if ((rc = narrow(ctx, a, d) ? feature_product<32, 9>(ctx, a, a.act, lda, b.w2, lda, (int)lda, in, out, b.res_scale, last)
                                    : feature_product<64, 7>(ctx, a, a.act, lda, b.w2, lda, (int)lda, in, out, b.res_scale, last)))
            return rc;
        in = out;
    }
    if (!a.logits) return PSSA_B200_OK;
    return product<64, 7, PutLogit>(ctx, a, a.x, d, a.unembed, d, (int)a.vocab, d, "step_product_kernel[head]");
}

}  // namespace pssa
