// Host arrays in and out of the entry points that take host pointers: see host_io.hpp.
#include "host_io.hpp"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>
#include <utility>

namespace pssa {
namespace {

constexpr size_t kKeepDevice = (size_t)256 << 20;  // device region kept between calls, at most
constexpr size_t kThreadsFrom = (size_t)1 << 20;   // outputs from here on are copied by several threads
constexpr size_t kPinnedKept = 4;                  // pinned buffers kept for the next context, while any context lives
constexpr size_t kPinnedInputs = (size_t)2 << 20;  // above this the driver's own pipelined pageable copy is as fast
constexpr size_t kPiece = (size_t)512 << 10;       // one device copy of a large transfer
constexpr size_t kShare = (size_t)128 << 10;       // what a copying thread takes at a time
constexpr int kHelpers = 3;

struct Span {  // one piece of a host array and where it lies in the pinned window
    char* dst;
    const char* src;
    size_t bytes;
};

}  // namespace

// Helper threads, one set for the process, started with the first large output. A context that finds them at work for
// another one copies alone. A job is a list of spans of which the first `ready` may be copied; the calling thread
// raises `ready` as the device delivers and takes spans itself.
struct CopyPool {
    std::mutex m;
    std::condition_variable wake;
    std::mutex busy;  // held for the length of a job
    bool started = false;
    const Span* spans = nullptr;
    size_t total = 0;
    std::atomic<size_t> ready{0}, next{0}, done{0};
    std::atomic<int> inside{0};
    uint64_t job = 0;

    void take(const Span* s, size_t n) {  // copies spans until all are taken
        for (;;) {
            size_t i = next.load(std::memory_order_relaxed);
            if (i >= n) return;
            if (i >= ready.load(std::memory_order_acquire)) {
                std::this_thread::yield();
                continue;
            }
            if (!next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed)) continue;
            std::memcpy(s[i].dst, s[i].src, s[i].bytes);
            done.fetch_add(1, std::memory_order_release);
        }
    }
    void run() {
        uint64_t seen = 0;
        for (;;) {
            const Span* s;
            size_t n;
            {
                std::unique_lock<std::mutex> l(m);
                wake.wait(l, [&] { return job != seen; });
                seen = job, s = spans, n = total;
                if (!s) continue;
                inside.fetch_add(1);
            }
            take(s, n);
            inside.fetch_sub(1);
        }
    }
    void begin(const Span* s, size_t n) {
        std::lock_guard<std::mutex> l(m);
        if (!started)
            for (int i = 0; i < kHelpers; ++i) std::thread([this] { run(); }).detach();
        started = true;
        ready.store(0), next.store(0), done.store(0);
        spans = s, total = n, ++job;
        wake.notify_all();
    }
    void raise(size_t upto) { ready.store(upto, std::memory_order_release); }
    // one span by the calling thread, if one is ready and not taken
    bool help(const Span* s) {
        size_t i = next.load(std::memory_order_relaxed);
        if (i >= ready.load(std::memory_order_acquire) || !next.compare_exchange_strong(i, i + 1)) return false;
        std::memcpy(s[i].dst, s[i].src, s[i].bytes);
        done.fetch_add(1, std::memory_order_release);
        return true;
    }
    void end(const Span* s, size_t n, bool finish) {
        if (!finish) next.store(n), ready.store(n);  // a failed transfer: nobody takes another span
        else take(s, n);
        if (finish)
            while (done.load(std::memory_order_acquire) < n) std::this_thread::yield();
        {
            std::lock_guard<std::mutex> l(m);
            spans = nullptr;
        }
        while (inside.load() != 0) std::this_thread::yield();  // the span list is about to go away
    }
};

namespace {
CopyPool& copy_pool() {
    static CopyPool* pool = new CopyPool();  // never destroyed: its threads wait in it until the process ends
    return *pool;
}
// Pinned buffers of contexts that are gone: pinning costs milliseconds, and a program may open many contexts. At most
// kPinnedKept buffers of kPinnedMax, all freed with the last context.
struct PinnedCache {
    std::mutex m;
    std::vector<std::pair<char*, size_t>> kept;
    size_t contexts = 0, pinned = 0;  // buffers that are pinned now, kept or in use
};
PinnedCache& pinned_cache() {
    static PinnedCache* c = new PinnedCache();
    return *c;
}
void pinned_give_back(char* p, size_t bytes) {
    PinnedCache& c = pinned_cache();
    std::lock_guard<std::mutex> l(c.m);
    if (bytes <= kPinnedMax && c.contexts > 0 && c.kept.size() < kPinnedKept) c.kept.push_back({p, bytes});
    else cudaFreeHost(p), --c.pinned;
}
}  // namespace

int32_t pinned_reserve(pssa_b200_ctx* ctx, size_t bytes) {
    if (ctx->staged) {
        PSSA_CUDA(ctx, cudaEventSynchronize(ctx->staged_ev));
        ctx->staged = false;
    }
    if (bytes <= ctx->pinned_bytes) return PSSA_B200_OK;
    if (ctx->pinned) {
        PSSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        pinned_give_back(ctx->pinned, ctx->pinned_bytes);
        ctx->pinned = nullptr, ctx->pinned_bytes = 0;
    }
    {
        PinnedCache& c = pinned_cache();
        std::lock_guard<std::mutex> l(c.m);
        for (auto& k : c.kept)
            if (k.second >= bytes) {
                ctx->pinned = k.first, ctx->pinned_bytes = k.second;
                k = c.kept.back();
                c.kept.pop_back();
                return PSSA_B200_OK;
            }
    }
    const size_t want = bytes <= kPinnedMin ? kPinnedMin : bytes <= kPinnedMax ? kPinnedMax : (bytes + 4095) & ~size_t(4095);
    cudaError_t e = cudaHostAlloc((void**)&ctx->pinned, want, cudaHostAllocPortable);
    if (e != cudaSuccess) {
        ctx->pinned = nullptr;
        return cuda_fail(ctx, e, "pinned staging allocation");
    }
    ctx->pinned_bytes = want;
    PinnedCache& c = pinned_cache();
    std::lock_guard<std::mutex> l(c.m);
    ++c.pinned;
    return PSSA_B200_OK;
}

bool want_pinned(pssa_b200_ctx* ctx, size_t bytes, bool out) {
    if (bytes <= ctx->pinned_bytes) return true;
    if (bytes > kPinnedMax) return false;
    {
        PinnedCache& c = pinned_cache();
        std::lock_guard<std::mutex> l(c.m);
        if (bytes <= kPinnedMin && c.pinned > 0) return true;
        for (auto& k : c.kept)
            if (k.second >= bytes) return true;
    }
    return std::exchange(ctx->asked[out][bytes > kPinnedMin], true);
}

int32_t pinned_send(pssa_b200_ctx* ctx, void* dst_dev, size_t off, size_t bytes) {
    if (!ctx->staged_ev) PSSA_CUDA(ctx, cudaEventCreateWithFlags(&ctx->staged_ev, cudaEventDisableTiming));
    PSSA_CUDA(ctx, cudaMemcpyAsync(dst_dev, ctx->pinned + off, bytes, cudaMemcpyHostToDevice, ctx->stream));
    PSSA_CUDA(ctx, cudaEventRecord(ctx->staged_ev, ctx->stream));
    ctx->staged = true;
    return PSSA_B200_OK;
}

// Copies `bytes` from consecutive device memory at `src` to the arrays in `to` (consecutive in the device order, with gaps).
namespace {
int32_t scatter(pssa_b200_ctx* ctx, const char* src, size_t bytes, const std::vector<HostSpan>& to, size_t window = kPinnedMax) {
    cudaStream_t st = ctx->stream;
    for (size_t w0 = 0; w0 < bytes; w0 += window) {
        const size_t wn = std::min(window, bytes - w0);
        int32_t rc = pinned_reserve(ctx, wn);
        if (rc) return rc;
        if (wn < kThreadsFrom) {
            PSSA_CUDA(ctx, cudaMemcpyAsync(ctx->pinned, src + w0, wn, cudaMemcpyDeviceToHost, st));
            PSSA_CUDA(ctx, cudaStreamSynchronize(st));
            for (const HostSpan& t : to) {
                const size_t a = std::max(t.off, w0), b = std::min(t.off + t.bytes, w0 + wn);
                if (a < b) std::memcpy(t.dst + (a - t.off), ctx->pinned + (a - w0), b - a);
            }
            continue;
        }
        const size_t pieces = (wn + kPiece - 1) / kPiece;
        while (ctx->io_events.size() < pieces) {
            cudaEvent_t e;
            PSSA_CUDA(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            ctx->io_events.push_back(e);
        }
        for (size_t i = 0; i < pieces; ++i) {
            const size_t a = i * kPiece, n = std::min(kPiece, wn - a);
            PSSA_CUDA(ctx, cudaMemcpyAsync(ctx->pinned + a, src + w0 + a, n, cudaMemcpyDeviceToHost, st));
            PSSA_CUDA(ctx, cudaEventRecord(ctx->io_events[i], st));
        }
        // spans in device order; upto[i] = how many of them piece i completes
        std::vector<Span> spans;
        std::vector<size_t> upto(pieces);
        size_t t = 0;
        for (size_t i = 0; i < pieces; ++i) {
            const size_t p0 = w0 + i * kPiece, p1 = std::min(w0 + wn, p0 + kPiece);
            while (t < to.size() && to[t].off + to[t].bytes <= p0) ++t;
            for (size_t u = t; u < to.size() && to[u].off < p1; ++u)
                for (size_t a = std::max(to[u].off, p0); a < std::min(to[u].off + to[u].bytes, p1); a += kShare) {
                    const size_t n = std::min({kShare, to[u].off + to[u].bytes - a, p1 - a});
                    spans.push_back({to[u].dst + (a - to[u].off), ctx->pinned + (a - w0), n});
                }
            upto[i] = spans.size();
        }
        // The kernels in front of the first piece may take long: only this thread waits for them, and the helpers stay free for
        // other contexts until there is something to copy.
        PSSA_CUDA(ctx, cudaEventSynchronize(ctx->io_events[0]));
        CopyPool& pool = copy_pool();
        std::unique_lock<std::mutex> mine(pool.busy, std::try_to_lock);
        if (!mine.owns_lock()) {
            size_t s = 0;
            for (size_t i = 0; i < pieces; ++i) {
                PSSA_CUDA(ctx, cudaEventSynchronize(ctx->io_events[i]));
                for (; s < upto[i]; ++s) std::memcpy(spans[s].dst, spans[s].src, spans[s].bytes);
            }
            continue;
        }
        pool.begin(spans.data(), spans.size());
        cudaError_t e = cudaSuccess;
        for (size_t i = 0; i < pieces && e == cudaSuccess; ++i) {
            while ((e = cudaEventQuery(ctx->io_events[i])) == cudaErrorNotReady)
                if (!pool.help(spans.data())) std::this_thread::yield();
            if (e == cudaSuccess) pool.raise(upto[i]);
        }
        (void)cudaGetLastError();  // "not ready" is no error
        pool.end(spans.data(), spans.size(), e == cudaSuccess);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "device to host copy");
    }
    return PSSA_B200_OK;
}
}  // namespace

int32_t copy_to_host(pssa_b200_ctx* ctx, void* dst, const void* src_dev, size_t bytes) {
    return scatter(ctx, (const char*)src_dev, bytes, {HostSpan{(char*)dst, 0, bytes}});
}

int32_t copy_spans_to_host(pssa_b200_ctx* ctx, const void* src_dev, size_t bytes, const std::vector<HostSpan>& to) {
    // Up to a megabyte through what the context has: a larger buffer would save 8 to 45 us a call and is not pinned for it. Us a decode step with
    // logits of 16384 words, rounds of 256 KB by one thread -> this: 32 lanes 322 -> 168, 64 582 -> 245, 256 2065 -> 740, 512 4020 -> 1370.
    // (The driver's own copy, for comparison: 224, 345, 1060, 2000; seven prompts into pages that nothing has touched 50 us slower than
    // two rounds.)
    if (bytes <= kThreadsFrom && ctx->pinned_bytes > 0) return scatter(ctx, (const char*)src_dev, bytes, to, ctx->pinned_bytes);
    if (bytes > kThreadsFrom && want_pinned(ctx, std::min(bytes, kPinnedMax), true)) return scatter(ctx, (const char*)src_dev, bytes, to);
    for (const HostSpan& t : to) PSSA_CUDA(ctx, cudaMemcpyAsync(t.dst, (const char*)src_dev + t.off, t.bytes, cudaMemcpyDeviceToHost, ctx->stream));
    PSSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return PSSA_B200_OK;
}

// In pieces, each copied into the pinned buffer by several threads while the one before is on the link: a carry of 2.4 MB in 75 us
// instead of the driver's 142 for pageable memory.
int32_t copy_to_device(pssa_b200_ctx* ctx, void* dst_dev, const void* src, size_t bytes) {
    if (!want_pinned(ctx, std::min(bytes, kPinnedMax), false)) {
        PSSA_CUDA(ctx, cudaMemcpyAsync(dst_dev, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
        PSSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        return PSSA_B200_OK;
    }
    for (size_t w0 = 0; w0 < bytes; w0 += kPinnedMax) {
        const size_t wn = std::min(kPinnedMax, bytes - w0);
        int32_t rc = pinned_reserve(ctx, wn);
        if (rc) return rc;
        CopyPool& pool = copy_pool();
        std::unique_lock<std::mutex> mine(pool.busy, std::defer_lock);
        const bool threads = wn >= kThreadsFrom && mine.try_lock();
        for (size_t a = 0; a < wn; a += kPiece) {
            const size_t n = std::min(kPiece, wn - a);
            if (threads) {
                std::vector<Span> spans;
                for (size_t b = 0; b < n; b += kShare) spans.push_back({ctx->pinned + a + b, (const char*)src + w0 + a + b, std::min(kShare, n - b)});
                pool.begin(spans.data(), spans.size());
                pool.raise(spans.size());
                pool.end(spans.data(), spans.size(), true);
            } else {
                std::memcpy(ctx->pinned + a, (const char*)src + w0 + a, n);
            }
            if ((rc = pinned_send(ctx, (char*)dst_dev + w0 + a, a, n))) return rc;
        }
    }
    PSSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return PSSA_B200_OK;
}

int32_t HostCall::upload() {
    // inputs first, then what goes both ways, then outputs: the inputs and the outputs are one contiguous range each
    size_t off = 0, in_end = 0;
    for (int pass = 0; pass < 4; ++pass) {
        for (Array& a : arrays_) {
            const int kind = a.src && !a.dst ? 0 : a.src ? 1 : a.dst ? 2 : 3;
            if (kind != pass) continue;
            a.off = off;
            off += arena_round(std::max<size_t>(a.bytes, 1));
        }
        if (pass == 1) in_end = off;
    }
    if (off <= kKeepDevice) {
        if (off > ctx_->io_bytes) {
            if (ctx_->io) {
                PSSA_CUDA(ctx_, cudaStreamSynchronize(ctx_->stream));
                PSSA_CUDA(ctx_, cudaFree(ctx_->io));
                ctx_->io = nullptr, ctx_->io_bytes = 0;
            }
            const size_t want = std::min(kKeepDevice, std::max<size_t>(off + off / 2, 1 << 20));
            cudaError_t e = cudaMalloc((void**)&ctx_->io, want);
            if (e != cudaSuccess) {
                ctx_->io = nullptr;
                return cuda_fail(ctx_, e, "host-array staging allocation");
            }
            ctx_->io_bytes = want;
        }
        base_ = ctx_->io;
    } else {
        cudaError_t e = cudaMalloc((void**)&base_, off);
        if (e != cudaSuccess) {
            base_ = nullptr;
            return cuda_fail(ctx_, e, "host-array staging allocation");
        }
        own_ = true;
    }
    if (in_end == 0) return PSSA_B200_OK;
    if (in_end <= kPinnedInputs) {
        int32_t rc = pinned_reserve(ctx_, in_end);
        if (rc) return rc;
        for (const Array& a : arrays_)
            if (a.src) std::memcpy(ctx_->pinned + a.off, a.src, a.bytes);
        PSSA_CUDA(ctx_, cudaMemcpyAsync(base_, ctx_->pinned, in_end, cudaMemcpyHostToDevice, ctx_->stream));
    } else {
        for (const Array& a : arrays_)
            if (a.src) PSSA_CUDA(ctx_, cudaMemcpyAsync(base_ + a.off, a.src, a.bytes, cudaMemcpyHostToDevice, ctx_->stream));
    }
    return PSSA_B200_OK;
}

int32_t HostCall::download(const char* what) {
    std::vector<HostSpan> to;
    size_t lo = SIZE_MAX, hi = 0;
    for (const Array& a : arrays_)
        if (a.dst && a.bytes) lo = std::min(lo, a.off), hi = std::max(hi, a.off + a.bytes);
    if (lo == SIZE_MAX) lo = hi = 0;
    for (const Array& a : arrays_)
        if (a.dst && a.bytes) to.push_back({(char*)a.dst, a.off - lo, a.bytes});
    std::sort(to.begin(), to.end(), [](const HostSpan& x, const HostSpan& y) { return x.off < y.off; });
    // With `what`, the status word comes back too and outputs stay untouched when a bounded wait has expired. The pinned
    // buffer may still be the source of the inputs' copy: it is only written by copies behind that one on the stream.
    int32_t rc;
    const size_t bytes = hi - lo;
    const bool small = bytes + 64 <= kThreadsFrom;
    int status = 0;
    if ((rc = pinned_reserve(ctx_, small ? bytes + 64 : 64))) return rc;
    if (what) PSSA_CUDA(ctx_, cudaMemcpyAsync(ctx_->pinned, ctx_->status_dev, sizeof(int), cudaMemcpyDeviceToHost, ctx_->stream));
    if (small && bytes) PSSA_CUDA(ctx_, cudaMemcpyAsync(ctx_->pinned + 64, base_ + lo, bytes, cudaMemcpyDeviceToHost, ctx_->stream));
    if (what || small) PSSA_CUDA(ctx_, cudaStreamSynchronize(ctx_->stream));
    if (what) std::memcpy(&status, ctx_->pinned, sizeof(int));
    if (status != 0) {
        cudaMemsetAsync(ctx_->status_dev, 0, sizeof(int), ctx_->stream);
        return fail(ctx_, status, "%s: a bounded device-side wait expired", what);
    }
    if (!small) return scatter(ctx_, base_ + lo, bytes, to);
    for (const HostSpan& t : to) std::memcpy(t.dst, ctx_->pinned + 64 + t.off, t.bytes);
    return PSSA_B200_OK;
}

HostCall::~HostCall() {
    if (!base_) return;
    cudaStreamSynchronize(ctx_->stream);  // an early return may have left work on the region
    if (own_) cudaFree(base_);
}

void host_io_create() {
    PinnedCache& c = pinned_cache();
    std::lock_guard<std::mutex> l(c.m);
    ++c.contexts;
}

void host_io_destroy(pssa_b200_ctx* ctx) {
    for (cudaEvent_t e : ctx->io_events) cudaEventDestroy(e);
    ctx->io_events.clear();
    if (ctx->staged_ev) cudaEventDestroy(ctx->staged_ev);
    ctx->staged_ev = nullptr, ctx->staged = false;
    if (ctx->io) cudaFree(ctx->io);
    if (ctx->pinned) pinned_give_back(ctx->pinned, ctx->pinned_bytes);
    ctx->io = ctx->pinned = nullptr, ctx->io_bytes = ctx->pinned_bytes = 0;
    PinnedCache& c = pinned_cache();
    std::lock_guard<std::mutex> l(c.m);
    if (--c.contexts == 0) {
        for (auto& k : c.kept) cudaFreeHost(k.first);
        c.pinned -= c.kept.size();
        c.kept.clear();
    }
}

}  // namespace pssa
