// Host arrays in and out of the entry points that take host pointers.
//
// A call's inputs lie side by side in one device region and go over in one copy from pinned memory, its outputs come back
// the same way; the device region and the pinned buffer belong to the context and are kept from call to call up to a bound.
// A cudaMalloc / cudaFree pair per array and a pageable copy each was most of such a call: 128 x 192 x 192 product 97 -> 60 us,
// memory stage of 128 tokens 537 -> 314 us. Large outputs are copied out of the pinned buffer by a few threads while the
// next piece is on its way (one thread moves 18 GB/s, the link 52).
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>

#include "context.hpp"

namespace pssa {

class HostCall {
  public:
    explicit HostCall(pssa_b200_ctx* ctx) : ctx_(ctx) {}
    ~HostCall();
    HostCall(const HostCall&) = delete;
    HostCall& operator=(const HostCall&) = delete;
    // declare every array first; each returns its index. `host` may be null: a device array without a host side
    int in(const void* host, size_t bytes) { return add(host, nullptr, bytes); }
    int out(void* host, size_t bytes) { return add(nullptr, host, bytes); }
    int inout(const void* src, void* dst, size_t bytes) { return add(src, dst, bytes); }
    int scratch(size_t bytes) { return add(nullptr, nullptr, bytes); }
    int32_t upload();  // allocates the device region and enqueues the inputs
    float* f(int i) const { return reinterpret_cast<float*>(base_ + arrays_[i].off); }
    // Waits for the stream and brings the outputs back. With `what` the host arrays stay untouched when a bounded device-side
    // wait has expired, whose status and `what` then become the error.
    int32_t download(const char* what);

  private:
    struct Array {
        const void* src;
        void* dst;
        size_t bytes, off;
    };
    int add(const void* src, void* dst, size_t bytes) {
        arrays_.push_back({src, dst, bytes, 0});
        return (int)arrays_.size() - 1;
    }
    pssa_b200_ctx* ctx_;
    std::vector<Array> arrays_;
    char* base_ = nullptr;
    bool own_ = false;  // the region is this call's alone (above the kept bound)
};

// device -> host through the context's pinned buffer, in stream order; waits for the stream
int32_t copy_to_host(pssa_b200_ctx* ctx, void* dst, const void* src_dev, size_t bytes);
// The same to several arrays, through pinned memory where that pays: `to` in the order of `off`, the places in `src_dev`.
struct HostSpan {
    char* dst;
    size_t off, bytes;
};
int32_t copy_spans_to_host(pssa_b200_ctx* ctx, const void* src_dev, size_t bytes, const std::vector<HostSpan>& to);
// host -> device through the context's pinned buffer (see want_pinned); waits for the stream
int32_t copy_to_device(pssa_b200_ctx* ctx, void* dst_dev, const void* src, size_t bytes);
// a context's first pinned buffer, and its largest: longer transfers go through it in windows
constexpr size_t kPinnedMin = (size_t)256 << 10, kPinnedMax = (size_t)4 << 20;
// pinned host memory of the context, at least `bytes`, valid until the next call; waits for the stream when it has to grow, and for
// a copy that pinned_send left behind
int32_t pinned_reserve(pssa_b200_ctx* ctx, size_t bytes);
// Whether words of a model's host call should pass through pinned memory: yes where the buffer holds them; otherwise a context's first
// such call goes without and the next one pins it. Pinning a process's first buffer takes 0.9 to 2.6 ms (3 us while another one is
// pinned: then at once), the largest 1.5 to 4.5 ms, and saves a call 10 us at 256 KB and 150 at 4 MB: a program that makes one call never
// gets it back (the small model's first step 2.8 ms with it and 0.2 without), one that makes many pays once.
bool want_pinned(pssa_b200_ctx* ctx, size_t bytes, bool out);
// enqueues the copy of `bytes` at `off` of the pinned buffer to the device and returns
int32_t pinned_send(pssa_b200_ctx* ctx, void* dst_dev, size_t off, size_t bytes);
void host_io_create();  // once per context
void host_io_destroy(pssa_b200_ctx* ctx);

}  // namespace pssa
