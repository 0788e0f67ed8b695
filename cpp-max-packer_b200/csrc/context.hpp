// Context: device, stream, device-memory arena, twiddle tables and the
// host-side stop/deadline poll shared by every entry point.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <initializer_list>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/spk_b200.h"
#include "common.cuh"

struct spk_context {
    int device {};
    std::uint64_t cap_bytes {};
    cudaStream_t stream {};
    std::atomic<std::uint64_t> launches { 0 };
    std::uint64_t bytes_in_use {};
    struct Buffer {
        void* ptr {};
        std::size_t bytes {};
        std::size_t counted {};  // against the cap
    };
    std::map<std::string, Buffer> device_buffers;
    std::map<std::string, Buffer> host_buffers;  // pinned staging
    // Device blocks given back by sessions for the next one to take
    // (take_block, give_block): at most kKeptBytes of them, within the cap, and
    // only as long as nothing else on the context needs the memory.
    static constexpr std::size_t kKeptBytes = 256ULL << 20;
    std::vector<Buffer> kept_blocks;
    std::vector<cudaEvent_t> copy_events;  // one per pinned copy slot (host_copy.cu)
    std::map<std::pair<int, int>, void*> twiddles;  // (sizeof scalar, L) -> table
    void* session {};                              // placement session (engine.cpp)
    bool profiling {};
    static constexpr int kPasses = 4;  // A, B1, B2, merge + exact
    std::uint64_t pass_launches[kPasses] {};
    double pass_ms[kPasses] {};
    double pass_bytes[kPasses] {};  // algorithmic bytes of the profiled launches
    std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> pending;  // (pass, events)
    const char* message { "" };  // static text of the last correlation failure on this context
};

namespace spk {

inline std::uint64_t kept_bytes(const spk_context* ctx)
{
    std::uint64_t sum = 0;
    for (const auto& b : ctx->kept_blocks) {
        sum += b.bytes;
    }
    return sum;
}

inline void release_kept_blocks(spk_context* ctx)
{
    for (const auto& b : ctx->kept_blocks) {
        cudaFree(b.ptr);
    }
    ctx->kept_blocks.clear();
}

// Device memory; the blocks kept for the next session go where there is none
// left.  nullptr on failure.
inline void* device_alloc(spk_context* ctx, std::size_t bytes)
{
    void* p {};
    if (cudaMalloc(&p, bytes ? bytes : 1) == cudaSuccess) {
        return p;
    }
    cudaGetLastError();
    if (ctx->kept_blocks.empty()) {
        return nullptr;
    }
    release_kept_blocks(ctx);
    if (cudaMalloc(&p, bytes ? bytes : 1) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

// Grows (never shrinks) a named device buffer; returns nullptr on failure.
// These buffers are what the context's cap is about; blocks kept for the next
// session take no room from it, and go where both would exceed it.  (An open
// session's kernel data, take_block, lies outside the cap, and so do `uncounted`
// bytes of a buffer: a call's bookkeeping.)
inline void* device_buffer(spk_context* ctx, const std::string& name, std::size_t bytes, int& status,
                           std::size_t uncounted = 0)
{
    auto& b = ctx->device_buffers[name];
    if (b.bytes >= bytes && b.ptr) {
        return b.ptr;
    }
    const std::size_t counted = bytes - uncounted;
    const std::uint64_t next = ctx->bytes_in_use - b.counted + counted;
    if (ctx->cap_bytes && next > ctx->cap_bytes) {
        status = kMemoryLimit;
        return nullptr;
    }
    if (ctx->cap_bytes && next + kept_bytes(ctx) > ctx->cap_bytes) {
        release_kept_blocks(ctx);
    }
    if (b.ptr) {
        cudaFree(b.ptr);
        ctx->bytes_in_use -= b.counted;
        b = {};
    }
    void* p = device_alloc(ctx, bytes);
    if (!p) {
        status = kAllocation;
        return nullptr;
    }
    b.ptr = p;
    b.bytes = bytes;
    b.counted = counted;
    ctx->bytes_in_use += counted;
    return p;
}

// What a capped context has left for a named buffer, its present size included.
inline std::uint64_t room_for(const spk_context* ctx, const char* name)
{
    const auto it = ctx->device_buffers.find(name);
    return ctx->cap_bytes - ctx->bytes_in_use + (it == ctx->device_buffers.end() ? 0 : it->second.counted);
}

// Gives named device buffers back.
inline void drop_buffers(spk_context* ctx, std::initializer_list<const char*> names)
{
    for (const char* name : names) {
        const auto it = ctx->device_buffers.find(name);
        if (it != ctx->device_buffers.end()) {
            cudaFree(it->second.ptr);
            ctx->bytes_in_use -= it->second.counted;
            ctx->device_buffers.erase(it);
        }
    }
}

// A device block of at least `bytes` (set to its size) for an object that gives
// it back with give_block; nullptr on failure.  Opening a session takes a few
// blocks; allocating and freeing them anew costs milliseconds each, and both
// wait for the device.  A kept block is reused only by work queued after its
// last use, on the same context's stream.
inline void* take_block(spk_context* ctx, std::size_t& bytes, int& status)
{
    auto best = ctx->kept_blocks.end();
    for (auto it = ctx->kept_blocks.begin(); it != ctx->kept_blocks.end(); ++it) {
        if (it->bytes >= bytes && it->bytes <= 2 * bytes + (16ULL << 20) &&
            (best == ctx->kept_blocks.end() || it->bytes < best->bytes)) {
            best = it;
        }
    }
    if (best != ctx->kept_blocks.end()) {
        void* p = best->ptr;
        bytes = best->bytes;
        ctx->kept_blocks.erase(best);
        return p;
    }
    void* p = device_alloc(ctx, bytes);
    if (!p) {
        status = kAllocation;
    }
    return p;
}

inline void give_block(spk_context* ctx, void* ptr, std::size_t bytes)
{
    const std::uint64_t kept = kept_bytes(ctx) + bytes;
    if (kept > spk_context::kKeptBytes || (ctx->cap_bytes && ctx->bytes_in_use + kept > ctx->cap_bytes)) {
        cudaFree(ptr);
        return;
    }
    ctx->kept_blocks.push_back({ ptr, bytes });
}

inline void* host_buffer(spk_context* ctx, const std::string& name, std::size_t bytes, int& status)
{
    auto& b = ctx->host_buffers[name];
    if (b.bytes >= bytes && b.ptr) {
        return b.ptr;
    }
    if (b.ptr) {
        cudaFreeHost(b.ptr);
        b = {};
    }
    void* p {};
    if (cudaMallocHost(&p, bytes ? bytes : 1) != cudaSuccess) {
        cudaGetLastError();
        status = kAllocation;
        return nullptr;
    }
    b.ptr = p;
    b.bytes = bytes;
    return p;
}

// Copies a host table into device memory and returns once the copy has
// landed.  A plain cudaMemcpy from pageable memory may return before its DMA
// reaches the device, and it runs on the legacy stream, which the context's
// non-blocking streams do not wait for: a kernel launched right after it
// could read the table half written.  Here the copy is ordered on the
// context's stream and that stream is drained before returning.
inline bool upload_table(spk_context* ctx, void* dst, const void* src, std::size_t bytes)
{
    if (cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return true;
}

// exp(-2 pi i m / L) for m < L, FP64-computed, stored as T.
template <typename T>
const cplx_t<T>* twiddle_table(spk_context* ctx, int L, int& status)
{
    const auto key = std::make_pair(static_cast<int>(sizeof(T)), L);
    auto it = ctx->twiddles.find(key);
    if (it != ctx->twiddles.end()) {
        return static_cast<const cplx_t<T>*>(it->second);
    }
    std::vector<cplx_t<T>> host(L);
    const double pi = 3.14159265358979323846264338327950288;
    for (int m = 0; m < L; ++m) {
        // Exact values at the quarter points keep the table symmetric.
        double c, s;
        if (4 * m % L == 0) {
            const int quadrant = 4 * m / L;
            c = quadrant == 0 ? 1.0 : quadrant == 2 ? -1.0 : 0.0;
            s = quadrant == 1 ? -1.0 : quadrant == 3 ? 1.0 : 0.0;
        }
        else {
            const double angle = -2.0 * pi * static_cast<double>(m) / static_cast<double>(L);
            c = std::cos(angle);
            s = std::sin(angle);
        }
        host[m].x = static_cast<T>(c);
        host[m].y = static_cast<T>(s);
    }
    void* p = device_alloc(ctx, sizeof(cplx_t<T>) * L);
    if (!p) {
        status = kAllocation;
        return nullptr;
    }
    if (!upload_table(ctx, p, host.data(), sizeof(cplx_t<T>) * L)) {
        cudaFree(p);
        status = kCuda;
        return nullptr;
    }
    ctx->twiddles[key] = p;
    return static_cast<const cplx_t<T>*>(p);
}

std::int64_t monotonic_ns();

// Records the reference's message for a failure site and returns its status.
inline int fail(spk_context* ctx, int status, const char* message)
{
    ctx->message = message;
    return status;
}

// A failing status whose site left no message gets the reference's wording
// for its code (correlation.cpp:268-270,587) or the library's own.
inline int finish(spk_context* ctx, int status)
{
    if (status && ctx && !*ctx->message) {
        switch (status) {
        case kCancelled:
        case kDeadline: ctx->message = "Correlation interrupted."; break;
        case kAllocation: ctx->message = "Correlation allocation failed."; break;
        case kMemoryLimit: ctx->message = "Correlation buffers and FFT workspace exceed their memory limit."; break;
        case kCuda: ctx->message = "CUDA runtime call failed."; break;
        case kInvalidArgument: ctx->message = "Invalid argument."; break;
        default: break;
        }
    }
    return status;
}

// The reference polls stop first, then the deadline (operation_control.hpp:33-42).
inline int poll(const spk_control* control)
{
    if (!control) {
        return kOk;
    }
    if (control->stop_word && *control->stop_word) {
        return kCancelled;
    }
    if (control->deadline_ns && monotonic_ns() >= control->deadline_ns) {
        return kDeadline;
    }
    return kOk;
}

// Brackets one pass launch with events when profiling is on.
inline std::pair<cudaEvent_t, cudaEvent_t> pass_begin(spk_context* ctx)
{
    std::pair<cudaEvent_t, cudaEvent_t> ev {};
    if (ctx->profiling) {
        cudaEventCreate(&ev.first);
        cudaEventCreate(&ev.second);
        cudaEventRecord(ev.first, ctx->stream);
    }
    return ev;
}
inline void pass_end(spk_context* ctx, int pass, std::pair<cudaEvent_t, cudaEvent_t> ev, double bytes = 0.0)
{
    if (ctx->profiling && ev.first) {
        cudaEventRecord(ev.second, ctx->stream);
        ctx->pending.push_back({ pass, ev });
        ctx->pass_bytes[pass] += bytes;
    }
}
inline void pass_collect(spk_context* ctx)
{
    for (auto& [pass, ev] : ctx->pending) {
        float ms = 0.f;
        if (cudaEventSynchronize(ev.second) == cudaSuccess && cudaEventElapsedTime(&ms, ev.first, ev.second) ==
                                                                 cudaSuccess) {
            ctx->pass_ms[pass] += ms;
            ctx->pass_launches[pass] += 1;
        }
        cudaEventDestroy(ev.first);
        cudaEventDestroy(ev.second);
    }
    ctx->pending.clear();
}

inline std::uint32_t next_pow2(std::uint64_t v)
{
    std::uint32_t p = 1;
    while (p < v) {
        p <<= 1;
    }
    return p;
}

}  // namespace spk
