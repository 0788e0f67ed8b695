// The staged copies (csrc/host_copy.cu) on the host: CUDA's calls are replaced
// by streams that do their work when they are asked about it, so that copies
// are in flight until then; helper threads are real.  argv[1] names the check.
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

// Every copy by the CPU is counted for its thread.
namespace std {
inline void* counted_memcpy(void* to, const void* from, size_t bytes);
}
#define memcpy counted_memcpy
#include "../../cpp-max-packer_b200/csrc/host_copy.cu"
#undef memcpy

namespace {

std::mutex copies_lock;
std::set<std::thread::id> copied_by;
std::chrono::microseconds memcpy_time { 0 };

struct Op {
    void* to;
    const void* from;
    std::size_t bytes;
    bool* event;  // null: a copy
};
struct FakeStream {
    std::deque<Op> queue;
    void run_one()
    {
        const Op op = queue.front();
        queue.pop_front();
        if (op.event) {
            *op.event = true;
        }
        else {
            std::memmove(op.to, op.from, op.bytes);
        }
    }
};
FakeStream* fake(cudaStream_t s) { return reinterpret_cast<FakeStream*>(s); }
struct FakeEvent {
    bool done;
    FakeStream* stream;
};

int fail_copy_after = -1;  // that many copies succeed
std::atomic<long long> pinned { 0 };
std::atomic<int> pin_calls { 0 };
bool pin_fails = false;
std::size_t largest_dma = 0;
const void* known_to_cuda = nullptr;  // pinned by the caller
std::function<void()> on_synchronize;

int failures = 0;
void check(bool ok, const char* what)
{
    if (!ok) {
        std::printf("FAILED: %s\n", what);
        ++failures;
    }
}

}  // namespace

namespace std {
inline void* counted_memcpy(void* to, const void* from, size_t bytes)
{
    {
        const lock_guard<mutex> hold(copies_lock);
        copied_by.insert(this_thread::get_id());
    }
    if (memcpy_time.count()) {
        this_thread::sleep_for(memcpy_time);
    }
    return memmove(to, from, bytes);
}
}  // namespace std

extern "C" {
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind, cudaStream_t s)
{
    if (fail_copy_after == 0) {
        return cudaErrorUnknown;
    }
    fail_copy_after -= fail_copy_after > 0;
    largest_dma = std::max(largest_dma, bytes);
    fake(s)->queue.push_back({ to, from, bytes, nullptr });
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int)
{
    *e = reinterpret_cast<cudaEvent_t>(new FakeEvent { true, nullptr });
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    auto* event = reinterpret_cast<FakeEvent*>(e);
    event->done = false;
    event->stream = fake(s);
    fake(s)->queue.push_back({ nullptr, nullptr, 0, &event->done });
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e)
{
    auto* event = reinterpret_cast<FakeEvent*>(e);
    if (!event->done) {
        event->stream->run_one();
    }
    return event->done ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    auto* event = reinterpret_cast<FakeEvent*>(e);
    while (!event->done) {
        event->stream->run_one();
    }
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    if (on_synchronize) {
        on_synchronize();
    }
    while (!fake(s)->queue.empty()) {
        fake(s)->run_one();
    }
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned int)
{
    if (pin_fails) {
        return cudaErrorMemoryAllocation;
    }
    *p = std::malloc(bytes);
    pinned += static_cast<long long>(bytes);
    ++pin_calls;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
    std::free(p);
    pinned -= static_cast<long long>(spk::kChunkSlots * spk::kSlotBytes);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    *a = {};
    a->type = p == known_to_cuda ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void**, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
}

namespace {

constexpr std::size_t KB = 1 << 10, MB = 1 << 20;

struct Context {
    FakeStream stream;
    spk_context ctx;
    Context()
    {
        ctx.stream = reinterpret_cast<cudaStream_t>(&stream);
        spk::copy_resources_acquire();
    }
    ~Context()
    {
        for (auto e : ctx.copy_events) {
            delete reinterpret_cast<FakeEvent*>(e);
        }
        spk::copy_resources_release();
    }
};

std::vector<char> pattern(std::size_t n, unsigned seed)
{
    std::vector<char> v(n);
    for (std::size_t i = 0; i < n; ++i) {
        v[i] = static_cast<char>((i * 2654435761u + seed) >> 7);
    }
    return v;
}

// Copies both ways, into memory that was touched and into memory that was not.
bool round_trip(Context& c, std::size_t n, unsigned seed)
{
    const auto want = pattern(n, seed);
    std::vector<char> device(n), back(n);
    if (spk::copy_to_device(&c.ctx, device.data(), want.data(), n) != spk::kOk) {
        return false;
    }
    cudaStreamSynchronize(c.ctx.stream);
    if (device != want || spk::copy_to_host(&c.ctx, back.data(), device.data(), n) != spk::kOk || back != want) {
        return false;
    }
    const std::size_t pages = (n + 3 + 4095) / 4096 * 4096;
    char* fresh = static_cast<char*>(mmap(nullptr, pages, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    char* to = fresh + 3;  // no alignment is promised
    const bool ok = spk::copy_to_host(&c.ctx, to, device.data(), n) == spk::kOk &&
                    std::memcmp(to, want.data(), n) == 0 && c.stream.queue.empty();
    munmap(fresh, pages);
    return ok;
}

void sizes()
{
    Context c;
    for (std::size_t n : { std::size_t { 1 }, 4 * KB, 512 * KB - 1, 512 * KB, 512 * KB + 1, 1 * MB, 4 * MB - 1, 4 * MB,
                           4 * MB + 1, 8 * MB - 1, 8 * MB, 8 * MB + 1, 12 * MB + 1, 33 * MB, 33 * MB + 5 }) {
        check(round_trip(c, n, static_cast<unsigned>(n)), "a copy's bytes");
    }
    check(spk::copy_to_host(&c.ctx, nullptr, nullptr, 0) == spk::kOk, "no bytes");
}

// Which copies go through slots: DMAs of a slot at most.
void ways()
{
    Context c;
    check(round_trip(c, 64 * MB, 1), "a copy that earns both chunks of slots");
    const bool helped = spk::most_helpers() > 1;
    const auto staged = [&](std::size_t n, bool to_device, bool touched, bool known = false) {
        char* host = static_cast<char*>(mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
        if (touched) {
            std::memset(host, 1, n);
        }
        known_to_cuda = known ? host : nullptr;
        std::vector<char> device(n, 2);
        largest_dma = 0;
        const int status = to_device ? spk::copy_to_device(&c.ctx, device.data(), host, n)
                                     : spk::copy_to_host(&c.ctx, host, device.data(), n);
        cudaStreamSynchronize(c.ctx.stream);
        check(status == spk::kOk && std::memcmp(host, device.data(), n) == 0, "a copy's bytes");
        munmap(host, n);
        return largest_dma < n;
    };
    for (std::size_t n : { 4 * KB, 512 * KB, 3 * MB / 2 }) {
        check(staged(n, false, true) == (n > 512 * KB) && staged(n, false, false) == (n > 512 * KB),
              "small copies take the slots, in one piece up to a slot");
    }
    for (std::size_t mb : { 2, 3, 5, 7 }) {
        check(!staged(mb * MB, false, true), "touched pages below 8 MB take the plain way");
        check(staged(mb * MB, false, false), "untouched pages take the slots");
        check(!staged(mb * MB, true, true), "sources below 12 MB take the plain way");
    }
    for (std::size_t mb : { 8, 11, 12, 16, 50 }) {
        check(staged(mb * MB, false, true) == helped, "larger copies take the slots where there are helpers");
        check(staged(mb * MB, true, true) == (helped && mb >= 12), "and larger sources");
        check(!staged(mb * MB, false, true, true) && !staged(mb * MB, true, true, true),
              "pinned memory takes the plain way");
    }
}

// Slots are pinned once copies have earned them, and go with the last context.
void pins()
{
    std::vector<char> device(80 * MB, 1);
    const auto untouched_copy = [&](Context& c, std::size_t n) {
        char* to = static_cast<char*>(mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
        check(spk::copy_to_host(&c.ctx, to, device.data(), n) == spk::kOk && std::memcmp(to, device.data(), n) == 0,
              "a copy's bytes");
        munmap(to, n);
    };
    for (int i = 0; i < 40; ++i) {
        Context c;
        untouched_copy(c, 2 * MB);
        untouched_copy(c, 400 * KB);
    }
    check(pin_calls == 0, "contexts that make a few small copies pin nothing");
    {
        Context c;
        for (int i = 0; i < 20; ++i) {
            untouched_copy(c, 2 * MB);
        }
        check(pin_calls == 1 && pinned == static_cast<long long>(4 * MB), "many small copies pin one chunk");
        for (int i = 0; i < 20; ++i) {
            untouched_copy(c, 20 * MB);
        }
        check(pin_calls == 2 && pinned == static_cast<long long>(8 * MB), "large ones two, and no more");
    }
    check(pinned == 0, "the last context gives them back");
    pin_calls = 0;
    {
        Context c;
        untouched_copy(c, 80 * MB);
        check(pin_calls == 2, "one large copy earns both at once");
    }
    check(pinned == 0, "and gives them back");
}

void pinned_by_the_caller()
{
    Context c;
    check(round_trip(c, 64 * MB, 1), "a copy that earns the slots");
    for (std::size_t n : { 700 * KB, 3 * MB / 2, 3 * MB, 9 * MB, 40 * MB }) {
        const auto want = pattern(n, 2);
        std::vector<char> to(n);
        known_to_cuda = to.data();
        largest_dma = 0;
        check(spk::copy_to_host(&c.ctx, to.data(), want.data(), n) == spk::kOk && to == want && largest_dma == n,
              "a pinned destination gets one DMA");
        known_to_cuda = want.data();
        largest_dma = 0;
        check(spk::copy_to_device(&c.ctx, to.data(), want.data(), n) == spk::kOk, "a copy to the device");
        cudaStreamSynchronize(c.ctx.stream);
        check(to == want && largest_dma == n, "a pinned source too");
        known_to_cuda = nullptr;
    }
}

void no_slots()
{
    pin_fails = true;
    Context c;
    check(round_trip(c, 9 * MB + 7, 1) && round_trip(c, 40 * MB, 2), "copies where nothing can be pinned");
    pin_fails = false;
}

void threads()
{
    std::vector<std::thread> all;
    std::atomic<int> bad { 0 };
    for (unsigned t = 0; t < 6; ++t) {
        all.emplace_back([&, t] {
            for (unsigned i = 0; i < 6; ++i) {
                Context c;
                bad += !round_trip(c, (5 + 7 * t) * MB + 11 * i, 100 * t + i);
                bad += !round_trip(c, 40 * MB + i, t + i);
            }
        });
    }
    for (auto& t : all) {
        t.join();
    }
    check(bad == 0, "copies of several threads and contexts");
    check(pinned == 0, "the last context gives the slots back");
}

// Contexts that close while others open: the next copies still have helpers.
void helpers_live()
{
    const std::size_t n = 64 * MB;
    const auto want = pattern(n, 3);
    std::vector<char> back(n);
    const auto copy = [&](Context& c) { check(spk::copy_to_host(&c.ctx, back.data(), want.data(), n) == spk::kOk, "a copy"); };
    for (int i = 0; i < 300; ++i) {
        auto* closing = new Context;
        if (i % 3 == 0) {
            copy(*closing);
        }
        std::thread other([&] { delete closing; });
        for (int k = 0; k < 20; ++k) {
            Context c;
            if (k % 7 == 0) {
                spk::Helpers wake(n, [] {});  // a copy's helpers, without its bytes
            }
        }
        other.join();
    }
    Context c;
    copy(c);
    copied_by.clear();
    memcpy_time = std::chrono::microseconds(300);  // the caller alone cannot keep up
    for (int i = 0; i < 4; ++i) {
        copy(c);
    }
    memcpy_time = std::chrono::microseconds(0);
    check(copied_by.size() == 1 + std::min<std::size_t>(spk::kMaxThreads, std::thread::hardware_concurrency() / 2),
          "every helper is at work after contexts came and went");
}

// A copy that fails keeps its slots until its DMAs are over.
void failing_copy()
{
    const std::size_t n = 40 * MB;
    const auto source = pattern(n, 5);
    std::vector<char> device(n);
    for (int after : { 0, 1, 5, 17, 40 }) {
        Context c;
        { Context warm; round_trip(warm, n, 1); }
        bool early = false;
        on_synchronize = [&] {
            const std::lock_guard<std::mutex> hold(spk::shared().lock);
            early = early || (!c.stream.queue.empty() &&
                              spk::shared().free.size() == spk::shared().chunks.size() * spk::kChunkSlots);
        };
        fail_copy_after = after;
        const int to_device = spk::copy_to_device(&c.ctx, device.data(), source.data(), n);
        const bool drained = c.stream.queue.empty();
        fail_copy_after = -1;
        on_synchronize = nullptr;
        check(to_device == spk::kCuda, "a failing copy to the device says so");
        check(drained, "and leaves nothing in flight");
        check(!early, "and holds its slots until then");
        fail_copy_after = after;
        const int to_host = spk::copy_to_host(&c.ctx, device.data(), source.data(), n);
        fail_copy_after = -1;
        check(to_host == spk::kCuda && c.stream.queue.empty(), "a failing copy to the host likewise");
        check(round_trip(c, n, 9), "the next copy is whole");
    }
}

}  // namespace

int main(int, char** argv)
{
    const std::string which = argv[1];
    if (which == "sizes") {
        sizes();
    }
    else if (which == "ways") {
        ways();
    }
    else if (which == "pins") {
        pins();
    }
    else if (which == "pinned_by_the_caller") {
        pinned_by_the_caller();
    }
    else if (which == "no_slots") {
        no_slots();
    }
    else if (which == "threads") {
        threads();
    }
    else if (which == "helpers_live") {
        helpers_live();
    }
    else if (which == "failing_copy") {
        failing_copy();
    }
    else {
        return 2;
    }
    std::printf(failures ? "%d failed\n" : "ok\n", failures);
    return failures ? 1 : 0;
}
