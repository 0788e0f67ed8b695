#include "host_copy.hpp"

#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "context.hpp"

namespace spk {

namespace {

constexpr std::size_t kSlotBytes = 512 << 10;
constexpr std::size_t kMaxThreads = 4;
constexpr std::size_t kChunkSlots = 8;  // slots pinned at once
constexpr std::size_t kMaxSlots = 16;
// Which way is the fastest depends on the size and on what the CPU last did
// with the destination's pages: medians in us, 200 to 300 us apart, so that
// helpers sleep in between and cost up to 300 us to wake (two machines).
//
//   MB to the host               0.5    1  1.5    2    4    8   10   16    33
//   touched, not lately  plain    50   84  116  139  249  484  576  866  1634
//                        slots    54   88  122  156  300  669  884 1681  2177
//                        helped                 208  401  405  660   980
//                                               511  614  651  587
//   just written         plain    82  133  180  218  302  576  831 1076
//                        slots    44   69  107  147  298  638  870 1555
//   never touched        plain   250  471       920 1828 3578 4543 7262 14934
//                        slots   152  282       557 1097 2159 2798 4454 11570
//                        helped                      981 1290 1253 1500  2897
//   to the device        plain    40   68       112  229  432  540  840  1728
//                        slots    44   73       154  285  541  683 1073  2201
//                        helped                      367  699  830 1237  1701
//
// The driver's own way faults untouched pages in as it goes: slots win at any
// size there, with helpers from 4 to 8 MB on.  Into touched pages slots cost at
// most 5 us more up to 1.5 MB and save up to 70; beyond, up to 40% more, until
// helpers pay: at 3 MB where they wake fast, at 12 where they do not, so from 8
// on (a program that asks for 11 MB proximity fields: 0.83 ms a call the plain
// way, 0.52 this way).  The sources above were read shortly before.  From memory,
// inputs of FP32 correlations, whole calls in ms with plain copies, slots from 4
// and helped slots from 8 MB: 4.2 MB 0.85, 1.08, 0.9; 6.5 MB 1.06, 1.45, 1.3; 9 MB
// 1.4, 1.58, 1.57; 12 MB 1.82, 1.74, 1.72; 15 MB 2.38, 2.06, 2.11; 26 MB 3.82, 3.08,
// 2.92: plain below 12 MB.
constexpr std::size_t kSmallBytes = 3 << 19;
constexpr std::size_t kHelpedBytes = 8 << 20;
constexpr std::size_t kSourceBytes = 12 << 20;
double mega(std::size_t bytes) { return static_cast<double>(bytes) / (1 << 20); }

// Pinning a chunk of slots and giving it back costs 2.5 to 8 ms, which a context
// that makes a few small copies never gets back.  Copies therefore take the
// plain way until what slots would have saved them (us per MB, from the table)
// comes to that.
constexpr double kPinCost = 3000;
constexpr double kSavedUntouched = 180, kSavedTouched = 30;
// Bytes that pay for a helper more.
constexpr std::size_t kBytesPerThread = 3 << 20;

// What the process keeps for its copies while it has contexts: pinned slots and
// helper threads.  Allocated once and never destroyed, so that no exit order
// matters.
struct Shared {
    std::mutex lock;
    int contexts {};
    std::vector<char*> free;     // slots nobody has checked out
    std::vector<void*> chunks;   // their allocations
    double earned {};            // us that slots have saved, or would have

    // Helpers wait for posted work.  A ticket is one helper's share of a copy.
    struct Work {
        std::function<void()> body;
        std::size_t tickets;  // not yet taken
        std::size_t running;
    };
    std::condition_variable posted, left;
    std::vector<Work*> work;
    std::vector<std::thread> helpers;
    // Helpers end when their generation is over.  The last context to go ends
    // it; contexts opened while it still joins them get helpers of the next.
    unsigned generation {};

    void serve(unsigned mine)
    {
        std::unique_lock<std::mutex> hold(lock);
        for (;;) {
            posted.wait(hold, [&] { return generation != mine || !work.empty(); });
            if (generation != mine) {
                return;
            }
            Work* w = work.back();
            ++w->running;
            if (--w->tickets == 0) {
                work.pop_back();
            }
            const bool more = !work.empty();
            hold.unlock();
            if (more) {
                posted.notify_one();
            }
            w->body();
            hold.lock();
            --w->running;
            left.notify_all();
        }
    }
};
Shared& shared()
{
    static Shared* s = new Shared;
    return *s;
}

// Up to `want` slots checked out for one copy, which saves `saved` us by them,
// with the context's events beside them; returned when the copy is done with them.
class Slots {
public:
    Slots(spk_context* ctx, std::size_t want, double saved)
    {
        Shared& p = shared();
        {
            const std::lock_guard<std::mutex> hold(p.lock);
            p.earned += saved;
            while (p.free.size() < want && p.chunks.size() * kChunkSlots < kMaxSlots &&
                   p.earned >= kPinCost * static_cast<double>(p.chunks.size() + 1)) {
                void* chunk {};
                if (cudaHostAlloc(&chunk, kChunkSlots * kSlotBytes, cudaHostAllocPortable) != cudaSuccess) {
                    cudaGetLastError();
                    break;
                }
                p.chunks.push_back(chunk);
                for (std::size_t i = 0; i < kChunkSlots; ++i) {
                    p.free.push_back(static_cast<char*>(chunk) + i * kSlotBytes);
                }
            }
            while (slot.size() < want && !p.free.empty()) {
                slot.push_back(p.free.back());
                p.free.pop_back();
            }
        }
        while (ctx->copy_events.size() < slot.size()) {
            cudaEvent_t e;
            if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                break;
            }
            ctx->copy_events.push_back(e);
        }
        usable_ = std::min(slot.size(), ctx->copy_events.size());
    }
    ~Slots()
    {
        Shared& p = shared();
        const std::lock_guard<std::mutex> hold(p.lock);
        p.free.insert(p.free.end(), slot.begin(), slot.end());
    }
    Slots(const Slots&) = delete;
    Slots& operator=(const Slots&) = delete;
    std::size_t usable() const { return usable_; }

    std::vector<char*> slot;

private:
    std::size_t usable_ {};
};

// Waits for the thread that drives the copy, which always gets there: after a
// failure it counts every chunk as arrived.
template <class Condition>
void wait_until(const Condition& condition)
{
    for (int spins = 0; !condition(); ++spins) {
        if (spins < 4096) {
#if defined(__x86_64__)
            __builtin_ia32_pause();
#endif
        }
        else {
            std::this_thread::yield();
        }
    }
}

// Whether CUDA knows the memory: the DMA reaches pinned or managed pages itself
// (STL files of 33 and 100 MB into pinned memory 0.65 and 1.9 ms, 0.93 and 2.9
// through slots).
bool registered(const void* at)
{
    cudaPointerAttributes a {};
    return cudaPointerGetAttributes(&a, at) == cudaSuccess && a.type != cudaMemoryTypeUnregistered;
}

// Whether more than a sixteenth of `bytes` from `at` on lies in pages that were
// never touched, as far as both ends tell: from there on the slots' 10 us per MB
// more are less than the 180 us per MB that they save on those pages.
bool untouched(const void* at, std::size_t bytes)
{
    constexpr std::size_t most = 256;  // pages asked about at each end
    const auto page = static_cast<std::uintptr_t>(sysconf(_SC_PAGESIZE));
    const std::uintptr_t first = reinterpret_cast<std::uintptr_t>(at) / page;
    const std::size_t pages = (reinterpret_cast<std::uintptr_t>(at) + bytes + page - 1) / page - first;
    const std::size_t head = std::min(pages, most), tail = std::min(pages - head, most);
    unsigned char resident[2 * most];
    if (!bytes || mincore(reinterpret_cast<void*>(first * page), head * page, resident) != 0 ||
        (tail && mincore(reinterpret_cast<void*>((first + pages - tail) * page), tail * page, resident + head) != 0)) {
        return false;
    }
    const auto missing = static_cast<std::size_t>(
        std::count_if(resident, resident + head + tail, [](unsigned char r) { return !(r & 1); }));
    return missing > (head + tail) / 16;
}

std::size_t most_helpers()
{
    return std::min<std::size_t>(kMaxThreads, std::thread::hardware_concurrency() / 2);
}

// Helper threads at work on a copy until the end of the scope.  There may be
// fewer than wanted, or none: the calling thread takes any chunk no helper has.
class Helpers {
public:
    Helpers(std::size_t bytes, std::function<void()> body) : work_ { std::move(body), 0, 0 }
    {
        const std::size_t want = std::min(most_helpers(), bytes / kBytesPerThread);
        if (bytes < kHelpedBytes || !want) {
            return;
        }
        Shared& p = shared();
        {
            const std::lock_guard<std::mutex> hold(p.lock);
            try {
                while (p.helpers.size() < want) {
                    p.helpers.emplace_back([&p, mine = p.generation] { p.serve(mine); });
                }
                work_.tickets = want;
                p.work.insert(p.work.begin(), &work_);
            }
            catch (...) {
                work_.tickets = 0;
            }
        }
        p.posted.notify_one();  // each helper wakes the next
    }
    ~Helpers()
    {
        Shared& p = shared();
        std::unique_lock<std::mutex> hold(p.lock);
        p.work.erase(std::remove(p.work.begin(), p.work.end(), &work_), p.work.end());
        p.left.wait(hold, [&] { return work_.running == 0; });
    }
    Helpers(const Helpers&) = delete;
    Helpers& operator=(const Helpers&) = delete;

private:
    Shared::Work work_;
};

// The chunks of one copy: claimed in order, each finished by whoever claimed it.
struct Chunks {
    Chunks(std::size_t bytes_, std::size_t slots_) :
        bytes(bytes_), slots(slots_), count((bytes_ + kSlotBytes - 1) / kSlotBytes),
        finished(new std::atomic<bool>[count])
    {
        for (std::size_t i = 0; i < count; ++i) {
            finished[i].store(false, std::memory_order_relaxed);
        }
    }
    std::size_t size(std::size_t i) const { return std::min(kSlotBytes, bytes - i * kSlotBytes); }

    const std::size_t bytes, slots, count;
    std::unique_ptr<std::atomic<bool>[]> finished;  // the host side of chunk i is done
    std::atomic<std::size_t> next { 0 };            // first chunk nobody has claimed
    std::atomic<std::size_t> arrived { 0 };         // DMAs complete, in order
};

}  // namespace

void copy_resources_acquire()
{
    Shared& p = shared();
    const std::lock_guard<std::mutex> hold(p.lock);
    ++p.contexts;
}

void copy_resources_release()
{
    Shared& p = shared();
    std::vector<std::thread> helpers;
    {
        const std::lock_guard<std::mutex> hold(p.lock);
        if (--p.contexts != 0) {
            return;
        }
        for (void* chunk : p.chunks) {
            cudaFreeHost(chunk);
        }
        p.chunks.clear();
        p.free.clear();
        p.earned = 0;
        helpers.swap(p.helpers);
        ++p.generation;
    }
    p.posted.notify_all();
    for (auto& t : helpers) {
        t.join();
    }
}

int copy_to_host(spk_context* ctx, void* dst, const void* d_src, std::size_t bytes)
{
    cudaStream_t st = ctx->stream;
    bool ok = true;
    const bool pageable = bytes && !registered(dst);
    const bool fresh = pageable && untouched(dst, bytes);
    const bool staged =
        fresh || (pageable && (bytes <= kSmallBytes || (bytes >= kHelpedBytes && most_helpers() > 1)));
    Slots slots(ctx, staged ? std::min((bytes + kSlotBytes - 1) / kSlotBytes, kMaxSlots) : 0,
                staged ? mega(bytes) * (fresh ? kSavedUntouched : kSavedTouched) : 0.0);
    if (!slots.usable()) {
        ok = !bytes || cudaMemcpyAsync(dst, d_src, bytes, cudaMemcpyDeviceToHost, st) == cudaSuccess;
    }
    else {
        Chunks c(bytes, slots.usable());
        const auto empty = [&](std::size_t i) {
            std::memcpy(static_cast<char*>(dst) + i * kSlotBytes, slots.slot[i % c.slots], c.size(i));
            c.finished[i].store(true, std::memory_order_release);
        };
        // After a failure nothing is in flight any more, and every chunk counts as
        // arrived, so that nobody waits.
        const auto broken = [&] {
            ok = false;
            cudaStreamSynchronize(st);
        };
        // This thread keeps the slots filling and sees them arrive; the helpers
        // empty them without calling CUDA.
        std::size_t issued = 0;
        const auto issue = [&] {
            while (issued < c.count &&
                   (issued < c.slots || c.finished[issued - c.slots].load(std::memory_order_acquire))) {
                const char* from = static_cast<const char*>(d_src) + issued * kSlotBytes;
                if (ok &&
                    (cudaMemcpyAsync(slots.slot[issued % c.slots], from, c.size(issued), cudaMemcpyDeviceToHost, st) !=
                         cudaSuccess ||
                     cudaEventRecord(ctx->copy_events[issued % c.slots], st) != cudaSuccess)) {
                    broken();
                }
                ++issued;
            }
        };
        issue();
        const auto help = [&] {
            for (;;) {
                const std::size_t i = c.next.fetch_add(1, std::memory_order_relaxed);
                if (i >= c.count) {
                    return;
                }
                wait_until([&] { return c.arrived.load(std::memory_order_acquire) > i; });
                empty(i);
            }
        };
        // Woken while the work before the copy runs.
        const Helpers helpers(bytes, help);
        if (ok && cudaEventSynchronize(ctx->copy_events[0]) != cudaSuccess) {
            broken();
        }
        std::size_t arrived = 0;
        while (arrived < c.count) {
            issue();
            const cudaError_t state = ok ? cudaEventQuery(ctx->copy_events[arrived % c.slots]) : cudaErrorUnknown;
            if (arrived < issued && state != cudaErrorNotReady) {
                if (ok && state != cudaSuccess) {
                    broken();
                }
                c.arrived.store(++arrived, std::memory_order_release);
                continue;
            }
            // Nothing new: take a chunk that is here.
            std::size_t i = c.next.load(std::memory_order_relaxed);
            if (i < arrived && c.next.compare_exchange_strong(i, i + 1, std::memory_order_relaxed)) {
                empty(i);
            }
        }
        help();
    }
    // Nothing of this copy stays in flight, whatever failed.
    const bool drained = cudaStreamSynchronize(st) == cudaSuccess;
    cudaGetLastError();  // an event found not ready is recorded like an error
    return ok && drained ? kOk : kCuda;
}

int copy_to_device(spk_context* ctx, void* d_dst, const void* src, std::size_t bytes)
{
    cudaStream_t st = ctx->stream;
    bool ok = true;
    if (bytes < kSourceBytes || most_helpers() < 2 || registered(src)) {
        ok = cudaMemcpyAsync(d_dst, src, bytes, cudaMemcpyHostToDevice, st) == cudaSuccess;
    }
    else {
        Slots slots(ctx, kMaxSlots, mega(bytes) * kSavedTouched);
        if (!slots.usable()) {
            ok = cudaMemcpyAsync(d_dst, src, bytes, cudaMemcpyHostToDevice, st) == cudaSuccess;
        }
        else {
            Chunks c(bytes, slots.usable());
            const auto fill = [&](std::size_t i) {
                std::memcpy(slots.slot[i % c.slots], static_cast<const char*>(src) + i * kSlotBytes, c.size(i));
                c.finished[i].store(true, std::memory_order_release);
            };
            const Helpers helpers(bytes, [&] {
                for (;;) {
                    const std::size_t i = c.next.fetch_add(1, std::memory_order_relaxed);
                    if (i >= c.count) {
                        return;
                    }
                    wait_until([&] { return i < c.slots + c.arrived.load(std::memory_order_acquire); });
                    fill(i);
                }
            });
            // As in copy_to_host: the slots go back with nothing in flight.
            const auto broken = [&] {
                ok = false;
                cudaStreamSynchronize(st);
            };
            std::size_t issued = 0, arrived = 0;
            while (arrived < c.count) {
                if (issued < c.count && c.finished[issued].load(std::memory_order_acquire)) {
                    if (ok &&
                        (cudaMemcpyAsync(static_cast<char*>(d_dst) + issued * kSlotBytes, slots.slot[issued % c.slots],
                                         c.size(issued), cudaMemcpyHostToDevice, st) != cudaSuccess ||
                         cudaEventRecord(ctx->copy_events[issued % c.slots], st) != cudaSuccess)) {
                        broken();
                    }
                    ++issued;
                    continue;
                }
                if (arrived < issued) {
                    const cudaError_t state =
                        ok ? cudaEventQuery(ctx->copy_events[arrived % c.slots]) : cudaErrorUnknown;
                    if (state != cudaErrorNotReady) {
                        if (ok && state != cudaSuccess) {
                            broken();
                        }
                        c.arrived.store(++arrived, std::memory_order_release);
                        continue;
                    }
                }
                // Nothing new: fill a chunk whose slot is free.
                std::size_t i = c.next.load(std::memory_order_relaxed);
                if (i < c.count && i < c.slots + arrived &&
                    c.next.compare_exchange_strong(i, i + 1, std::memory_order_relaxed)) {
                    fill(i);
                }
            }
        }
    }
    if (!ok) {
        cudaStreamSynchronize(st);
    }
    cudaGetLastError();
    return ok ? kOk : kCuda;
}

}  // namespace spk
