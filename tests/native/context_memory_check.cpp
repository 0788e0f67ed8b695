// The context's device memory (csrc/context.hpp) against a device of limited
// size: CUDA's allocation calls are replaced by an accounting one.
#include <cstdio>
#include <cstdlib>
#include <unordered_map>

#include "../../cpp-max-packer_b200/csrc/context.hpp"

namespace {

std::uint64_t device_bytes = 0, used = 0;
std::unordered_map<void*, std::uint64_t> blocks;
int failures = 0;

void check(bool ok, const char* what)
{
    if (!ok) {
        std::printf("FAILED: %s\n", what);
        ++failures;
    }
}

}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t bytes)
{
    if (used + bytes > device_bytes) {
        return cudaErrorMemoryAllocation;
    }
    *p = std::malloc(1);
    blocks[*p] = bytes;
    used += bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    if (!p) {
        return cudaSuccess;
    }
    used -= blocks.at(p);
    blocks.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

int main()
{
    constexpr std::uint64_t MB = 1 << 20;
    device_bytes = 300 * MB;
    {
        // A closed session's block gives way to a buffer the device has no
        // other room for, and to a second session's larger block.
        spk_context ctx;
        int status = spk::kOk;
        std::size_t bytes = 200 * MB;
        void* block = spk::take_block(&ctx, bytes, status);
        check(block && status == spk::kOk, "a session's block");
        spk::give_block(&ctx, block, bytes);
        check(used == 200 * MB, "the block is kept for the next session");
        check(spk::device_buffer(&ctx, "large", 150 * MB, status) && status == spk::kOk, "a buffer in its place");
        check(used == 150 * MB, "the kept block went");
        check(!spk::device_buffer(&ctx, "larger", 200 * MB, status) && status == spk::kAllocation,
              "more than the device has is refused");
        spk::drop_buffers(&ctx, { "large", "larger" });
        check(used == 0 && ctx.bytes_in_use == 0, "all is given back");
    }
    {
        // A reused block: the next session takes what the last one left.
        spk_context ctx;
        int status = spk::kOk;
        std::size_t bytes = 100 * MB;
        void* first = spk::take_block(&ctx, bytes, status);
        spk::give_block(&ctx, first, bytes);
        bytes = 90 * MB;
        check(spk::take_block(&ctx, bytes, status) == first && bytes == 100 * MB, "the kept block is taken again");
        spk::give_block(&ctx, first, bytes);
        spk::release_kept_blocks(&ctx);
        check(used == 0, "and given back");
    }
    {
        // Under a cap, buffers and kept blocks together stay within it.
        spk_context ctx;
        ctx.cap_bytes = 120 * MB;
        int status = spk::kOk;
        std::size_t bytes = 100 * MB;
        void* block = spk::take_block(&ctx, bytes, status);
        spk::give_block(&ctx, block, bytes);
        check(used == 100 * MB, "a block within the cap is kept");
        check(spk::device_buffer(&ctx, "b", 60 * MB, status) && status == spk::kOk, "a buffer within the cap");
        check(used == 60 * MB, "the kept block went for the cap");
        block = spk::take_block(&ctx, bytes, status);
        spk::give_block(&ctx, block, bytes);
        check(used == 60 * MB, "a block past the cap is not kept");
        check(!spk::device_buffer(&ctx, "b", 121 * MB, status) && status == spk::kMemoryLimit && used == 60 * MB,
              "a buffer past the cap is refused");
        check(spk::room_for(&ctx, "b") == 120 * MB && spk::room_for(&ctx, "c") == 60 * MB,
              "room for a buffer counts what it has");
        spk::drop_buffers(&ctx, { "b" });
    }
    std::printf(failures ? "%d failed\n" : "ok\n", failures);
    return failures ? 1 : 0;
}
