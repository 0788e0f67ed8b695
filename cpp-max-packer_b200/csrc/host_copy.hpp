// Copies between pageable host memory and the device.
#pragma once

#include <cstddef>

struct spk_context;

namespace spk {

// Copies `bytes` from the device to host memory after the work queued on the
// context's stream, and waits.
//
// A plain copy to pageable memory runs through the driver's staging on one
// thread: 20 GB/s, 2.2 where the pages were never touched.  Small and large
// copies, and those into untouched pages, go through pinned slots that up to
// four helper threads empty side by side behind the DMA (host_copy.cu has the
// sizes).
//
// The slots (16 of 512 KB at most) and the helpers belong to the process:
// pinning costs about a millisecond per megabyte and a thread started per copy
// about 200 us around its start and end, which every context or copy would pay
// anew.  The slots are pinned once the copies made have earned that.  Any number
// of contexts and threads may copy at once: a copy checks out the slots that are
// free, or takes the plain way where none is, and gets the helpers that are idle.
// The last context to go gives all of it back.
int copy_to_host(spk_context* ctx, void* dst, const void* d_src, std::size_t bytes);

// The other way, queued on the context's stream; the source may be reused on
// return.
int copy_to_device(spk_context* ctx, void* d_dst, const void* src, std::size_t bytes);

// Counts the contexts there are, for the slots' and helpers' lifetime.
void copy_resources_acquire();
void copy_resources_release();

}  // namespace spk
