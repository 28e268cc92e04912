// Device and page-locked memory blocks, kept for the next request of about
// the same size instead of going back to the driver.
//
// Why: an upload, a release or a new batch takes some tens of blocks and gives
// them back a moment later, and on B200 one cudaMalloc of 1 MiB to 256 MiB
// measures 0.36-0.38 ms, its cudaFree 0.29-0.41 ms, a 1 GiB pair 1.7 ms, a
// 64 MiB cudaMallocHost 41 ms: more than the steps of a small run.
//
// Rules:
//  - release_device() may be called with work in flight on the block, as
//    cudaFree may: the block is handed out again only after a
//    cudaDeviceSynchronize() that began after the release (one such wait
//    covers every block released before it). cudaFree waits the same way.
//  - release_pinned() is called when no copy uses the block any more.
//  - The blocks kept are bounded per device (1/16 of its memory while a
//    context lives, IDLE_BYTES after the last one closed; page-locked memory:
//    PINNED_BYTES, IDLE_BYTES / 4), and all of a device's go back to the
//    driver when an allocation fails, before it is tried again.
//  - A block belongs to the device that was current when it was taken.
//  - One mutex guards the lists: any thread may take and release blocks.
//  - Contents are undefined, as cudaMalloc's are.
#pragma once

#include <cstddef>

namespace slab {

void* take_device(size_t bytes);  // throws Error{SLAB_E_OOM | SLAB_E_CUDA}
void release_device(void* p) noexcept;
void* take_pinned(size_t bytes);
void release_pinned(void* p) noexcept;
size_t kept_device_bytes();  // kept on the current device, handed back if an allocation needs them

// One per context (slab_ctx, slab_batch, slab_server): the last to go trims
// the kept blocks to the idle bound. First member of its context, so that it
// is destroyed after the context's buffers.
struct MemoryUser {
    MemoryUser();
    ~MemoryUser();
    MemoryUser(const MemoryUser&) = delete;
    MemoryUser& operator=(const MemoryUser&) = delete;
};

}  // namespace slab
