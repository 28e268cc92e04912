// Device and page-locked memory blocks, kept for the next request of about
// the same size instead of going back to the driver.
//
// Why: an upload, a release or a new batch takes some tens of blocks and gives
// them back a moment later, and on B200 one cudaMalloc of 1 MiB to 256 MiB
// measures 0.36-0.38 ms, its cudaFree 0.29-0.41 ms, a 1 GiB pair 1.7 ms, a
// 64 MiB cudaMallocHost 41 ms: more than the steps of a small run.
//
// Rules:
//  - A block may be released with work in flight on it, if that work is on the
//    stream of the calling thread's BlockScope. The scope holds the block: the
//    same scope may take it again at once, since what it does with the block
//    comes later on the same stream; everybody else gets it after the scope
//    has waited for its stream, at its end. Released outside a scope a block
//    goes to the driver, which waits by itself. So a kept block has no work in
//    flight, and no wait is wider than one stream: CUDA refuses to wait for a
//    device, whatever the capture mode, while any stream of it is being
//    captured, and other contexts' threads capture their step graphs at any time.
//  - The blocks kept are bounded per device (LIVE_BYTES, at most 1/16 of its
//    memory, while a context lives, IDLE_BYTES after the last one closed;
//    page-locked memory: PINNED_BYTES, IDLE_BYTES / 4). All of a device's go
//    back to the driver when an allocation fails, before it is tried again,
//    and all there are on trim_blocks().
//  - A kept block serves a request of at least 4/5 of its size, and no more
//    than SPARE_BYTES below it.
//  - A block belongs to the device that was current when it was taken.
//  - One mutex guards the lists: any thread may take and release blocks. No
//    driver call is made while it is held.
//  - Contents are undefined, as cudaMalloc's are.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

namespace slab {

void* take_device(size_t bytes);  // throws Error{SLAB_E_OOM | SLAB_E_CUDA}
void release_device(void* p) noexcept;
void* take_pinned(size_t bytes);
void release_pinned(void* p) noexcept;
void trim_blocks() noexcept;  // every kept block, of any device, back to the driver
size_t kept_device_bytes();  // kept on the current device, handed back if an allocation needs them

// One per call into a context, on the calling thread: all that the call does
// with blocks is on `st`, or over before it releases them. nullptr: the stream
// is not known, releases go to the driver. Scopes may nest.
class BlockScope {
  public:
    explicit BlockScope(cudaStream_t st) noexcept;
    ~BlockScope();
    BlockScope(const BlockScope&) = delete;
    BlockScope& operator=(const BlockScope&) = delete;

    struct Held {
        void* p;
        size_t size;
        int dev;
    };
    // Waits for the stream and puts the held blocks on the kept lists.
    void flush() noexcept;

    const cudaStream_t stream;
    std::vector<Held> held;

  private:
    BlockScope* const outer;
};

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
