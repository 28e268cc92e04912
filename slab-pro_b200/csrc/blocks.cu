// The kept blocks of blocks.hpp.
#include "blocks.hpp"

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <string>
#include <unordered_map>

#include "error.hpp"

namespace slab {
namespace {

constexpr size_t MIB = (size_t)1 << 20;
constexpr size_t LIVE_BYTES = 4096 * MIB;  // an upload's release or a context of the 8192 x 8192 terrain; 2 % of a B200
constexpr size_t IDLE_BYTES = 1024 * MIB;
constexpr size_t SPARE_BYTES = 16 * MIB;
constexpr size_t PINNED_BYTES = 1024 * MIB;
constexpr int PINNED = -1;  // "device" of the page-locked blocks

struct Kept {
    void* p;
    uint64_t released;  // release number
};

struct Pool {
    std::multimap<size_t, Kept> kept;  // by size; nothing uses them
    size_t bytes = 0;
    size_t bound = 0;                  // of `bytes` while a context lives (0: not yet asked)
};

struct Live {
    size_t size;
    int dev;
};

struct Blocks {
    std::mutex mu;
    std::map<int, Pool> pools;
    std::unordered_map<void*, Live> live;
    uint64_t releases = 0;
    int users = 0;
};

// never destroyed: buffers of static lifetime may still release blocks at exit
Blocks& blocks() {
    static Blocks* b = new Blocks();
    return *b;
}

thread_local BlockScope* t_scope = nullptr;

// Size classes: four per octave up to 1 MiB, then multiples of 2 MiB (the
// driver's own granularity).
size_t size_class(size_t n) {
    if (n > MIB) return (n + 2 * MIB - 1) / (2 * MIB) * (2 * MIB);
    size_t step = 128;
    while (step * 8 < n) step *= 2;
    return std::max<size_t>(512, (n + step - 1) / step * step);
}

// a block of size `got` serves a request of class `size`
bool serves(size_t got, size_t size) { return got >= size && got <= size + std::min(size / 4, SPARE_BYTES); }

void driver_free(int dev, void* p) noexcept {
    if (dev == PINNED) cudaFreeHost(p);
    else cudaFree(p);
}

// kept blocks of `dev` back to the driver, oldest first, down to `bound`
// bytes; true if any went
bool trim(int dev, size_t bound) noexcept {
    Blocks& B = blocks();
    bool any = false;
    for (;;) {
        void* p;
        {
            std::lock_guard<std::mutex> lk(B.mu);
            const auto at = B.pools.find(dev);
            if (at == B.pools.end() || at->second.bytes <= bound || at->second.kept.empty()) return any;
            Pool& pool = at->second;
            auto old = pool.kept.begin();
            for (auto it = pool.kept.begin(); it != pool.kept.end(); ++it)
                if (it->second.released < old->second.released) old = it;
            p = old->second.p;
            pool.bytes -= old->first;
            pool.kept.erase(old);
        }
        driver_free(dev, p);
        any = true;
    }
}

// every device's kept blocks down to dev_bound bytes, the page-locked ones to pinned_bound
void trim_all(size_t dev_bound, size_t pinned_bound) noexcept {
    Blocks& B = blocks();
    for (int dev = PINNED - 1;;) {
        {
            std::lock_guard<std::mutex> lk(B.mu);
            const auto next = B.pools.upper_bound(dev);
            if (next == B.pools.end()) return;
            dev = next->first;
        }
        trim(dev, dev == PINNED ? pinned_bound : dev_bound);
    }
}

// a block that nothing uses, to its kept list
void keep(const BlockScope::Held& h) noexcept {
    Blocks& B = blocks();
    size_t bound = 0;
    try {
        {
            std::lock_guard<std::mutex> lk(B.mu);
            bound = B.pools[h.dev].bound;
        }
        if (!bound) {
            size_t free_b = 0, total_b = 0;
            if (h.dev == PINNED) bound = PINNED_BYTES;
            else if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) bound = std::max(std::min(total_b / 16, LIVE_BYTES), MIB);
            else bound = MIB;
        }
        if (h.size <= bound) {
            {
                std::lock_guard<std::mutex> lk(B.mu);
                Pool& pool = B.pools[h.dev];
                pool.bound = bound;
                pool.kept.emplace(h.size, Kept{h.p, ++B.releases});
                pool.bytes += h.size;
            }
            trim(h.dev, bound);
            return;
        }
    } catch (...) {  // no room for the bookkeeping: back to the driver
    }
    driver_free(h.dev, h.p);
}

void* driver_alloc(int dev, size_t size, cudaError_t& e) {
    void* p = nullptr;
    e = dev == PINNED ? cudaMallocHost(&p, size) : cudaMalloc(&p, size);
    if (e != cudaSuccess) cudaGetLastError();
    return p;
}

void* take(int dev, size_t bytes, const char* what) {
    Blocks& B = blocks();
    const size_t size = size_class(bytes ? bytes : 1);
    void* p = nullptr;
    size_t got = size;
    // one that this scope released, the smallest that serves
    BlockScope* const s = t_scope;
    if (s) {
        auto best = s->held.end();
        for (auto it = s->held.begin(); it != s->held.end(); ++it)
            if (it->dev == dev && serves(it->size, size) && (best == s->held.end() || it->size < best->size)) best = it;
        if (best != s->held.end()) {
            p = best->p;
            got = best->size;
            s->held.erase(best);
        }
    }
    if (!p) {
        std::lock_guard<std::mutex> lk(B.mu);
        const auto at = B.pools.find(dev);
        if (at != B.pools.end()) {
            const auto it = at->second.kept.lower_bound(size);
            if (it != at->second.kept.end() && serves(it->first, size)) {
                p = it->second.p;
                got = it->first;
                at->second.bytes -= got;
                at->second.kept.erase(it);
            }
        }
    }
    if (!p) {
        cudaError_t e;
        p = driver_alloc(dev, size, e);
        if (e != cudaSuccess) {
            if (s) s->flush();
            if (trim(dev, 0)) p = driver_alloc(dev, size, e);
        }
        if (e != cudaSuccess)
            throw Error{SLAB_E_OOM, std::string(what) + " of " + std::to_string(bytes) + " bytes failed: " + cudaGetErrorString(e)};
    }
    try {
        std::lock_guard<std::mutex> lk(B.mu);
        B.live[p] = Live{got, dev};
    } catch (...) {
        driver_free(dev, p);
        throw;
    }
    return p;
}

void release(void* p) noexcept {
    if (!p) return;
    Blocks& B = blocks();
    BlockScope::Held h{p, 0, 0};
    {
        std::lock_guard<std::mutex> lk(B.mu);
        const auto it = B.live.find(p);
        if (it == B.live.end()) return;
        h.size = it->second.size;
        h.dev = it->second.dev;
        B.live.erase(it);
    }
    if (t_scope && t_scope->stream) {
        try {
            t_scope->held.push_back(h);
            return;
        } catch (...) {  // no room for the bookkeeping: back to the driver
        }
    }
    driver_free(h.dev, p);
}

}  // namespace

BlockScope::BlockScope(cudaStream_t st) noexcept : stream(st), outer(t_scope) { t_scope = this; }

BlockScope::~BlockScope() {
    flush();
    t_scope = outer;
}

void BlockScope::flush() noexcept {
    if (held.empty()) return;
    const bool idle = cudaStreamSynchronize(stream) == cudaSuccess;
    for (const Held& h : held) {
        if (idle) keep(h);
        else driver_free(h.dev, h.p);
    }
    held.clear();
}

void* take_device(size_t bytes) {
    int dev = 0;
    SLAB_CUDA(cudaGetDevice(&dev));
    return take(dev, bytes, "cudaMalloc");
}
void release_device(void* p) noexcept { release(p); }
void* take_pinned(size_t bytes) { return take(PINNED, bytes, "cudaMallocHost"); }
void release_pinned(void* p) noexcept { release(p); }

void trim_blocks() noexcept { trim_all(0, 0); }

size_t kept_device_bytes() {
    int dev = 0;
    SLAB_CUDA(cudaGetDevice(&dev));
    Blocks& B = blocks();
    std::lock_guard<std::mutex> lk(B.mu);
    return B.pools[dev].bytes;
}

MemoryUser::MemoryUser() {
    Blocks& B = blocks();
    std::lock_guard<std::mutex> lk(B.mu);
    ++B.users;
}
MemoryUser::~MemoryUser() {
    Blocks& B = blocks();
    {
        std::lock_guard<std::mutex> lk(B.mu);
        if (--B.users != 0) return;
    }
    trim_all(IDLE_BYTES, IDLE_BYTES / 4);
}

}  // namespace slab
