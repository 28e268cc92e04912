// The kept blocks of blocks.hpp.
#include "blocks.hpp"

#include <cstdint>
#include <map>
#include <mutex>
#include <string>
#include <unordered_map>

#include "engine.hpp"

namespace slab {
namespace {

constexpr size_t MIB = (size_t)1 << 20;
constexpr size_t IDLE_BYTES = 1024 * MIB;
constexpr size_t PINNED_BYTES = 1024 * MIB;
constexpr int PINNED = -1;  // "device" of the page-locked blocks

struct Kept {
    void* p;
    uint64_t released;  // release number; in flight until a wait that began later is over
};

struct Pool {
    std::multimap<size_t, Kept> kept;  // by size
    size_t bytes = 0;
    size_t bound = 0;                  // of `bytes` while a context lives (0: not yet asked)
    uint64_t idle_upto = 0;            // blocks released up to this number have no work in flight
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

// Size classes: four per octave up to 1 MiB, then multiples of 2 MiB (the
// driver's own granularity).
size_t size_class(size_t n) {
    if (n > MIB) return (n + 2 * MIB - 1) / (2 * MIB) * (2 * MIB);
    size_t step = 128;
    while (step * 8 < n) step *= 2;
    return std::max<size_t>(512, (n + step - 1) / step * step);
}

void driver_free(int dev, void* p) {
    if (dev == PINNED) cudaFreeHost(p);
    else cudaFree(p);
}

// oldest first, down to `bound` bytes
void trim(int dev, Pool& pool, size_t bound) {
    while (pool.bytes > bound && !pool.kept.empty()) {
        auto old = pool.kept.begin();
        for (auto it = pool.kept.begin(); it != pool.kept.end(); ++it)
            if (it->second.released < old->second.released) old = it;
        pool.bytes -= old->first;
        driver_free(dev, old->second.p);
        pool.kept.erase(old);
    }
}

void* take(int dev, size_t bytes, const char* what) {
    Blocks& B = blocks();
    const size_t size = size_class(bytes ? bytes : 1);
    std::lock_guard<std::mutex> lk(B.mu);
    Pool& pool = B.pools[dev];
    // a kept block of at most a quarter more; one without work in flight if there is one
    auto best = pool.kept.end();
    int looked = 0;
    for (auto it = pool.kept.lower_bound(size); it != pool.kept.end() && it->first <= size + size / 4 && looked < 16; ++it, ++looked) {
        if (best == pool.kept.end()) best = it;
        if (dev == PINNED || it->second.released <= pool.idle_upto) {
            best = it;
            break;
        }
    }
    if (best != pool.kept.end()) {
        if (dev != PINNED && best->second.released > pool.idle_upto) {
            SLAB_CUDA(cudaDeviceSynchronize());
            pool.idle_upto = B.releases;
        }
        void* p = best->second.p;
        const size_t got = best->first;
        B.live[p] = Live{got, dev};
        pool.bytes -= got;
        pool.kept.erase(best);
        return p;
    }
    void* p = nullptr;
    cudaError_t e = dev == PINNED ? cudaMallocHost(&p, size) : cudaMalloc(&p, size);
    if (e != cudaSuccess && pool.bytes) {
        cudaGetLastError();
        trim(dev, pool, 0);
        e = dev == PINNED ? cudaMallocHost(&p, size) : cudaMalloc(&p, size);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw Error{SLAB_E_OOM, std::string(what) + " of " + std::to_string(bytes) + " bytes failed: " + cudaGetErrorString(e)};
    }
    B.live[p] = Live{size, dev};
    return p;
}

void release(void* p) noexcept {
    if (!p) return;
    Blocks& B = blocks();
    std::lock_guard<std::mutex> lk(B.mu);
    const auto it = B.live.find(p);
    if (it == B.live.end()) return;
    const Live l = it->second;
    B.live.erase(it);
    try {
        Pool& pool = B.pools[l.dev];
        if (!pool.bound) {
            size_t free_b = 0, total_b = 0;
            if (l.dev == PINNED) pool.bound = PINNED_BYTES;
            else if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) pool.bound = std::max<size_t>(total_b / 16, MIB);
            else pool.bound = MIB;
        }
        if (l.size <= pool.bound) {
            pool.kept.emplace(l.size, Kept{p, ++B.releases});
            pool.bytes += l.size;
            trim(l.dev, pool, pool.bound);
            return;
        }
    } catch (...) {  // no room for the bookkeeping: back to the driver
    }
    driver_free(l.dev, p);
}

}  // namespace

void* take_device(size_t bytes) {
    int dev = 0;
    SLAB_CUDA(cudaGetDevice(&dev));
    return take(dev, bytes, "cudaMalloc");
}
void release_device(void* p) noexcept { release(p); }
void* take_pinned(size_t bytes) { return take(PINNED, bytes, "cudaMallocHost"); }
void release_pinned(void* p) noexcept { release(p); }

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
    std::lock_guard<std::mutex> lk(B.mu);
    if (--B.users == 0)
        for (auto& kv : B.pools) trim(kv.first, kv.second, kv.first == PINNED ? IDLE_BYTES / 4 : IDLE_BYTES);
}

}  // namespace slab
