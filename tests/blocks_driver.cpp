// Drives the kept memory blocks (csrc/blocks.cu) over a CUDA runtime made of
// counters: addresses without memory behind them, streams that are busy with
// blocks until they are waited for, a device of a given size. Compiled and run
// by test_blocks.py; prints "ok" or the first rule that does not hold.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <random>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "blocks.hpp"
#include "error.hpp"

#define CHECK(c)                                                       \
    do {                                                               \
        if (!(c)) {                                                    \
            std::printf("line %d: %s\n", __LINE__, #c);                \
            std::fflush(stdout);                                       \
            std::_Exit(1);                                             \
        }                                                              \
    } while (0)

namespace {

constexpr size_t MIB = (size_t)1 << 20, GIB = (size_t)1 << 30;

struct Fake {
    std::recursive_mutex mu;
    size_t total = 160 * GIB, used = 0, pinned = 0;
    uintptr_t next = (uintptr_t)1 << 40;
    std::map<void*, size_t> dev, host;            // what the driver has handed out
    std::map<cudaStream_t, std::set<void*>> busy;  // work in flight
    std::map<cudaStream_t, int> waits;
    int mallocs = 0, frees = 0, device = 0;
    std::vector<void*> freed;
} F;

cudaStream_t stream(int k) { return reinterpret_cast<cudaStream_t>((uintptr_t)0x1000 + 16 * k); }
void work(cudaStream_t s, void* p) {
    std::lock_guard<std::recursive_mutex> lk(F.mu);
    F.busy[s].insert(p);
}
bool busy_elsewhere(cudaStream_t own, void* p) {
    std::lock_guard<std::recursive_mutex> lk(F.mu);
    for (const auto& kv : F.busy)
        if (kv.first != own && kv.second.count(p)) return true;
    return false;
}

cudaError_t give(std::map<void*, size_t>& m, size_t& used, size_t total, void** p, size_t n) {
    std::lock_guard<std::recursive_mutex> lk(F.mu);
    ++F.mallocs;
    if (used + n > total) return cudaErrorMemoryAllocation;
    used += n;
    *p = reinterpret_cast<void*>(F.next);
    F.next += n + 4096;
    m[*p] = n;
    return cudaSuccess;
}
cudaError_t take_back(std::map<void*, size_t>& m, size_t& used, void* p) {
    std::lock_guard<std::recursive_mutex> lk(F.mu);
    CHECK(m.count(p) == 1);
    used -= m[p];
    m.erase(p);
    ++F.frees;
    F.freed.push_back(p);
    for (auto& kv : F.busy) kv.second.erase(p);  // the driver waits by itself
    return cudaSuccess;
}

}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return give(F.dev, F.used, F.total, p, n); }
cudaError_t cudaFree(void* p) { return take_back(F.dev, F.used, p); }
cudaError_t cudaMallocHost(void** p, size_t n) { return give(F.host, F.pinned, 64 * GIB, p, n); }
cudaError_t cudaFreeHost(void* p) { return take_back(F.host, F.pinned, p); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> lk(F.mu);
    F.busy[s].clear();
    ++F.waits[s];
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {  // refused while another thread captures: nothing here may need it
    CHECK(!"a wait for the whole device");
    return cudaErrorStreamCaptureUnsupported;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    std::lock_guard<std::recursive_mutex> lk(F.mu);
    *f = F.total - F.used;
    *t = F.total;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = F.device;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

using namespace slab;

static void same_scope() {
    const MemoryUser u;
    BlockScope s(stream(1));
    void* a = take_device(3 * MIB);
    work(stream(1), a);
    release_device(a);
    void* b = take_device(3 * MIB);  // the same stream's later work may use it at once
    CHECK(a == b);
    CHECK(F.waits[stream(1)] == 0);
    release_device(b);
    void* c = take_device(2 * MIB);  // 4 MiB held for 2 asked: more than a quarter too large
    CHECK(c != a);
    release_device(c);
    void* d = take_device(100 * MIB);
    release_device(d);
    void* e = take_device(90 * MIB);
    CHECK(e == d);
    release_device(e);
    e = take_device(82 * MIB);  // a quarter, but more than 16 MiB
    CHECK(e != d);
    release_device(e);
}

static void other_scope() {
    const MemoryUser u;
    void *a, *h;
    {
        BlockScope s(stream(2));
        a = take_device(5 * MIB);
        h = take_pinned(5 * MIB);
        work(stream(2), a);
        work(stream(2), h);
        release_device(a);
        release_pinned(h);
        std::thread([&] {  // held back from everybody else while the scope lasts
            BlockScope t(stream(3));
            void* b = take_device(5 * MIB);
            CHECK(b != a);
            work(stream(3), b);
            release_device(b);
        }).join();
        CHECK(F.waits[stream(2)] == 0);
    }
    CHECK(F.waits[stream(2)] == 1);  // once for both
    BlockScope t(stream(4));
    void *b = take_device(5 * MIB), *g = take_pinned(5 * MIB);
    CHECK(F.dev.count(b) && F.host.count(g));
    CHECK(!busy_elsewhere(stream(4), b) && !busy_elsewhere(stream(4), g));
    CHECK(g == h);
    release_device(b);
    release_pinned(g);
}

static void no_scope() {
    const MemoryUser u;
    void* a = take_device(7 * MIB);
    work(stream(5), a);
    release_device(a);
    CHECK(!F.dev.count(a));  // to the driver, which waits
    void* b;
    {
        BlockScope s(nullptr);  // stream not known: the same
        b = take_device(7 * MIB);
        release_device(b);
    }
    CHECK(!F.dev.count(b));
    release_device(nullptr);
    int x;
    release_device(&x);  // not one of these blocks: left alone
}

static void bounds() {
    {
        const MemoryUser u;
        BlockScope s(stream(6));
        std::vector<void*> v;
        for (int k = 0; k < 40; ++k) v.push_back(take_device(512 * MIB));
        void* big = take_device(11 * GIB);  // above the bound by itself
        for (void* p : v) release_device(p);
        release_device(big);
        s.flush();
        CHECK(kept_device_bytes() <= 4 * GIB && kept_device_bytes() > 4 * GIB - 512 * MIB);
        CHECK(!F.dev.count(big));
        CHECK(!F.dev.count(v.front()) && F.dev.count(v.back()));  // the oldest went
        void* h[5];
        for (void*& p : h) p = take_pinned(300 * MIB);
        for (void* p : h) release_pinned(p);
        s.flush();
        CHECK(F.pinned <= GIB && F.pinned > 0);
    }
    CHECK(F.used <= GIB && F.pinned <= GIB / 4);  // the last context is gone
}

static void failed_allocation() {
    const MemoryUser u;
    BlockScope s(stream(7));
    void* a = take_device(2 * GIB);
    release_device(a);  // still held by the scope
    {
        std::lock_guard<std::recursive_mutex> lk(F.mu);
        F.total = F.used + GIB;
    }
    void* b = take_device(3 * GIB);  // fits once the held block is back at the driver
    CHECK(!F.dev.count(a) && kept_device_bytes() == 0);
    bool refused = false;
    const int before = F.mallocs;
    try {
        take_device(8 * GIB);
    } catch (const Error& e) {
        refused = e.code == SLAB_E_OOM && e.msg.find("8589934592") != std::string::npos;
    }
    CHECK(refused && F.mallocs == before + 1);  // nothing kept: not tried twice
    release_device(b);
    s.flush();
    F.total = 160 * GIB;
}

static void trimmed() {
    {
        const MemoryUser u;
        BlockScope s(stream(8));
        void *a = take_device(GIB), *h = take_pinned(64 * MIB), *live = take_device(GIB);
        release_device(a);
        release_pinned(h);
        trim_blocks();
        CHECK(F.dev.count(a) && F.host.count(h));  // still the scope's
        s.flush();
        trim_blocks();
        CHECK(!F.dev.count(a) && !F.host.count(h) && F.dev.count(live) && kept_device_bytes() == 0);
        release_device(live);
    }
    trim_blocks();
    CHECK(F.used == 0 && F.pinned == 0);
    {
        std::lock_guard<std::recursive_mutex> lk(F.mu);
        F.total = 32 * GIB;  // a small device: 1/16 of it (the bound is asked for once per device, so of the next one)
        F.device = 1;
    }
    {
        const MemoryUser u;
        BlockScope s(stream(9));
        std::vector<void*> v;
        for (int k = 0; k < 12; ++k) v.push_back(take_device(256 * MIB));
        for (void* p : v) release_device(p);
        s.flush();
        CHECK(kept_device_bytes() == 2 * GIB);
    }
    trim_blocks();
    F.total = 160 * GIB;
    F.device = 0;
}

static void threads() {
    const MemoryUser u;
    std::mutex mu;
    std::set<void*> out;  // handed out and not released
    std::vector<std::thread> th;
    for (int t = 0; t < 8; ++t)
        th.emplace_back([&, t] {
            std::mt19937 rng(t);
            const cudaStream_t st = stream(100 + t);
            for (int call = 0; call < 200; ++call) {
                BlockScope s(st);
                std::vector<void*> mine;
                for (int k = 0; k < 20; ++k) {
                    if (mine.empty() || rng() % 2) {
                        void* p = rng() % 4 ? take_device((size_t)1 << (rng() % 30)) : take_pinned((size_t)1 << (rng() % 24));
                        CHECK(!busy_elsewhere(st, p));
                        {
                            std::lock_guard<std::mutex> lk(mu);
                            CHECK(out.insert(p).second);
                        }
                        work(st, p);
                        mine.push_back(p);
                    } else {
                        void* p = mine.back();
                        mine.pop_back();
                        {
                            std::lock_guard<std::mutex> lk(mu);
                            out.erase(p);
                        }
                        release_device(p);
                    }
                }
                for (void* p : mine) {
                    {
                        std::lock_guard<std::mutex> lk(mu);
                        out.erase(p);
                    }
                    release_device(p);
                }
            }
        });
    for (auto& t : th) t.join();
}

int main() {
    same_scope();
    other_scope();
    no_scope();
    bounds();
    failed_allocation();
    trimmed();
    threads();
    CHECK(F.used <= GIB && F.pinned <= GIB / 4);
    for (const auto& kv : F.waits) CHECK(kv.first != nullptr);  // never the default stream
    std::puts("ok");
}
