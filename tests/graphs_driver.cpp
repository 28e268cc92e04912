// Drives the step graphs (csrc/graphs.hpp) over a CUDA runtime made of flags:
// a stream that is or is not being captured, graphs that are or are not
// destroyed. Compiled and run by test_graphs.py; prints "ok" or the first rule
// that does not hold.
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "graphs.hpp"

#define CHECK(c)                                         \
    do {                                                 \
        if (!(c)) {                                      \
            std::printf("line %d: %s\n", __LINE__, #c);  \
            std::fflush(stdout);                         \
            std::_Exit(1);                               \
        }                                                \
    } while (0)

static bool capturing = false, invalidated = false, refuse_instance = false;
static int graphs = 0, execs = 0, launches = 0;
static cudaError_t last = cudaSuccess;
static cudaError_t fail(cudaError_t e) { return last = e; }

extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode m) {
    CHECK(m == cudaStreamCaptureModeThreadLocal);
    if (capturing) return fail(cudaErrorIllegalState);
    capturing = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    CHECK(capturing);
    capturing = false;
    *g = nullptr;
    if (invalidated) {
        invalidated = false;
        return fail(cudaErrorStreamCaptureInvalidated);
    }
    *g = reinterpret_cast<cudaGraph_t>((uintptr_t)16);
    ++graphs;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    if (refuse_instance) return fail(cudaErrorMemoryAllocation);
    *x = reinterpret_cast<cudaGraphExec_t>((uintptr_t)32);
    ++execs;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) {
    --graphs;
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) {
    --execs;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
    CHECK(!capturing);
    ++launches;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

using namespace slab;

template <typename F> static slab_status status(F f) {
    try {
        f();
    } catch (const Error& e) {
        return e.code;
    }
    return SLAB_OK;
}

int main() {
    {
        StepGraphs G;
        const cudaStream_t st = nullptr;
        int steps = 0;
        // a launch that is refused in the middle of a capture
        CHECK(status([&] { G.launch(8, st, [&] { if (++steps == 3) throw Error{SLAB_E_CUDA, "launch"}; }); }) == SLAB_E_CUDA);
        CHECK(!capturing && graphs == 0 && execs == 0 && launches == 0);
        // the same in a capture that the refusal has invalidated
        steps = 0;
        CHECK(status([&] { G.launch(8, st, [&] { if (++steps == 3) { invalidated = true; throw Error{SLAB_E_CUDA, "launch"}; } }); }) == SLAB_E_CUDA);
        CHECK(!capturing && graphs == 0 && cudaGetLastError() == cudaSuccess);
        // a capture that ends invalidated, and an instance that is refused
        CHECK(status([&] { G.launch(8, st, [&] { invalidated = true; }); }) == SLAB_E_CUDA);
        CHECK(!capturing && graphs == 0 && cudaGetLastError() == cudaSuccess);
        refuse_instance = true;
        CHECK(status([&] { G.launch(8, st, [] {}); }) == SLAB_E_OOM);
        CHECK(!capturing && graphs == 0 && G.g.empty() && cudaGetLastError() == cudaSuccess);
        refuse_instance = false;
        // afterwards the stream takes captures and launches as ever
        steps = 0;
        for (int k = 0; k < 2; ++k) G.launch(8, st, [&] { ++steps; });
        G.launch(8, st, [&] { ++steps; }, 1);
        CHECK(steps == 16 && execs == 2 && graphs == 0 && launches == 3);
    }
    CHECK(execs == 0);
    std::puts("ok");
}
