// CUDA graphs of `chunk` consecutive steps, one per chunk size and kind of step used.
#pragma once

#include <cuda_runtime.h>

#include <functional>
#include <map>
#include <utility>

#include "error.hpp"

namespace slab {

struct StepGraphs {
    std::map<std::pair<int, int>, cudaGraphExec_t> g;
    ~StepGraphs() { clear(); }
    void clear() {
        for (auto& kv : g) cudaGraphExecDestroy(kv.second);
        g.clear();
    }
    void launch(int chunk, cudaStream_t st, const std::function<void()>& one_step, int kind = 0) {
        const std::pair<int, int> key{chunk, kind};
        auto it = g.find(key);
        if (it == g.end()) it = g.emplace(key, capture(chunk, st, one_step)).first;
        SLAB_CUDA(cudaGraphLaunch(it->second, st));
    }

  private:
    // Whatever fails in between, the stream is out of its capture afterwards
    // (inside one it would refuse every later call) and the error is not left
    // for the next check of a launch to find.
    static cudaGraphExec_t capture(int chunk, cudaStream_t st, const std::function<void()>& one_step) {
        cudaGraph_t gr = nullptr;
        SLAB_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        try {
            for (int k = 0; k < chunk; ++k) one_step();
        } catch (...) {
            if (cudaStreamEndCapture(st, &gr) == cudaSuccess && gr) cudaGraphDestroy(gr);
            cudaGetLastError();
            throw;
        }
        cudaGraphExec_t ex = nullptr;
        cudaError_t e = cudaStreamEndCapture(st, &gr);
        if (e == cudaSuccess) {
            e = cudaGraphInstantiate(&ex, gr, 0);
            cudaGraphDestroy(gr);
        }
        if (e != cudaSuccess) cudaGetLastError();
        SLAB_CUDA(e);
        return ex;
    }
};

}  // namespace slab
