// A kernel's opt-in to more dynamic shared memory than the default.  The limit belongs to the
// kernel on one device, not to a launch: it is raised per (kernel, device), by the first
// launch that needs more, and never lowered, so that launches from several threads, of several
// sizes and held in graphs stay valid.  A failed attempt is not remembered.
#pragma once

#include <cuda_runtime_api.h>

#include <map>
#include <mutex>
#include <utility>

namespace hb2
{
    // the current device's limit of `kernel` to at least `bytes`
    inline cudaError_t smem_opt_in(const void * kernel, size_t bytes)
    {
        static std::mutex mu;
        static std::map<std::pair<const void *, int>, size_t> limit;
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        std::lock_guard<std::mutex> lock(mu);
        size_t & have = limit[std::make_pair(kernel, dev)];
        if (have >= bytes) return cudaSuccess;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e == cudaSuccess) have = bytes;
        return e;
    }
}
