// occupancy.cuh -- resident blocks per SM of a kernel, queried once per device.
#pragma once

#include <mutex>

#include "slcs_internal.cuh"

namespace slcs {

constexpr int MAX_DEVICES = 64;

// Resident blocks per SM of one kernel on the current device (queried once
// per kernel and device: occupancy belongs to a device, like function
// attributes).  The kernel is a template argument, so that every kernel
// keeps its own table.
template <auto Kernel>
slcs_status occupancy_of(int threads, int *occ_out, size_t smem = 0)
{
    static int per_dev[MAX_DEVICES] = {}; // 0: not queried yet
    static std::mutex mu;
    int dev = 0;
    SLCS_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(mu);
    int *slot = (dev >= 0 && dev < MAX_DEVICES) ? &per_dev[dev] : nullptr;
    if (!slot || *slot == 0) {
        int occ = 0;
        // Dynamic shared memory beyond 48 KB is opted into once per device.
        if (smem > 0)
            SLCS_CUDA(cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        SLCS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, Kernel, threads, smem));
        if (occ < 1) occ = 1;
        if (!slot) {
            *occ_out = occ;
            return SLCS_OK;
        }
        *slot = occ;
    }
    *occ_out = *slot;
    return SLCS_OK;
}

} // namespace slcs
