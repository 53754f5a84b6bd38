// Launch shape of a persistent kernel whose CTAs must all fit on the GPU at once.
#pragma once
#include <cuda_runtime.h>
#include <map>
#include <mutex>

namespace zl {

// The CTAs of one kernel that the current device holds at once, and the kernel's opt-in to its dynamic
// shared memory (needed above 48 KB).  Both belong to a device, so both are settled once per device of the
// process; host threads may ask at the same time.
class PersistentGrid {
public:
    // A launch of `kernel` with `threads` threads and `smem` bytes of dynamic shared memory per CTA, of
    // which at most max_per_sm may share an SM.
    cudaError_t get(const void* kernel, int threads, int smem, int max_per_sm, int* grid) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        std::lock_guard<std::mutex> lock(mu_);
        const auto known = grid_.find(dev);
        if (known != grid_.end()) {
            *grid = known->second;
            return cudaSuccess;
        }
        int sms = 0, regs_sm = 0, smem_sm = 0, reserved = 0;
        cudaFuncAttributes fa;
        if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) != cudaSuccess ||
            (e = cudaFuncGetAttributes(&fa, kernel)) != cudaSuccess)
            return e;
        // registers are allocated per warp in units of 256
        const int regs_cta = threads / 32 * ((fa.numRegs * 32 + 255) / 256 * 256);
        const int by_regs = regs_cta > 0 ? regs_sm / regs_cta : max_per_sm;
        const int by_smem = smem_sm / (int)(smem + fa.sharedSizeBytes + reserved);
        int per_sm = by_regs < by_smem ? by_regs : by_smem;
        per_sm = per_sm < max_per_sm ? per_sm : max_per_sm;
        *grid = grid_[dev] = sms * (per_sm > 0 ? per_sm : 1);
        return cudaSuccess;
    }

private:
    std::mutex mu_;
    std::map<int, int> grid_;  // by device
};

}  // namespace zl
