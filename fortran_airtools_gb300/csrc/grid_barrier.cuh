// grid_barrier.cuh -- cooperative launches and a barrier of all their blocks.
#pragma once

#include <cuda_runtime.h>

namespace fair {

// A barrier of all blocks of a cooperative launch on one counter, gbar[0]
// (zero at the launch): block 0 adds 2^31 - (blocks - 1), every other block
// 1, so the counter's top bit flips exactly when the last block arrives -- one
// reduction per block, nothing to reset (the counter wraps) and, the barriers
// being counted (phase: the top bit before this one), no value to wait for.
// The arrival releases the block's earlier writes; the waiting thread
// reads the counter with acquire semantics. A block that waits more than
// kGridSpinLimit polls, or sees *gerr set (checked every 1024 polls), sets
// *gerr and returns false; the kernel then stops, and the host reports the
// error.
constexpr unsigned long long kGridSpinLimit = 1ull << 26;

__device__ __forceinline__ bool grid_barrier(unsigned *gbar, int *gerr, unsigned phase) {
    __shared__ int ok_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned add = blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1u) : 1u;
        int ok = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(gbar), "r"(add) : "memory");
        for (unsigned long long it = 1;; ++it) {
            unsigned cur;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(gbar) : "memory");
            if ((cur >> 31) != phase) break;
            if ((it & 1023u) == 0 && (it > kGridSpinLimit || *(volatile int *)gerr)) {
                atomicExch(gerr, 1);
                ok = 0;
                break;
            }
        }
        ok_s = ok;
    }
    __syncthreads();
    return ok_s != 0;
}

// Launches `kern` cooperatively; false, and nothing launched, where that is refused
// (its blocks cannot all be resident at once).
template <class K, class... A>
bool launch_cooperative(int blocks, int threads, cudaStream_t s, K kern, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, kern, args...) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

}  // namespace fair
