// grid_barrier.cuh -- a barrier of all blocks of a cooperative launch.
#pragma once

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

}  // namespace fair
