/* Stands before the CUDA runtime (LD_PRELOAD): a device with less memory, and one
 * that refuses cooperative launches. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <stddef.h>

#define SLOTS 65536
static struct { void *p; size_t n; } held[SLOTS];
static size_t used, peak, limit;
static long refused, allocs, copies;
static int no_cooperative;

void fake_limit(size_t bytes) { limit = bytes; }
void fake_no_cooperative(int on) { no_cooperative = on; }
size_t fake_used(void) { return used; }
size_t fake_peak(int reset) {
    const size_t p = peak;
    if (reset) peak = used;
    return p;
}
long fake_refused(void) { return refused; }
long fake_allocs(void) { return allocs; }
long fake_copies(void) { return copies; }

static void *next(const char *name) { return dlsym(RTLD_NEXT, name); }

cudaError_t cudaMalloc(void **p, size_t n) {
    if (limit && used + n > limit) {
        ++refused;
        *p = NULL;
        return cudaErrorMemoryAllocation;
    }
    const cudaError_t e = ((cudaError_t(*)(void **, size_t))next("cudaMalloc"))(p, n);
    if (e != cudaSuccess) return e;
    ++allocs;
    used += n;
    if (used > peak) peak = used;
    for (int i = 0; i < SLOTS; ++i)
        if (!held[i].p) {
            held[i].p = *p;
            held[i].n = n;
            break;
        }
    return e;
}

cudaError_t cudaFree(void *p) {
    if (p)
        for (int i = 0; i < SLOTS; ++i)
            if (held[i].p == p) {
                used -= held[i].n;
                held[i].p = NULL;
                break;
            }
    return ((cudaError_t(*)(void *))next("cudaFree"))(p);
}

cudaError_t cudaMemcpy(void *dst, const void *src, size_t n, enum cudaMemcpyKind kind) {
    ++copies;
    return ((cudaError_t(*)(void *, const void *, size_t, enum cudaMemcpyKind))next("cudaMemcpy"))(dst, src, n, kind);
}

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *cfg, const void *f, void **args) {
    if (no_cooperative)
        for (unsigned i = 0; i < cfg->numAttrs; ++i)
            if (cfg->attrs[i].id == cudaLaunchAttributeCooperative && cfg->attrs[i].val.cooperative) {
                ++refused;
                return cudaErrorCooperativeLaunchTooLarge;
            }
    return ((cudaError_t(*)(const cudaLaunchConfig_t *, const void *, void **))next("cudaLaunchKernelExC"))(cfg, f,
                                                                                                         args);
}
