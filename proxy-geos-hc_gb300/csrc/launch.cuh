// launch.cuh -- launch helpers: programmatic dependent launches (the next kernel of a stream starts
// its prologue while the one before drains) and the resident CTAs of a kernel per device.
#pragma once
#include <atomic>
#include <cuda_runtime.h>

namespace semgb {

// Wait for the preceding launch of the stream to complete, its writes visible; no effect in an
// ordinary launch.  Nothing that earlier work wrote may be read before.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Let the next launch of the stream start once every CTA of this one has started (without it: once
// they have exited).  Only for launches that leave SMs idle: the passes of the step, which fill
// them, measured slower with it (the waiting CTAs of the next pass take the slots and issue time of
// the running ones: 6.4 against 4.7 us per step on 40^3 elements of order 2).
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch; dependent: as a programmatic dependent of the preceding kernel of the stream.
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, bool dependent,
                         A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

constexpr int kMaxLaunchDevices = 64;

// CTAs of the kernel resident at once on the current device; `cache` holds what was found before.
template <class K>
cudaError_t resident_ctas(K kernel, int threads, size_t smem, std::atomic<int> (&cache)[kMaxLaunchDevices], int &n)
{
    int dev = 0, sms = 152, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool known = dev >= 0 && dev < kMaxLaunchDevices;
    if (known && (n = cache[dev].load(std::memory_order_relaxed)) > 0) return cudaSuccess;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    n = sms * per_sm;
    if (known) cache[dev].store(n, std::memory_order_relaxed);
    return cudaSuccess;
}

}  // namespace semgb
