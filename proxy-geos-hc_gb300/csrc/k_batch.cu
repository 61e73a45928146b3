// k_batch.cu -- source injection of the many-shot form.  Shot s's source adds
// dt^2 c_e^2 r_s(t_n) at local node 0 of its element (SEMsolver.cpp:39-43 for one shot) in its
// own field of the shot-stacked level.  Launched once per run of steps; between, the pass adds
// the next step's sources itself (StencilArgs::inject).
#include <cuda_runtime.h>

#include "batch.h"
#include "launch.cuh"

namespace semgb {

namespace {

// One block; the step counter advances to the next source launch (ctr[1]: this step).
__global__ void k_batch_source(const BatchSourceArgs a)
{
    grid_launch_dependents();
    const int n = a.ctr[0];
    __syncthreads();  // every thread has read the step before thread 0 advances the counter
    if (n < a.nsamples)
        for (int s = threadIdx.x; s < a.nshot; s += blockDim.x)
            if (a.node[s] >= 0)
                a.cur[(int64_t)s * a.shot_stride + a.node[s]] += a.coef[s] * a.wavelet[(int64_t)s * a.nsamples + n];
    if (threadIdx.x == 0) {
        a.ctr[1] = n;
        a.ctr[0] = n + a.advance;
    }
}

}  // namespace

cudaError_t launch_batch_source(const BatchSourceArgs &a, cudaStream_t st)
{
    k_batch_source<<<1, 256, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace semgb
