// noalloc.cu -- an element-path step that allocates no device memory.
//
// Some callers cannot allocate device memory while they advance the wavefield: a host code that
// hands all device memory to its own pool manager up front, or one that runs its time loop in a
// section where allocation is forbidden (a latency-critical loop, for instance).
// sem_element_step_noalloc serves them: the caller owns every input and output buffer, and the
// scratch memory the step needs -- the K.p accumulator that the element kernel scatters into --
// is a fixed array in this library's device image instead of a cudaMalloc'd buffer.  Two launches
// per call, the update as a programmatic dependent of the element kernel.
//
// The array holds kNoAllocFloats floats (16 MiB on every GPU that loads the library, held until
// the process exits); meshes up to kNoAllocMaxNodes nodes fit.  Every call uses the same array:
// two calls whose work overlaps on the GPU (different streams, or different host threads) race
// on it.
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>
#include <string>

#include "../../include/semgb.h"
#include "host_util.h"
#include "kernels.h"
#include "launch.cuh"

namespace semgb {

void set_last_error(const std::string &msg);  // api.cu

namespace {

constexpr int64_t kNoAllocFloats = int64_t(1) << 22;      // 4,194,304 floats
constexpr int64_t kNoAllocMaxNodes = kNoAllocFloats - 128;  // largest mesh

// The scratch array.  In host code this name denotes a host-side stand-in for the symbol, not a
// device address; the device address comes from cudaGetSymbolAddress.
static __device__ __align__(256) float g_noalloc_scratch[kNoAllocFloats];

constexpr int kMaxDevices = 64;
std::mutex g_mu;
float *g_scratch_dev[kMaxDevices] = {nullptr};
// The accumulator is zero between calls: the array starts as zeros and the update clears behind
// itself.  Set while a call's launches are under way, and left set if one of them fails: the next
// call on the device then clears the array first.
std::atomic<bool> g_dirty[kMaxDevices];

// Four consecutive nodes per thread (reference numbering; VEC: the caller's arrays are 16-byte
// aligned, so whole groups move as one 16-byte access).  Interior nodes:
// p_next = 2 p_cur - p_prev - coef * y, boundary nodes: p_prev; then both levels take the sponge
// factor, as the solver's sponge does after each step.  Clears y behind it for the next call.
// Bound by memory (L2 for meshes of this size): 4 reads and 3 writes of 4 bytes per node.  One
// 32-bit division pair per four nodes: with 64-bit divisions per node it took 46.6 us on 2.67 M
// nodes (order 4, 35 x 33 x 36 elements), more than the element kernel (21.9 us); a whole step,
// with the accumulator's separate clear and the coefficient table's launch gone too, 82 -> 30 us.
template <bool VEC>
__global__ void __launch_bounds__(256) k_update_ref(float *p_cur, float *p_prev, float *y, const float *coef,
                                                    const float *sx, const float *sy, const float *sz, unsigned nx,
                                                    unsigned ny, unsigned nz)
{
    const unsigned n = nx * ny * nz, i0 = (blockIdx.x * 256u + threadIdx.x) * 4u;
    grid_dependency_wait();
    grid_launch_dependents();
    if (i0 >= n) return;
    unsigned row = i0 / nx, ix = i0 - row * nx, iy = row / nz, iz = row - iy * nz;
    const bool whole = i0 + 4 <= n;
    float pc[4], q[4], yy[4], cf[4];
    auto load = [&](const float *p, float (&v)[4]) {
        if (VEC && whole) {
            const float4 t = *reinterpret_cast<const float4 *>(p + i0);
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = i0 + j < n ? p[i0 + j] : 0.f;
        }
    };
    load(p_cur, pc);
    load(p_prev, q);
    load(y, yy);
    load(coef, cf);
    float syv = 1.f, szv = 1.f;
    if (sx) { syv = sy[iy]; szv = sz[iz]; }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (i0 + j < n) {
            const bool interior = ix > 0 && ix < nx - 1 && iz > 0 && iz < nz - 1 && iy > 0 && iy < ny - 1;
            const float v = interior ? (2.f * pc[j] - q[j]) - cf[j] * yy[j] : q[j];
            q[j] = v;
            if (sx) {
                const float s = sx[ix] * syv * szv;
                q[j] = s * v;
                pc[j] = s * pc[j];
            }
            if (++ix == nx) {
                ix = 0;
                if (++iz == nz) { iz = 0; iy++; }
                if (sx && iy < ny) { syv = sy[iy]; szv = sz[iz]; }
            }
        }
    }
    auto store = [&](float *p, const float (&v)[4]) {
        if (VEC && whole) {
            *reinterpret_cast<float4 *>(p + i0) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (i0 + j < n) p[i0 + j] = v[j];
        }
    };
    const float zero[4] = {0.f, 0.f, 0.f, 0.f};
    store(p_prev, q);
    store(y, zero);
    if (sx) store(p_cur, pc);
}

// Device address of the scratch array on the current device: resolved on the first call made
// with that device current, then cached.  That first call also loads, under CUDA's lazy module
// loading, the code of every kernel the step launches and the array itself: this is the one
// point at which the entry point can make the driver allocate device memory.
int scratch_for_current_device(float **out, int &dev)
{
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        set_last_error(std::string("cudaGetDevice: ") + cudaGetErrorString(e));
        return SEM_ERR_CUDA;
    }
    if (dev < 0 || dev >= kMaxDevices) {
        set_last_error("device index out of range");
        return SEM_ERR_ARG;
    }
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_scratch_dev[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) {
            set_last_error(std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
            return SEM_ERR_CUDA;
        }
        e = element_kernel_setup();
        cudaFuncAttributes fa;
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_update_ref<true>);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_update_ref<false>);
        if (e != cudaSuccess) {
            set_last_error(std::string("element kernel set-up: ") + cudaGetErrorString(e));
            return SEM_ERR_CUDA;
        }
        g_scratch_dev[dev] = static_cast<float *>(p);
    }
    *out = g_scratch_dev[dev];
    return SEM_OK;
}

}  // namespace

}  // namespace semgb

using namespace semgb;

extern "C" int sem_element_step_noalloc(int ex, int ey, int ez, float lx, float ly, float lz, int order,
                                        const int32_t *conn, float *p_cur, float *p_prev, const float *coef,
                                        const float *sx, const float *sy, const float *sz, void *stream)
{
    Box b;
    if (!make_box(ex, ey, ez, lx, ly, lz, order, b)) {
        set_last_error("box needs ex,ey,ez >= 1, positive lengths and order 1..5");
        return SEM_ERR_ARG;
    }
    if (!conn || !p_cur || !p_prev || !coef || (!sx != !sy) || (!sx != !sz)) {
        set_last_error("NULL device buffer (the sponge factors are all given or all NULL)");
        return SEM_ERR_ARG;
    }
    if (b.n_nodes > kNoAllocMaxNodes) {
        set_last_error("mesh has " + std::to_string(b.n_nodes) + " nodes; sem_element_step_noalloc handles at most " +
                       std::to_string(kNoAllocMaxNodes) + " (the size of its fixed scratch array)");
        return SEM_ERR_ARG;
    }
    float *y = nullptr;
    int dev = 0;
    int rc = scratch_for_current_device(&y, dev);
    if (rc != SEM_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    Gll g;
    gll_tables(order, g);
    const double jx = 0.5 * lx / ex, jz = 0.5 * lz / ez, jy = 0.5 * ly / ey, detJ = jx * jz * jy;
    ElementArgs ea{};
    ea.g[0] = (float)(detJ / (jx * jx));
    ea.g[1] = (float)(detJ / (jz * jz));
    ea.g[2] = (float)(detJ / (jy * jy));
    for (int i = 0; i <= order; i++) ea.w[i] = (float)g.w[i];
    ea.conn = conn;
    ea.p = p_cur;
    ea.y = y;
    ea.n_elem = b.n_elem;
    ea.n_check = b.n_nodes;  // the caller's map: indices outside [0, n_nodes) are skipped
    element_stiffness_1d(g, ea.S);

    cudaError_t e = cudaSuccess;
    if (g_dirty[dev].exchange(true)) e = cudaMemsetAsync(y, 0, kNoAllocFloats * sizeof(float), s);
    if (e == cudaSuccess) e = launch_element(order, ea, s);
    if (e == cudaSuccess) {
        const uintptr_t bits = reinterpret_cast<uintptr_t>(p_cur) | reinterpret_cast<uintptr_t>(p_prev) |
                               reinterpret_cast<uintptr_t>(coef);
        const dim3 grid((unsigned)((b.n_nodes + 1023) / 1024));
        e = launch_after(bits & 15 ? k_update_ref<false> : k_update_ref<true>, grid, 256, 0, s, true, p_cur, p_prev, y,
                         coef, sx, sy, sz, b.nx, b.ny, b.nz);
    }
    if (e == cudaSuccess) g_dirty[dev] = false;
    if (e != cudaSuccess) {
        set_last_error(std::string("CUDA: ") + cudaGetErrorString(e));
        return SEM_ERR_CUDA;
    }
    return SEM_OK;
}
