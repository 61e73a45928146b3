// k_bptt.cu -- the adjoint of the time loop with the boundary network on the boundary nodes
// (layer 0), for training the network through it (sem_abc_bptt).
//
// Forward (stored levels; c = p^n after the source, q = p^{n-1}, s = (sx*sz)*sy per node):
//   interior i:  out_i = s_i ((2 c_i - s_i q_i) - a_i (K c)_i)            (the stencil pass)
//   boundary b:  out_b = N(f_b),  N(f) = scale clip(MLP(f / scale), -1, 1),  scale = max_k |f_k|
//   with the 81 features of b over its 3x3x3 neighbourhood j (the face kernel's):
//     level 0: out_j (j not on the boundary) or s_j (s_j q_j) (j on the boundary: what the step
//              leaves there before the network), level 1: s_j c_j, level 2: s_j q_j.
// Backward, with A0, A1, A2 the adjoints of out^m, out^{m-1}, out^{m-2} (complete for out^m):
//   1. (mlp_boundary_grad, k_mlp_train.cu) g_b = A0_b; dy_b = g_b scale_b [|y_b| < 1] (N = scale h);
//      the network's backward gives
//      the parameter gradient and dx = dy dy/dx; with d = dx / scale = g dh/dx
//      (h = clip(MLP(x)), x = f / scale) the feature gradient is
//      G_k = d_k + [k = k*] sgn(f_k*) (g h - sum_m x_m d_m)   (scale = |f_k*|);
//   2. (bptt_scatter) G is gathered back (a node collects from the boundary nodes whose neighbourhood holds it,
//      in a fixed order): level 0 -> A0 (j not on the boundary) or s_j^2 A2; level 1 -> s_j A1;
//      level 2 -> s_j A2;
//   3. (bptt_interior) interior adjoint with lambda = A0 on interior nodes and v = a s lambda:
//      A1_j += 2 s_j lambda_j - (K^T v)_j,  A2_j -= s_j^2 lambda_j.
// K^T is gathered from the rows of K (K_ij from node i's local indices and weights), so the
// rows of the domain's boundary nodes, which the forward never forms, are not needed.
#include <cuda_runtime.h>

#include <algorithm>

#include "launch.cuh"
#include "mlp.h"

namespace semgb {

namespace {

struct Geo {
    int nx, ny, nz;
    int64_t nxp;
    const float *sx, *sy, *sz;  // null: no sponge
};

__device__ __forceinline__ void coords_of(const Geo &g, int64_t q, int &ix, int &iy, int &iz)
{
    const int64_t plane = g.nxp * g.nz;
    iy = (int)(q / plane);
    const int64_t r = q - (int64_t)iy * plane;
    iz = (int)(r / g.nxp);
    ix = (int)(r - (int64_t)iz * g.nxp);
}

__device__ __forceinline__ int64_t index_of(const Geo &g, int ix, int iy, int iz)
{
    return ix + (int64_t)iz * g.nxp + (int64_t)iy * g.nxp * g.nz;
}

__device__ __forceinline__ float sponge_of(const Geo &g, int ix, int iy, int iz)
{
    return g.sx ? (g.sx[ix] * g.sz[iz]) * g.sy[iy] : 1.f;
}

__device__ __forceinline__ bool inside(const Geo &g, int ix, int iy, int iz)
{
    return ix >= 0 && ix < g.nx && iy >= 0 && iy < g.ny && iz >= 0 && iz < g.nz;
}

__device__ __forceinline__ bool on_boundary(const Geo &g, int ix, int iy, int iz)
{
    return ix == 0 || ix == g.nx - 1 || iy == 0 || iy == g.ny - 1 || iz == 0 || iz == g.nz - 1;
}

// Gather, then v.  The first blocks take the shell (nodes within one of the boundary: only these lie
// in a boundary node's neighbourhood), 64 nodes each with one thread per node and level; the other
// blocks the rest of the box, which only needs v = a s lambda on interior nodes (lambda = A0), zero
// elsewhere.  Bound by the latency of two dependent loads (the neighbour's boundary index, its
// gradient): the shell list keeps full warps on it, a thread's 27 loads of each kind are in flight
// together and three threads share a node (15.2 us at 49^3 nodes over all nodes with one thread
// each, 10 with the list and one thread per node).
constexpr int kShellNodes = 64;
__global__ void __launch_bounds__(3 * kShellNodes) k_bptt_gather(const Geo g, int64_t n_int, const int64_t *shell,
                                                                 int64_t n_shell, int shell_blocks, const int *sidx,
                                                                 const float *G, int64_t gs, const float *am,
                                                                 float *a0, float *a1, float *a2, float *v)
{
    int jx, jy, jz;
    if ((int)blockIdx.x >= shell_blocks) {
        const int64_t q = (int64_t)(blockIdx.x - shell_blocks) * (3 * kShellNodes) + threadIdx.x;
        const float am_q = q < n_int ? am[q] : 0.f;
        grid_dependency_wait();
        if (q >= n_int) return;
        coords_of(g, q, jx, jy, jz);
        if (jx >= g.nx) v[q] = 0.f;  // padding column
        if (jx <= 1 || jx >= g.nx - 2 || jy <= 1 || jy >= g.ny - 2 || jz <= 1 || jz >= g.nz - 2) return;
        v[q] = am_q * sponge_of(g, jx, jy, jz) * a0[q];
        return;
    }
    __shared__ float sum[3][kShellNodes];
    const int l = threadIdx.x / kShellNodes, u = threadIdx.x % kShellNodes;
    const int64_t i = (int64_t)blockIdx.x * kShellNodes + u;
    const int64_t q = i < n_shell ? shell[i] : 0;
    coords_of(g, q, jx, jy, jz);
    // j = b + (dx, dy, dz): the gradients of the 27 boundary nodes b around j, in a fixed order
    int sb[27];
#pragma unroll
    for (int o = 0; o < 27; o++) {
        const int bx = jx - (o % 3 - 1), by = jy - ((o / 3) % 3 - 1), bz = jz - (o / 9 - 1);
        sb[o] = inside(g, bx, by, bz) ? sidx[index_of(g, bx, by, bz)] : -1;
    }
    grid_dependency_wait();
    float t[27], s = 0.f;
#pragma unroll
    for (int o = 0; o < 27; o++) t[o] = sb[o] >= 0 ? G[(27 * l + o) * gs + sb[o]] : 0.f;
#pragma unroll
    for (int o = 0; o < 27; o++) s += t[o];
    sum[l][u] = s;
    __syncthreads();
    if (l != 0 || i >= n_shell) return;
    const float sj = sponge_of(g, jx, jy, jz);
    const float s0 = s, s1 = sum[1][u], s2 = sum[2][u];
    float n2 = a2[q], lam = 0.f;
    const bool bj = on_boundary(g, jx, jy, jz);
    if (bj) {
        n2 += sj * sj * s0;
    } else {
        lam = a0[q] + s0;
        a0[q] = lam;
    }
    a1[q] += sj * s1;
    a2[q] = n2 + sj * s2;
    v[q] = bj ? 0.f : am[q] * sj * lam;
}

// Interior adjoint: A1 += 2 s lambda - K^T v, A2 -= s^2 lambda; A0 is cleared behind it (it is the
// newest level's adjoint two steps on), and the loss gradient of the level that becomes the
// newest, 2 (out - ref) on the region of interest, added to A1 (ridx: index in the region, -1
// elsewhere; null: not added here).  K^T v is summed in order of d, its x, z and y terms in turn; the
// row's coefficients come from shared memory by the node's own local index
// (t[l][d]: row (l - d) mod O of the operator).  Order a template argument: the 6O + 1 loads are
// in flight together (12.4 us at 49^3 nodes with run-time order and indices).
template <int O>
__global__ void __launch_bounds__(128) k_bptt_interior(const Geo g, int64_t n_int, const BpttOperator op,
                                                       const float *v, float *a0, float *a1, float *a2,
                                                       const int *ridx, const float *out, const float *ref)
{
    constexpr int W = 2 * O + 1;
    __shared__ float t[O][W], wa[O];
    if (threadIdx.x < O * W) {
        const int l = threadIdx.x / W, d = threadIdx.x % W - O;
        t[l][d + O] = op.T[((l - d + 2 * O) % O) * W + d + O];
    }
    if (threadIdx.x < O) wa[threadIdx.x] = op.wa[threadIdx.x];
    __syncthreads();
    const int64_t q = (int64_t)blockIdx.x * 128 + threadIdx.x;
    if (q >= n_int) return;
    int jx, jy, jz;
    coords_of(g, q, jx, jy, jz);
    grid_dependency_wait();
    if (jx >= g.nx) return;
    const int lx = jx % O, ly = jy % O, lz = jz % O;
    const int64_t pl = g.nxp * g.nz;
    const float cx = op.g[0] * (wa[lz] * wa[ly]), cz = wa[lx] * (op.g[1] * wa[ly]), cy = wa[lx] * (op.g[2] * wa[lz]);
    float vx[W], vz[W], vy[W];
#pragma unroll
    for (int d = -O; d <= O; d++) {
        vx[d + O] = jx - d >= 0 && jx - d < g.nx ? v[q - d] : 0.f;
        vz[d + O] = jz - d >= 0 && jz - d < g.nz ? v[q - (int64_t)d * g.nxp] : 0.f;
        vy[d + O] = jy - d >= 0 && jy - d < g.ny ? v[q - (int64_t)d * pl] : 0.f;
    }
    float acc = 0.f;
#pragma unroll
    for (int d = 0; d < W; d++) {
        acc = fmaf(cx * t[lx][d], vx[d], acc);
        acc = fmaf(cz * t[lz][d], vz[d], acc);
        acc = fmaf(cy * t[ly][d], vy[d], acc);
    }
    const bool in = jx > 0 && jx < g.nx - 1 && jy > 0 && jy < g.ny - 1 && jz > 0 && jz < g.nz - 1;
    const float sj = sponge_of(g, jx, jy, jz);
    const float lam = in ? a0[q] : 0.f;
    float n1 = a1[q] + (2.f * sj * lam - acc);
    if (ridx) {
        const int r = ridx[q];
        if (r >= 0) n1 += 2.f * (out[q] - ref[r]);
    }
    a1[q] = n1;
    a2[q] -= sj * sj * lam;
    a0[q] = 0.f;
}

// Loss gradient 2 (out - ref) of one level into its adjoint (atomic: a node may be listed twice)
__global__ void k_bptt_seed(const int64_t *roi, int n_roi, const float *out, const float *ref, float *a0)
{
    grid_dependency_wait();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n_roi) atomicAdd(a0 + roi[r], 2.f * (out[roi[r]] - ref[r]));
}

// loss sum_r (out_r - ref_r)^2 of every step, one block per step (fixed-order reduction)
__global__ void __launch_bounds__(1024) k_bptt_loss(const int64_t *roi, int n_roi, const float *levels, int64_t stride,
                                                    const float *ref, double *loss)
{
    __shared__ double part[1024];
    const float *out = levels + blockIdx.x * stride;
    ref += (int64_t)blockIdx.x * n_roi;
    double acc = 0.0;
    for (int r = threadIdx.x; r < n_roi; r += blockDim.x) {
        const float e = out[roi[r]] - ref[r];
        acc += (double)e * e;
    }
    part[threadIdx.x] = acc;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) part[threadIdx.x] += part[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) loss[blockIdx.x] = part[0];
}

__global__ void k_bptt_copy(const float *src, float *dst, int64_t n4)
{
    grid_dependency_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x)
        reinterpret_cast<float4 *>(dst)[i] = reinterpret_cast<const float4 *>(src)[i];
}

}  // namespace

cudaError_t bptt_scatter(const BpttFields &f, const float *a_mass, cudaStream_t s)
{
    const Geo g{f.nx, f.ny, f.nz, f.nxp, f.sx, f.sy, f.sz};
    const int sb = (int)((f.n_shell + kShellNodes - 1) / kShellNodes);
    const int nb = (int)((f.n_int + 3 * kShellNodes - 1) / (3 * kShellNodes));
    return launch_after(k_bptt_gather, dim3((unsigned)(sb + nb)), 3 * kShellNodes, 0, s, true, g, f.n_int, f.shell, f.n_shell, sb,
                        f.sidx, f.dx, f.dx_stride, a_mass, f.a[0], f.a[1], f.a[2], f.v);
}

cudaError_t bptt_interior(const BpttFields &f, const BpttOperator &op, const float *next_out, const float *next_ref,
                          cudaStream_t s)
{
    const Geo g{f.nx, f.ny, f.nz, f.nxp, f.sx, f.sy, f.sz};
    const dim3 grid((unsigned)((f.n_int + 127) / 128));
    const int *ridx = next_out ? f.ridx : nullptr;
    auto go = [&](auto kernel) {
        return launch_after(kernel, grid, 128, 0, s, true, g, f.n_int, op, f.v, f.a[0], f.a[1], f.a[2], ridx, next_out,
                            next_ref);
    };
    switch (op.order) {
    case 1: return go(k_bptt_interior<1>);
    case 2: return go(k_bptt_interior<2>);
    case 3: return go(k_bptt_interior<3>);
    case 4: return go(k_bptt_interior<4>);
    case 5: return go(k_bptt_interior<5>);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t bptt_seed(const BpttFields &f, const float *out, const float *ref, cudaStream_t s)
{
    if (f.n_roi <= 0) return cudaSuccess;
    return launch_after(k_bptt_seed, dim3((unsigned)((f.n_roi + 255) / 256)), 256, 0, s, true, f.roi, f.n_roi, out, ref,
                        f.a[0]);
}

cudaError_t bptt_losses(const BpttFields &f, const float *levels, int64_t stride, const float *ref, int n_steps,
                        double *loss, cudaStream_t s)
{
    k_bptt_loss<<<n_steps, 1024, 0, s>>>(f.roi, f.n_roi, levels, stride, ref, loss);
    return cudaGetLastError();
}

cudaError_t bptt_copy_level(const float *src, float *dst, int64_t n, cudaStream_t s)
{
    return launch_after(k_bptt_copy, dim3((unsigned)std::min<int64_t>((n / 4 + 255) / 256, 152 * 8)), 256, 0, s, true,
                        src, dst, n / 4);
}

}  // namespace semgb
