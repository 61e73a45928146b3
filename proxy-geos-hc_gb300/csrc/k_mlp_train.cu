// k_mlp_train.cu -- training kernels of the boundary network (mlp.h): loss and parameter gradients
// over samples, the network's part of the adjoint of the time loop, Adam.
//
// Three launches per pass over n rows (samples or boundary nodes), where one CTA per 128-row tile
// did everything before (16 CTAs for a batch of 2048 rows, 32-way shared-memory conflicts in its
// row passes, one dependent chain of 128 multiply-adds per gradient entry and thread):
//  - k_mlp_rows, row-parallel (16 or 32 rows per CTA): the forward on the tensor cores, the output
//    gradient, dZ2 and dZ1 (and, for the adjoint, the features before and the feature gradient
//    after them); writes the rows' inputs, activations and dZ for the next launch;
//  - k_mlp_outer, entry-parallel: dW = sum over the rows of dZ x input.  A CTA owns 8 or 16 hidden
//    units of one 128-row tile; a thread a block of 2 x 4 or 4 x 4 entries in registers;
//  - k_mlp_reduce: the tiles' partial sums added in order, and for training Adam and the BF16
//    weights of the next batch in the same pass.
// Every sum runs in the order of the one-CTA kernel (over the 64 units or the 128 rows of a tile
// one fused multiply-add at a time, tiles of a slot, then slots in order), so the gradients are the
// same bits: the training of the learned boundary is a feedback loop over whole runs that follows
// last-bit differences far (k_mlp.cu).
//
// Measured on GB300, minibatch of 2048 rows (16 tiles): 19.6 us per Adam step inside a training run
// (launches and the host's shuffle included) against 150 us with the one-CTA kernel, its second
// forward for dW3, and separate gather, reduction, Adam and packing launches (kernels alone 125 us);
// 7.6 + 6.5 + 7.6 us for the three launches under the profiler, which adds about 3 us to each.
// Bound by latency: one warp per scheduler in dependent phases (stage, two MMA layers, GELU, dZ),
// not by bytes (0.66 MB of samples) or multiply-adds (27 M).  The adjoint's pass over 13,826
// boundary nodes: 25 us for the rows and, the entries and sums of five steps taken together, 10 + 3
// us per step, against 350 us for the separate feature, forward, gradient and feature-gradient
// kernels; there the row kernel issues on half of all cycles and waits on its phase barriers.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "launch.cuh"
#include "mlp_device.cuh"

namespace semgb {

namespace {

constexpr int KXB = kMlpXbStride;  // row stride (bf16) of the stored inputs
constexpr int HS = H + 4;          // row stride (float) of pre-activations and dZ in shared memory
constexpr int KX4 = (kMlpIn + 3) / 4 * 4;  // inputs rounded up to whole groups of four: 84
constexpr int DXS = KX4 + 1;               // row stride of the feature gradient in shared memory

// four BF16 at p (8-byte aligned) as floats
__device__ __forceinline__ float4 bf4(const uint16_t *p)
{
    const uint2 u = *reinterpret_cast<const uint2 *>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xffff0000u));
}

// Asynchronous 16-byte copies global -> shared: all of a thread's are in flight together, so a
// block of weights or rows costs one memory latency (plain loops of loads and stores, one latency
// per few iterations: 15.4 and 13.0 us for the row and entry kernels on 2048 rows, against 7.6
// and 6.5 so).
__device__ __forceinline__ void copy16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_landed()
{
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// Weights into shared memory (copies issued; copies_landed and a barrier before use).
__device__ void copy_net(NetSmem &s, const MlpDev &net)
{
    constexpr int C1 = kMlpInPad / 8, C2 = H / 8, CB = H / 4;
    for (int i = threadIdx.x; i < H * C1; i += blockDim.x) {
        const int nn = i / C1, j = i - nn * C1;
        copy16(s.w1 + nn * KP1 + j * 8, net.w1 + i * 8);
    }
    for (int i = threadIdx.x; i < H * C2; i += blockDim.x) {
        const int nn = i / C2, j = i - nn * C2;
        copy16(s.w2 + nn * KP2 + j * 8, net.w2 + i * 8);
    }
    if (threadIdx.x < 3 * CB) {
        const int v = threadIdx.x / CB, j = (threadIdx.x - v * CB) * 4;
        copy16((v == 0 ? s.b1 : v == 1 ? s.b2 : s.w3) + j, (v == 0 ? net.b1 : v == 1 ? net.b2 : net.w3) + j);
    }
    if (threadIdx.x == 0) s.b3 = net.b3[0];
}

struct SampleRows {
    const float *x, *t;    // [..][81], [..]
    const int64_t *idx;    // row r is sample idx[r] (null: r)
    int64_t n;             // rows of the whole pass
    int64_t row0;          // first row of this launch
    int64_t rows;          // rows of this launch, whole tiles (past n: zero inputs, zero gradient)
    float inv_n;
};

// Shared memory of k_mlp_rows for NROW rows.
template <int NROW, bool BOUNDARY>
struct RowSmem {
    NetSmem net;
    alignas(16) uint16_t xs[NROW * KP1];
    alignas(16) uint16_t h1[NROW * KP2];
    alignas(16) float z1[NROW * HS];
    alignas(16) float z2[NROW * HS];
    float d[NROW];
    // boundary: features (then inputs), feature gradient, per-row scale, arg-max, node coordinates
    alignas(16) float xf[BOUNDARY ? NROW * (KX4 + 1) : 4];
    alignas(16) float dx[BOUNDARY ? NROW * (KX4 + 1) : 4];
    float scale[BOUNDARY ? NROW : 1], gb[BOUNDARY ? NROW : 1], y[BOUNDARY ? NROW : 1];
    int kstar[BOUNDARY ? NROW : 1];
    int4 at[BOUNDARY ? NROW : 1];
};

// Forward and backward of the NROW rows staged in s.xs (8 * NROW threads; the caller
// synchronises before).  out_grad(row, y) gives the output gradient of a row, called by one
// thread per row.  On return (synchronised) s.z1 holds dZ1, s.z2 dZ2, s.h1 the hidden
// activations and s.d the output gradients; g2 (global, [NROW][64]) the second layer's GELU.
template <int NROW, bool BOUNDARY, class OutGrad>
__device__ __forceinline__ void rows_backward(RowSmem<NROW, BOUNDARY> &s, float *g2, const OutGrad &out_grad)
{
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int mt = w >> 2, n0 = (w & 3) * 16;  // the warp's 16 rows and 16 hidden units of a layer
    const int a_row = mt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, a_col = (lane >> 4) * 8;
    const int b_row = lane & 7, b_col = ((lane >> 3) & 1) * 8;
    auto layer = [&](const uint16_t *in, int ki, int ks_n, const uint16_t *wt, int kw, float (&acc)[2][4]) {
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[nt][j] = 0.f;
#pragma unroll
        for (int ks = 0; ks < ks_n; ks++) {
            uint32_t a[4];
            ldsm_x4(a, in + a_row * ki + ks * 16 + a_col);
#pragma unroll
            for (int nt = 0; nt < 2; nt++) {
                uint32_t b[2];
                ldsm_x2(b, wt + (n0 + nt * 8 + b_row) * kw + ks * 16 + b_col);
                mma16816(acc[nt], a, b);
            }
        }
    };
    float acc[2][4];
    layer(s.xs, KP1, kMlpInPad / 16, s.net.w1, KP1, acc);
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = mt * 16 + g + h * 8, c = n0 + nt * 8 + q * 2;
            const float za = acc[nt][h * 2] + s.net.b1[c], zb = acc[nt][h * 2 + 1] + s.net.b1[c + 1];
            *reinterpret_cast<float2 *>(s.z1 + r * HS + c) = make_float2(za, zb);
            *reinterpret_cast<uint32_t *>(s.h1 + r * KP2 + c) = pack_bf2(gelu(za), gelu(zb));
        }
    __syncthreads();
    layer(s.h1, KP2, H / 16, s.net.w2, KP2, acc);
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = mt * 16 + g + h * 8, c = n0 + nt * 8 + q * 2;
            *reinterpret_cast<float2 *>(s.z2 + r * HS + c) =
                make_float2(acc[nt][h * 2] + s.net.b2[c], acc[nt][h * 2 + 1] + s.net.b2[c + 1]);
        }
    __syncthreads();
    // y = b3 + sum_c w3[c] GELU(z2[c]) in the forward's order: four partial sums per row, each
    // over the columns one thread of the MMA's accumulator holds
    if (tid < 4 * NROW) {
        const int r = tid >> 2;
        float part = 0.f;
#pragma unroll
        for (int nt = 0; nt < 8; nt++) {
            const int c = nt * 8 + q * 2;
            const float2 z = *reinterpret_cast<const float2 *>(s.z2 + r * HS + c);
            const float ga = gelu(z.x), gb = gelu(z.y);
            part = fmaf(s.net.w3[c], ga, part);
            part = fmaf(s.net.w3[c + 1], gb, part);
            *reinterpret_cast<float2 *>(g2 + (int64_t)r * H + c) = make_float2(ga, gb);
        }
        part += __shfl_xor_sync(0xffffffffu, part, 1);
        part += __shfl_xor_sync(0xffffffffu, part, 2);
        if (q == 0) s.d[r] = out_grad(r, part + s.net.b3);
    }
    __syncthreads();
    // dZ2 = dy w3 GELU'(z2) in place of z2
#pragma unroll
    for (int i = tid; i < NROW * H; i += 8 * NROW) {
        const int r = i / H, c = i - r * H;
        s.z2[r * HS + c] = s.d[r] * s.net.w3[c] * gelu_d(s.z2[r * HS + c]);
    }
    __syncthreads();
    // dZ1 = GELU'(z1) sum_n dZ2[n] W2[n][k] in place of z1: two rows and four units k per thread
    {
        const int r = (tid >> 4) * 2, k = (tid & 15) * 4;
        float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int n = 0; n < H; n += 4) {
            const float4 a4 = *reinterpret_cast<const float4 *>(s.z2 + r * HS + n);
            const float4 b4 = *reinterpret_cast<const float4 *>(s.z2 + (r + 1) * HS + n);
            const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float4 w4 = bf4(s.net.w2 + (n + j) * KP2 + k);
                d0[0] = fmaf(av[j], w4.x, d0[0]); d0[1] = fmaf(av[j], w4.y, d0[1]);
                d0[2] = fmaf(av[j], w4.z, d0[2]); d0[3] = fmaf(av[j], w4.w, d0[3]);
                d1[0] = fmaf(bv[j], w4.x, d1[0]); d1[1] = fmaf(bv[j], w4.y, d1[1]);
                d1[2] = fmaf(bv[j], w4.z, d1[2]); d1[3] = fmaf(bv[j], w4.w, d1[3]);
            }
        }
        float *z0 = s.z1 + r * HS + k, *z1 = z0 + HS;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            z0[j] = d0[j] * gelu_d(z0[j]);
            z1[j] = d1[j] * gelu_d(z1[j]);
        }
    }
    __syncthreads();
}

// The rows' inputs, hidden activations and dZ to the work arrays (rows rg.. of the launch).
template <int NROW, bool BOUNDARY>
__device__ __forceinline__ void store_rows(const RowSmem<NROW, BOUNDARY> &s, const MlpWork &w, int64_t rg)
{
    const int tid = threadIdx.x;
    constexpr int CX = KXB / 8, CH = H / 8, C4 = H / 4;
    for (int i = tid; i < NROW * CX; i += 8 * NROW) {
        const int r = i / CX, j = i - r * CX;
        reinterpret_cast<uint4 *>(w.xb + (rg + r) * KXB)[j] = *reinterpret_cast<const uint4 *>(s.xs + r * KP1 + j * 8);
    }
    for (int i = tid; i < NROW * CH; i += 8 * NROW) {
        const int r = i / CH, j = i - r * CH;
        reinterpret_cast<uint4 *>(w.h1 + (rg + r) * H)[j] = *reinterpret_cast<const uint4 *>(s.h1 + r * KP2 + j * 8);
    }
    for (int i = tid; i < NROW * C4; i += 8 * NROW) {
        const int r = i / C4, j = i - r * C4;
        reinterpret_cast<float4 *>(w.dz1 + (rg + r) * H)[j] = *reinterpret_cast<const float4 *>(s.z1 + r * HS + j * 4);
        reinterpret_cast<float4 *>(w.dz2 + (rg + r) * H)[j] = *reinterpret_cast<const float4 *>(s.z2 + r * HS + j * 4);
    }
    if (tid < NROW) w.dy[rg + tid] = s.d[tid];
}

template <int NROW>
__global__ void __launch_bounds__(8 * NROW) k_mlp_rows(const MlpDev net, const SampleRows a, const MlpWork wk)
{
    extern __shared__ __align__(16) unsigned char smem[];
    RowSmem<NROW, false> &s = *reinterpret_cast<RowSmem<NROW, false> *>(smem);
    grid_launch_dependents();
    const int tid = threadIdx.x;
    // the samples do not depend on the preceding launches: staged before the wait
    // (eight threads per row, its twelve loads per thread in flight together)
    auto stage = [&](int64_t rg) {
        const int r = tid >> 3, k0 = tid & 7;
        const int64_t row = a.row0 + rg + r;
        const bool in = row < a.n;
        const float *xr = a.x + (in ? (a.idx ? a.idx[row] : row) : 0) * kMlpIn;
        float v[kMlpInPad / 8];
#pragma unroll
        for (int j = 0; j < kMlpInPad / 8; j++) v[j] = in && k0 + 8 * j < kMlpIn ? xr[k0 + 8 * j] : 0.f;
#pragma unroll
        for (int j = 0; j < kMlpInPad / 8; j++) s.xs[r * KP1 + k0 + 8 * j] = f2bf(v[j]);
    };
    int64_t rg = (int64_t)blockIdx.x * NROW;
    if (rg < a.rows) stage(rg);
    grid_dependency_wait();
    copy_net(s.net, net);
    copies_landed();
    for (; rg < a.rows; rg += (int64_t)gridDim.x * NROW) {
        if (rg >= (int64_t)gridDim.x * NROW) {
            __syncthreads();  // the previous rows are stored
            stage(rg);
        }
        __syncthreads();
        rows_backward<NROW, false>(s, wk.g2 + rg * H, [&](int r, float y) {
            const int64_t row = a.row0 + rg + r;
            float e = 0.f, d = 0.f;
            if (row < a.n) {
                e = y - a.t[a.idx ? a.idx[row] : row];
                d = 2.f * e * a.inv_n;
            }
            wk.err[rg + r] = e;
            return d;
        });
        store_rows<NROW, false>(s, wk, rg);
    }
}

// The network's share of one step of the adjoint of the time loop (k_bptt.cu), per boundary node:
// the 81 features of the node from the recorded levels, divided by their largest magnitude; the
// forward; dy = g scale where the output is not clipped; the backward down to the inputs; and
// the feature gradient G = dx / scale plus the scale's share on its arg-max feature.
// A box of 12^3 elements of order 4 is one wave of 32-row CTAs, so what counts is a CTA's chain of phases:
// the node coordinates before the wait, a row's features by eight threads with all loads in flight and
// kept in registers to the inputs, dx in packed f32x2 (scalar: 21.5 us) and scaled where it is formed.
// 24.3 -> 20.1 us a launch; with a pass per phase through shared memory the features took 7 k of the 36 k cycles.
template <int NROW>
__global__ void __launch_bounds__(8 * NROW, 3) k_mlp_boundary(const MlpDev net, const BpttFields f, const float *lm,
                                                           const float *lm1, const float *lm2, const MlpWork wk,
                                                           int64_t row0, int64_t rows)
{
    extern __shared__ __align__(16) unsigned char smem[];
    RowSmem<NROW, true> &s = *reinterpret_cast<RowSmem<NROW, true> *>(smem);
    const int tid = threadIdx.x;
    copy_net(s.net, net);  // constant over the time loop: staged before the wait
    const int64_t plane = f.nxp * f.nz;
    // coordinates of a tile's nodes (the node list is constant too)
    auto place = [&](int64_t rg) {
        if (tid >= NROW) return;
        const int64_t b = row0 + rg + tid;
        int4 c = make_int4(0, 0, 0, 0);
        if (b < f.nb) {
            const int64_t q = f.nodes[b];
            const int iy = (int)(q / plane);
            const int64_t r = q - (int64_t)iy * plane;
            const int iz = (int)(r / f.nxp);
            c = make_int4((int)(r - (int64_t)iz * f.nxp), iy, iz, 1);
        }
        s.at[tid] = c;
    };
    int64_t rg = (int64_t)blockIdx.x * NROW;
    if (rg < rows) place(rg);
    copies_landed();
    grid_dependency_wait();
    for (; rg < rows; rg += (int64_t)gridDim.x * NROW) {
        if (rg >= (int64_t)gridDim.x * NROW) {
            __syncthreads();  // the previous rows are stored
            place(rg);
        }
        __syncthreads();
        // Features, eight threads per row, four neighbours of three levels each with all their loads in
        // flight: level 0 (what the step leaves before the network: s (s q) on the boundary), 1, 2.
        // Their largest magnitude and its first feature over the eight threads, then the inputs.
        {
            const int r = tid >> 3, p = tid & 7;
            const int4 c = s.at[r];
            float v[3][4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int nbh = p + 8 * j;
                const int jx = c.x + nbh % 3 - 1, jy = c.y + (nbh / 3) % 3 - 1, jz = c.z + nbh / 9 - 1;
                v[0][j] = v[1][j] = v[2][j] = 0.f;
                if (c.w && nbh < 27 && jx >= 0 && jx < f.nx && jy >= 0 && jy < f.ny && jz >= 0 && jz < f.nz) {
                    const int64_t qn = jx + (int64_t)jz * f.nxp + (int64_t)jy * plane;
                    const float sj = f.sx ? (f.sx[jx] * f.sz[jz]) * f.sy[jy] : 1.f;
                    const bool bnd = jx == 0 || jx == f.nx - 1 || jy == 0 || jy == f.ny - 1 || jz == 0 || jz == f.nz - 1;
                    const float q0 = lm[qn], q1 = lm1[qn], q2 = lm2[qn];
                    const float hq = q2 * sj;  // s q: the history the step keeps
                    v[0][j] = bnd ? hq * sj : q0;
                    v[1][j] = q1 * sj;
                    v[2][j] = hq;
                }
            }
            if (p == 7 && c.w) s.gb[r] = f.a[0][c.x + (int64_t)c.z * f.nxp + (int64_t)c.y * plane];
            float m = 0.f;
            int km = 0;  // the feature, 0x100: negative
#pragma unroll
            for (int l = 0; l < 3; l++)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (fabsf(v[l][j]) > m) { m = fabsf(v[l][j]); km = (27 * l + p + 8 * j) | (v[l][j] < 0.f ? 0x100 : 0); }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const float mo = __shfl_xor_sync(0xffffffffu, m, o);
                const int ko = __shfl_xor_sync(0xffffffffu, km, o);
                if (mo > m || (mo == m && (ko & 0xff) < (km & 0xff))) { m = mo; km = ko; }
            }
            const float sc = m + 1e-30f, inv = 1.f / sc;
            if (p == 0) {
                s.scale[r] = sc;
                // -1: an all-zero neighbourhood (the value is 0 there, its gradient taken as 0)
                s.kstar[r] = m > 0.f ? km : -1;
            }
#pragma unroll
            for (int l = 0; l < 3; l++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int k = 27 * l + p + 8 * j;
                    if (p + 8 * j < 27) {
                        const float x = v[l][j] * inv;
                        s.xf[r * DXS + k] = x;
                        s.xs[r * KP1 + k] = f2bf(x);
                    }
                }
            for (int k = kMlpIn + p; k < kMlpInPad; k += 8) s.xs[r * KP1 + k] = 0;
        }
        __syncthreads();
        rows_backward<NROW, true>(s, wk.g2 + rg * H, [&](int r, float y) {
            s.y[r] = y;
            if (!s.at[r].w) return 0.f;
            return (y > -1.f && y < 1.f) ? s.gb[r] * s.scale[r] : 0.f;
        });
        store_rows<NROW, true>(s, wk, rg);
        // dx[k] = sum_n dZ1[n] W1[n][k], divided by the scale: four rows and four inputs per thread
        if (tid < NROW / 4 * (KX4 / 4)) {
            const int r = tid / (KX4 / 4) * 4, k = tid % (KX4 / 4) * 4;
            float d[4][4], inv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                inv[i] = 1.f / s.scale[r + i];
#pragma unroll
                for (int j = 0; j < 4; j++) d[i][j] = 0.f;
            }
#pragma unroll 2
            for (int n = 0; n < H; n += 4) {
                float a[4][4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float4 v = *reinterpret_cast<const float4 *>(s.z1 + (r + i) * HS + n);
                    a[i][0] = v.x; a[i][1] = v.y; a[i][2] = v.z; a[i][3] = v.w;
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float4 w4 = bf4(s.net.w1 + (n + j) * KP1 + k);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float2 aa = make_float2(a[i][j], a[i][j]);
                        const float2 u = fma2(aa, make_float2(w4.x, w4.y), make_float2(d[i][0], d[i][1]));
                        const float2 v = fma2(aa, make_float2(w4.z, w4.w), make_float2(d[i][2], d[i][3]));
                        d[i][0] = u.x; d[i][1] = u.y; d[i][2] = v.x; d[i][3] = v.y;
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) s.dx[(r + i) * DXS + k + j] = d[i][j] * inv[i];
        }
        __syncthreads();
        // the scale's own share of the feature gradient: one thread per row, features in order
        if (tid < NROW && row0 + rg + tid < f.nb) {
            const float *xr = s.xf + tid * DXS;
            float *d = s.dx + tid * DXS;
            const int ks = s.kstar[tid];
            if (ks < 0) {
                for (int k = 0; k < kMlpIn; k++) d[k] = 0.f;
            } else {
                float xd = 0.f;
#pragma unroll 27
                for (int k = 0; k < kMlpIn; k++) xd = fmaf(xr[k], d[k], xd);
                const float h = fminf(fmaxf(s.y[tid], -1.f), 1.f);
                const float sg = (ks & 0x100) ? -1.f : 1.f;
                d[ks & 0xff] += sg * (s.gb[tid] * h - xd);
            }
        }
        __syncthreads();
        // (feature-major: the gather reads neighbouring boundary nodes together)
        for (int i = tid; i < NROW * kMlpIn; i += 8 * NROW) {
            const int k = i / NROW, r = i - k * NROW;
            if (row0 + rg + r < f.nb) f.dx[k * f.dx_stride + row0 + rg + r] = s.dx[r * DXS + k];
        }
    }
}

// Parameter gradients of tile `slot` of this launch into part[slot] (added to it unless `first`):
// hidden units NR*blockIdx.x.. of both layers.  Threads 0..83: 4 x 21 blocks of dW1, 84..147:
// 4 x 16 blocks of dW2, NR/4 units by 4 inputs each; from 160 on the bias and output-layer sums;
// the last warp of slice 0 the loss.
template <int NR>
__global__ void __launch_bounds__(NR == 16 ? 256 : 224) k_mlp_outer(const MlpWork wk, bool first)
{
    constexpr int UN = NR / 4;
    extern __shared__ __align__(16) unsigned char smem[];
    uint16_t *sx = reinterpret_cast<uint16_t *>(smem);       // [128][KXB]
    uint16_t *sh = sx + kMlpTile * KXB;                      // [128][64]
    float *s1 = reinterpret_cast<float *>(sh + kMlpTile * H);  // dZ1 of the units [128][NR]
    float *s2 = s1 + kMlpTile * NR;                          // dZ2
    float *sg = s2 + kMlpTile * NR;                          // GELU(z2)
    float *sd = sg + kMlpTile * NR;                          // dy [128]
    const int tid = threadIdx.x, nth = blockDim.x, n0 = blockIdx.x * NR, slot = blockIdx.y;
    const int64_t r0 = (int64_t)slot * kMlpTile;
    grid_launch_dependents();
    grid_dependency_wait();
    for (int i = tid; i < kMlpTile * KXB / 8; i += nth) copy16(sx + i * 8, wk.xb + r0 * KXB + i * 8);
    for (int i = tid; i < kMlpTile * H / 8; i += nth) copy16(sh + i * 8, wk.h1 + r0 * H + i * 8);
    constexpr int C = NR / 4;
    for (int i = tid; i < kMlpTile * C; i += nth) {
        const int64_t o = (r0 + i / C) * H + n0 + i % C * 4;
        copy16(s1 + i * 4, wk.dz1 + o);
        copy16(s2 + i * 4, wk.dz2 + o);
        copy16(sg + i * 4, wk.g2 + o);
    }
    if (tid < kMlpTile / 4) copy16(sd + tid * 4, wk.dy + r0 + tid * 4);
    copies_landed();
    __syncthreads();
    float *part = wk.part + (int64_t)slot * kMlpParams;
    auto put = [&](int i, float a) { part[i] = (first ? 0.f : part[i]) + a; };
    if (tid < 148) {
        const bool l1 = tid < 84;
        const int u = l1 ? tid : tid - 84, kg = l1 ? 21 : 16;
        const int un = u / kg * UN, k = u % kg * 4;
        const float *pd = (l1 ? s1 : s2) + un;
        const uint16_t *pk = (l1 ? sx : sh) + k;
        const int st = l1 ? KXB : H;
        // units in pairs, packed f32x2 (each half rounds as the scalar fused multiply-add)
        float2 a[UN / 2][4];
#pragma unroll
        for (int i = 0; i < UN / 2; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) a[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int r = 0; r < kMlpTile; r++) {
            const float4 v = bf4(pk);
            float2 d[UN / 2];
            if constexpr (UN == 2) {
                d[0] = *reinterpret_cast<const float2 *>(pd);
            } else {
#pragma unroll
                for (int i = 0; i < UN / 4; i++) {
                    const float4 t = *reinterpret_cast<const float4 *>(pd + 4 * i);
                    d[2 * i] = make_float2(t.x, t.y);
                    d[2 * i + 1] = make_float2(t.z, t.w);
                }
            }
            const float2 vx = make_float2(v.x, v.x), vy = make_float2(v.y, v.y), vz = make_float2(v.z, v.z),
                         vw = make_float2(v.w, v.w);
#pragma unroll
            for (int i = 0; i < UN / 2; i++) {
                a[i][0] = fma2(d[i], vx, a[i][0]); a[i][1] = fma2(d[i], vy, a[i][1]);
                a[i][2] = fma2(d[i], vz, a[i][2]); a[i][3] = fma2(d[i], vw, a[i][3]);
            }
            pd += NR;
            pk += st;
        }
#pragma unroll
        for (int i = 0; i < UN; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float x = i & 1 ? a[i / 2][j].y : a[i / 2][j].x;
                if (l1) {
                    if (k + j < kMlpIn) put(kOffW1 + (n0 + un + i) * kMlpIn + k + j, x);
                } else {
                    put(kOffW2 + (n0 + un + i) * H + k + j, x);
                }
            }
    } else if (tid >= 160) {
        const int u = tid - 160;
        if (u < 2 * NR) {  // db1, db2
            const float *p = u < NR ? s1 + u : s2 + u - NR;
            float a = 0.f;
#pragma unroll 8
            for (int r = 0; r < kMlpTile; r++) a += p[r * NR];
            put((u < NR ? kOffB1 + u : kOffB2 + u - NR) + n0, a);
        } else if (u < 3 * NR) {  // dw3
            const float *p = sg + u - 2 * NR;
            float a = 0.f;
#pragma unroll 8
            for (int r = 0; r < kMlpTile; r++) a = fmaf(sd[r], p[r * NR], a);
            put(kOffW3 + n0 + u - 2 * NR, a);
        } else if (u == 3 * NR && n0 == 0) {  // db3
            float a = 0.f;
#pragma unroll 8
            for (int r = 0; r < kMlpTile; r++) a += sd[r];
            put(kOffB3, a);
        }
        if (n0 == 0 && wk.lsum && tid >= nth - 32) {
            // squared errors in 32 partial sums (four rows of the tile each)
            const int l = tid & 31;
            const float *e = wk.err + r0 + l / 8 * 32 + l % 8;
            double *ls = wk.lsum + (int64_t)slot * 32 + l;
            double a = first ? 0.0 : *ls;
#pragma unroll
            for (int j = 0; j < 4; j++) a += (double)e[8 * j] * e[8 * j];
            *ls = a;
        }
    }
}

struct AdamArgs {
    float *p, *m, *v;   // master parameters and moments
    float lr, c1, c2;
    uint16_t *w1, *w2;  // the network as the kernels read it
    float *b1, *b2, *w3, *b3;
};

__device__ __forceinline__ float adam_param(const AdamArgs &o, int i, float gi)
{
    const float mi = 0.9f * o.m[i] + 0.1f * gi;
    const float vi = 0.999f * o.v[i] + 0.001f * gi * gi;
    o.m[i] = mi;
    o.v[i] = vi;
    const float p = o.p[i] - o.lr * (mi * o.c1) / (sqrtf(vi * o.c2) + 1e-8f);
    o.p[i] = p;
    return p;
}

// Parameter i of the master layout into the kernels' form (the zero padding of W1's rows is laid
// down once by k_mlp_pack).
__device__ __forceinline__ void pack_param(const AdamArgs &o, int i, float p)
{
    if (i < kOffB1) {
        const int nn = i / kMlpIn;
        o.w1[nn * kMlpInPad + i - nn * kMlpIn] = f2bf(p);
    } else if (i < kOffW2) {
        o.b1[i - kOffB1] = p;
    } else if (i < kOffB2) {
        o.w2[i - kOffW2] = f2bf(p);
    } else if (i < kOffW3) {
        o.b2[i - kOffB2] = p;
    } else if (i < kOffB3) {
        o.w3[i - kOffW3] = p;
    } else {
        o.b3[0] = p;
    }
}

// sum over the slots b (in order) of part[b][i]: added to grad[i], or (kReduceAdam) the gradient of
// one Adam step; kReduceGroups: so for each of ng consecutive groups of nb slots in turn.  The last
// block: the loss, lsum's 32 partial sums per slot as the quad leaders and warps of a tile add them,
// slots in order, into *loss (added to it unless kReduceAdam).
enum ReduceMode { kReduceAdd, kReduceGroups, kReduceAdam };
template <ReduceMode MODE>
__global__ void __launch_bounds__(128) k_mlp_reduce(const float *part, const double *lsum, int nb, int ng, double n,
                                                    float *grad, double *loss, const AdamArgs o)
{
    grid_launch_dependents();
    grid_dependency_wait();
    if (blockIdx.x == gridDim.x - 1) {
        if (!lsum) return;
        __shared__ double tile[kMlpMaxSlots];
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
        for (int b = w; b < nb; b += 4) {
            double l = lsum[(int64_t)b * 32 + lane];
            l += __shfl_xor_sync(0xffffffffu, l, 1);
            l += __shfl_xor_sync(0xffffffffu, l, 2);
            l += __shfl_xor_sync(0xffffffffu, l, 4);
            const double w1 = __shfl_sync(0xffffffffu, l, 8), w2 = __shfl_sync(0xffffffffu, l, 16),
                         w3 = __shfl_sync(0xffffffffu, l, 24);
            if (lane == 0) tile[b] = (((l + w1) + w2) + w3) / n;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double l = 0.0;
            for (int b = 0; b < nb; b++) l += tile[b];
            *loss = (MODE == kReduceAdam ? 0.0 : *loss) + l;
        }
        return;
    }
    auto slots = [&](int k, int i) {  // group k's slots of parameter i, in order
        const float *p = part + (int64_t)k * nb * kMlpParams + i;
        float a = 0.f;
        int b = 0;
        for (; b + 16 <= nb; b += 16, p += 16 * kMlpParams) {
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = p[j * kMlpParams];
#pragma unroll
            for (int j = 0; j < 16; j++) a += v[j];
        }
        for (; b < nb; b++, p += kMlpParams) a += *p;
        return a;
    };
    if constexpr (MODE == kReduceGroups) {
        // 32 parameters per block, the groups' chains of additions over its four warps (one thread
        // per parameter: 23 us for five groups of 109 slots, 13.6 us so)
        __shared__ float gsum[4][32];
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, i = blockIdx.x * 32 + lane;
        float sum = i < kMlpParams ? grad[i] : 0.f;
        for (int k0 = 0; k0 < ng; k0 += 4) {
            gsum[w][lane] = k0 + w < ng && i < kMlpParams ? slots(k0 + w, i) : 0.f;
            __syncthreads();
            for (int k = k0; k < min(k0 + 4, ng); k++) sum += gsum[k - k0][lane];
            __syncthreads();
        }
        if (w == 0 && i < kMlpParams) grad[i] = sum;
    } else {
        const int i = blockIdx.x * blockDim.x + threadIdx.x;
        if (i >= kMlpParams) return;
        if constexpr (MODE == kReduceAdam) pack_param(o, i, adam_param(o, i, 0.f + slots(0, i)));
        else grad[i] += slots(0, i);
    }
}

__global__ void k_mlp_pack(const float *m, uint16_t *w1, uint16_t *w2, float *b1, float *b2, float *w3, float *b3)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < H * kMlpInPad) {
        const int nn = i / kMlpInPad, k = i - nn * kMlpInPad;
        w1[i] = f2bf(k < kMlpIn ? m[kOffW1 + nn * kMlpIn + k] : 0.f);
    }
    if (i < H * H) w2[i] = f2bf(m[kOffW2 + i]);
    if (i < H) {
        b1[i] = m[kOffB1 + i];
        b2[i] = m[kOffB2 + i];
        w3[i] = m[kOffW3 + i];
    }
    if (i == 0) b3[0] = m[kOffB3];
}

__global__ void k_mlp_adam(const AdamArgs o, const float *g)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kMlpParams) pack_param(o, i, adam_param(o, i, g[i]));
}

AdamArgs adam_args(const MlpAdam &m)
{
    AdamArgs o{};
    o.p = m.master; o.m = m.m; o.v = m.v;
    o.lr = m.lr;
    o.c1 = 1.f / (1.f - powf(0.9f, (float)m.t));
    o.c2 = 1.f / (1.f - powf(0.999f, (float)m.t));
    o.w1 = m.w1; o.w2 = m.w2; o.b1 = m.b1; o.b2 = m.b2; o.w3 = m.w3; o.b3 = m.b3;
    return o;
}

template <int NR>
constexpr size_t smem_outer() { return kMlpTile * ((KXB + H) * sizeof(uint16_t) + (3 * NR + 1) * sizeof(float)); }

cudaError_t launch_outer(const MlpWork &w, int slots, bool first, cudaStream_t s)
{
    // 8 units per CTA (8 CTAs per tile) while 16 would leave most SMs idle (a batch of 2048 rows: 128
    // CTAs against 64); 16 beyond: twice the multiply-adds per shared load
    if (slots * 8 <= 2 * 152) return launch_after(k_mlp_outer<8>, dim3(8, slots), 224, smem_outer<8>(), s, true, w, first);
    return launch_after(k_mlp_outer<16>, dim3(4, slots), 256, smem_outer<16>(), s, true, w, first);
}

constexpr int kReduceBlocks = (kMlpParams + 127) / 128 + 1, kGroupBlocks = (kMlpParams + 31) / 32 + 1;

// Rows of a pass per round: every slot one tile.
int64_t round_rows(int64_t n) { return std::min<int64_t>((n + kMlpTile - 1) / kMlpTile, kMlpMaxSlots) * kMlpTile; }

// All rounds of a pass over samples up to the partial sums; nb: slots used.
cudaError_t sample_pass(const MlpDev &net, const float *x, const float *t, const int64_t *idx, int64_t n,
                        const MlpWork &w, int &nb, cudaStream_t s, bool dependent)
{
    SampleRows a{x, t, idx, n, 0, 0, 1.f / (float)n};
    const int64_t step = round_rows(n);
    nb = (int)(step / kMlpTile);
    for (int64_t r0 = 0; r0 < n; r0 += step) {
        a.row0 = r0;
        a.rows = round_rows(std::min(step, n - r0));
        // 16 rows per CTA spread a minibatch over the SMs; 32 share one copy of the weights
        cudaError_t e;
        if (a.rows <= 152 * 2 * 16)
            e = launch_after(k_mlp_rows<16>, dim3((unsigned)(a.rows / 16)), 128, sizeof(RowSmem<16, false>), s,
                       dependent || r0 > 0, net, a, w);
        else
            e = launch_after(k_mlp_rows<32>, dim3((unsigned)std::min<int64_t>(a.rows / 32, 152 * 4)), 256,
                       sizeof(RowSmem<32, false>), s, dependent || r0 > 0, net, a, w);
        if (e != cudaSuccess) return e;
        if ((e = launch_outer(w, (int)(a.rows / kMlpTile), r0 == 0, s)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

int64_t mlp_work_rows(int64_t n) { return n > 0 ? round_rows(n) : 0; }

cudaError_t mlp_train_setup()
{
    cudaError_t e;
    auto dyn = [](auto kernel, size_t sm) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    };
    if ((e = dyn(k_mlp_rows<16>, sizeof(RowSmem<16, false>))) != cudaSuccess) return e;
    if ((e = dyn(k_mlp_rows<32>, sizeof(RowSmem<32, false>))) != cudaSuccess) return e;
    if ((e = dyn(k_mlp_boundary<32>, sizeof(RowSmem<32, true>))) != cudaSuccess) return e;
    if ((e = dyn(k_mlp_outer<8>, smem_outer<8>())) != cudaSuccess) return e;
    return dyn(k_mlp_outer<16>, smem_outer<16>());
}

cudaError_t mlp_pack(const float *master, uint16_t *w1, uint16_t *w2, float *b1, float *b2, float *w3, float *b3,
                     cudaStream_t s)
{
    k_mlp_pack<<<(H * kMlpInPad + 255) / 256, 256, 0, s>>>(master, w1, w2, b1, b2, w3, b3);
    return cudaGetLastError();
}

cudaError_t mlp_loss_grad(const MlpDev &net, const float *x, const float *t, int64_t n, double *loss, float *grad,
                          const MlpWork &w, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    int nb = 0;
    cudaError_t e = sample_pass(net, x, t, nullptr, n, w, nb, s, false);
    if (e != cudaSuccess) return e;
    return launch_after(k_mlp_reduce<kReduceAdd>, dim3(kReduceBlocks), 128, 0, s, true, w.part, w.lsum, nb, 1, (double)n, grad, loss,
                  AdamArgs{});
}

cudaError_t mlp_train_step(const MlpDev &net, const float *x, const float *t, const int64_t *idx, int64_t n,
                           double *loss, const MlpAdam &adam, const MlpWork &w, cudaStream_t s, bool dependent)
{
    if (n <= 0) return cudaErrorInvalidValue;
    int nb = 0;
    cudaError_t e = sample_pass(net, x, t, idx, n, w, nb, s, dependent);
    if (e != cudaSuccess) return e;
    return launch_after(k_mlp_reduce<kReduceAdam>, dim3(kReduceBlocks), 128, 0, s, true, w.part, w.lsum, nb, 1, (double)n, nullptr,
                  loss, adam_args(adam));
}

static MlpWork work_at(const MlpWork &w, int64_t row)
{
    MlpWork r = w;
    r.xb += row * KXB; r.h1 += row * H; r.dz1 += row * H; r.dz2 += row * H; r.g2 += row * H; r.dy += row; r.err += row;
    r.lsum = nullptr;
    return r;
}

// Steps whose rows fit the work arrays together: one entry-parallel launch for all of them fills the
// SMs and is paid once (109 tiles alone 13.7 us, five steps' 545 tiles 52 us: the tiles' 63 KB each
// come from L2), and one reduction for all of them.
int mlp_boundary_groups(int64_t nb)
{
    const int64_t tiles = (nb + kMlpTile - 1) / kMlpTile;
    return (int)std::max<int64_t>(1, kMlpMaxSlots / std::max<int64_t>(tiles, 1));
}

cudaError_t mlp_boundary_rows(const MlpDev &net, const BpttFields &f, const float *lm, const float *lm1,
                              const float *lm2, int group, const MlpWork &w, float *grad, cudaStream_t s)
{
    if (f.nb <= 0) return cudaSuccess;
    const int64_t step = round_rows(f.nb);
    const bool rounds = step < f.nb;
    const MlpWork ww = work_at(w, group * step);
    cudaError_t e = cudaSuccess;
    for (int64_t r0 = 0; r0 < f.nb && e == cudaSuccess; r0 += step) {
        const int64_t rows = round_rows(std::min(step, f.nb - r0));
        // three CTAs of 32 rows fit an SM
        e = launch_after(k_mlp_boundary<32>, dim3((unsigned)std::min<int64_t>(rows / 32, 152 * 3)), 256,
                         sizeof(RowSmem<32, true>), s, true, net, f, lm, lm1, lm2, ww, r0, rows);
        if (e == cudaSuccess && rounds) e = launch_outer(ww, (int)(rows / kMlpTile), r0 == 0, s);
    }
    if (e == cudaSuccess && rounds)
        e = launch_after(k_mlp_reduce<kReduceAdd>, dim3(kReduceBlocks), 128, 0, s, true, w.part, (const double *)nullptr,
                         (int)(step / kMlpTile), 1, 1.0, grad, (double *)nullptr, AdamArgs{});
    return e;
}

cudaError_t mlp_boundary_params(int64_t nb, int n, float *grad, const MlpWork &w, cudaStream_t s)
{
    const int64_t step = round_rows(nb);
    if (nb <= 0 || n <= 0 || step < nb) return cudaSuccess;  // (in rounds: already added)
    const int tiles = (int)(step / kMlpTile);
    cudaError_t e = launch_outer(work_at(w, 0), tiles * n, true, s);
    if (e != cudaSuccess) return e;
    return launch_after(k_mlp_reduce<kReduceGroups>, dim3(kGroupBlocks), 128, 0, s, true, w.part, (const double *)nullptr,
                        tiles, n, 1.0, grad, (double *)nullptr, AdamArgs{});
}

cudaError_t mlp_adam(const MlpAdam &adam, const float *grad, cudaStream_t s)
{
    k_mlp_adam<<<(kMlpParams + 255) / 256, 256, 0, s>>>(adam_args(adam), grad);
    return cudaGetLastError();
}

}  // namespace semgb
