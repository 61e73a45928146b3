// mlp_device.cuh -- device pieces of the boundary network shared by its forward, boundary and
// training kernels: BF16 conversion, GELU, the m16n8k16 tensor-core step, fragment loads and the
// network staged in shared memory.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "mlp.h"
#include "tma.cuh"

namespace semgb {

namespace {

// Fragment loads of the register-resident inference forward (compile-time knob: 1 = ldmatrix,
// 0 = one 32-bit shared load per fragment register; the same fragments either way, so the same
// bits).  ldmatrix: a quarter of the load instructions, 162 registers, no spill.
#ifndef SEM_MLP_LDSM
#define SEM_MLP_LDSM 1
#endif

constexpr int H = kMlpHidden;
constexpr int KP1 = kMlpInPad + 8;  // row stride (bf16) of X and W1
constexpr int KP2 = H + 8;          // row stride (bf16) of H1 and W2
constexpr int T = kMlpTile;

__device__ __forceinline__ uint16_t f2bf(float x)
{
    const __nv_bfloat16 b = __float2bfloat16_rn(x);
    return *reinterpret_cast<const uint16_t *>(&b);
}

// two floats to BF16 (round to nearest even, as f2bf) in one conversion: lo in the low half
__device__ __forceinline__ uint32_t pack_bf2(float lo, float hi)
{
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&b);
}

// GELU in the tanh form of Hendrycks & Gimpel (2016), GELU(z) = z/2 (1 + tanh(u)),
// u = sqrt(2/pi) (z + 0.044715 z^3), and its derivative; tanh from the hardware approximation
// (tanh.approx.f32, relative error about 2^-11, below the BF16 rounding of the activations)
__device__ __forceinline__ float tanh_hw(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
constexpr float kGeluC = 0.7978845608028654f;  // sqrt(2/pi)
constexpr float kGeluCA = 0.7978845608028654f * 0.044715f;
// u = z (c + c a z^2): two multiplies and one fma
__device__ __forceinline__ float gelu_u(float z) { return z * fmaf(kGeluCA, z * z, kGeluC); }
__device__ __forceinline__ float gelu(float z)
{
    const float t = tanh_hw(gelu_u(z));
    const float h = 0.5f * z;
    return fmaf(h, t, h);
}
// gelu of two values with packed f32x2 arithmetic: the same operations in the same order as gelu,
// each half rounded as the scalar instruction would round it
__device__ __forceinline__ float2 gelu2(float2 z)
{
    const float2 w = fma2(make_float2(kGeluCA, kGeluCA), mul2(z, z), make_float2(kGeluC, kGeluC));
    const float2 u = mul2(z, w);
    const float2 t = make_float2(tanh_hw(u.x), tanh_hw(u.y));
    const float2 h = mul2(make_float2(0.5f, 0.5f), z);
    return fma2(h, t, h);
}
__device__ __forceinline__ float gelu_d(float z)
{
    // d/dz [z/2 (1 + tanh u)] = (1 + t)/2 + z/2 (1 - t^2) (c + 3 c a z^2)
    const float t = tanh_hw(gelu_u(z));
    return fmaf(0.5f, t, 0.5f) + (0.5f * z) * fmaf(-t, t, 1.f) * fmaf(3.f * kGeluCA, z * z, kGeluC);
}

__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// 8x8 b16 matrices from shared memory (fragment layout of the mma operands): x4 takes row
// addresses from lanes 0-31 (matrix lane/8), x2 from lanes 0-15.
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))));
}
__device__ __forceinline__ void ldsm_x2(uint32_t (&r)[2], const void *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1])
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))));
}

struct NetSmem {
    uint16_t w1[H * KP1];
    uint16_t w2[H * KP2];
    float b1[H], b2[H], w3[H], b3;
};

__device__ void load_net(NetSmem &s, const MlpDev &net)
{
    // 16-byte chunks: W1 rows are 96 bf16 (12 chunks), W2 rows 64 (8 chunks); shared rows are
    // padded to 104 and 72 elements, still 16-byte aligned
    constexpr int C1 = kMlpInPad / 8, C2 = H / 8;
    static_assert((KP1 * 2) % 16 == 0 && (KP2 * 2) % 16 == 0, "16-byte aligned shared rows");
#pragma unroll 4
    for (int i = threadIdx.x; i < H * C1; i += blockDim.x) {
        const int nn = i / C1, j = i - nn * C1;
        *reinterpret_cast<uint4 *>(s.w1 + nn * KP1 + j * 8) = __ldg(reinterpret_cast<const uint4 *>(net.w1) + i);
    }
#pragma unroll 4
    for (int i = threadIdx.x; i < H * C2; i += blockDim.x) {
        const int nn = i / C2, j = i - nn * C2;
        *reinterpret_cast<uint4 *>(s.w2 + nn * KP2 + j * 8) = __ldg(reinterpret_cast<const uint4 *>(net.w2) + i);
    }
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        s.b1[i] = net.b1[i];
        s.b2[i] = net.b2[i];
        s.w3[i] = net.w3[i];
    }
    if (threadIdx.x == 0) s.b3 = net.b3[0];
}

}  // namespace

}  // namespace semgb
