// Device-side helpers shared by the kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>

#include "../../include/darknet_b200.h"

namespace dnb {

// Darknet's activation functions (src/activations.h:19-53), evaluated in fp32
// as the reference's device code does (src/activation_kernels.cu:13-77).  The
// CPU reference evaluates the constants in double; the difference is at most
// one fp32 ulp and far inside the layer tolerances.
__device__ __forceinline__ float activate(float x, int a)
{
    switch (a) {
    case DNB_LINEAR:   return x;
    case DNB_LEAKY:    return x > 0.f ? x : 0.1f * x;
    case DNB_LOGISTIC: return 1.f / (1.f + expf(-x));
    case DNB_RELU:     return x > 0.f ? x : 0.f;
    case DNB_RELIE:    return x > 0.f ? x : 0.01f * x;
    case DNB_RAMP:     return (x > 0.f ? x : 0.f) + 0.1f * x;
    case DNB_TANH:     return (expf(2.f * x) - 1.f) / (expf(2.f * x) + 1.f);
    case DNB_LOGGY:    return 2.f / (1.f + expf(-x)) - 1.f;
    case DNB_ELU:      return x >= 0.f ? x : expf(x) - 1.f;
    case DNB_SELU:     return x >= 0.f ? 1.0507f * x : 1.0507f * 1.6732f * (expf(x) - 1.f);
    case DNB_PLSE:
        if (x < -4.f) return 0.01f * (x + 4.f);
        if (x > 4.f) return 0.01f * (x - 4.f) + 1.f;
        return 0.125f * x + 0.5f;
    case DNB_STAIR: {
        int n = (int)floorf(x);
        if (n % 2 == 0) return floorf(x / 2.f);
        return (x - n) + floorf(x / 2.f);
    }
    case DNB_HARDTAN:  return x < -1.f ? -1.f : (x > 1.f ? 1.f : x);
    case DNB_LHTAN:
        if (x < 0.f) return 0.001f * x;
        if (x > 1.f) return 0.001f * (x - 1.f) + 1.f;
        return x;
    }
    return 0.f;
}

// Same function for hot loops: the two common activations inline, the 14-way switch out of line (inlined
// into an unrolled epilogue it multiplies the code size).
static __device__ __noinline__ float activate_call(float x, int a) { return activate(x, a); }
__device__ __forceinline__ float activate_fast(float x, int a)
{
    if (a == DNB_LEAKY) return fmaxf(x, 0.1f * x);   // x > 0 ? x : 0.1x
    if (a == DNB_LINEAR) return x;
    return activate_call(x, a);
}

// Round an fp32 value to the nearest TF32 (10-bit mantissa) value, ties away from zero, low 13 mantissa
// bits clear: what cvt.rna.tf32.f32 computes for finite values, written as an integer add and a mask
// because the conversion instruction issues at a fraction of the rate and the epilogues run it per element.
// (Infinity stays infinity; a NaN may become infinity, and one with all of its bits set, which arithmetic makes, becomes -0.)
__device__ __forceinline__ float round_tf32(float x)
{
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
}

template <typename T> __device__ __forceinline__ float to_float(T v);
template <> __device__ __forceinline__ float to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Four 16-byte pieces (floats, or bf16 values) of a 2x2 maxpool's window: its largest values, as forward_maxpool_layer finds them, from the
// lowest float up (src/maxpool_layer.c:103-105), so that a NaN never wins.
template <bool BF16>
__device__ __forceinline__ uint4 largest_of_four(const uint4 (&v)[4])
{
    uint32_t out[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float a = -FLT_MAX, b = -FLT_MAX;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t w = e == 0 ? v[i].x : e == 1 ? v[i].y : e == 2 ? v[i].z : v[i].w;
            if (!BF16) a = fmaxf(a, __uint_as_float(w));
            else { a = fmaxf(a, __uint_as_float(w << 16)); b = fmaxf(b, __uint_as_float(w & 0xffff0000u)); }
        }
        if (!BF16) out[e] = __float_as_uint(a);
        else { const __nv_bfloat162 h = __floats2bfloat162_rn(a, b); out[e] = *reinterpret_cast<const uint32_t *>(&h); }
    }
    return make_uint4(out[0], out[1], out[2], out[3]);
}

// The larger of two floats, or of two pairs of bf16 values; a NaN never wins.  lowest: what a maxpool starts from (in bf16 it rounds to -infinity).
template <bool BF16>
__device__ __forceinline__ uint32_t larger(uint32_t a, uint32_t b)
{
    if (!BF16) return __float_as_uint(fmaxf(__uint_as_float(a), __uint_as_float(b)));
    const __nv_bfloat162 m = __hmax2(*reinterpret_cast<const __nv_bfloat162 *>(&a), *reinterpret_cast<const __nv_bfloat162 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&m);
}
template <bool BF16> __device__ __forceinline__ uint32_t lowest() { return BF16 ? 0xff80ff80u : 0xff7fffffu; }

// Signs of four floats as bytes: +1 where > 0, else -1.
__device__ __forceinline__ uint32_t four_signs(uint4 v)
{
    return (__uint_as_float(v.x) > 0.f ? 0x01u : 0xFFu) | (__uint_as_float(v.y) > 0.f ? 0x01u : 0xFFu) << 8 | (__uint_as_float(v.z) > 0.f ? 0x01u : 0xFFu) << 16 |
           (__uint_as_float(v.w) > 0.f ? 0x01u : 0xFFu) << 24;
}

// The same of four that are no NaN.  As integers the value itself, or one less, which for +0 wraps, has its top bit set where it is not > 0 (-0 among them):
// so has the larger of the two.
__device__ __forceinline__ uint32_t four_signs_no_nan(uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    auto not_positive = [](uint32_t v) { return __viaddmax_u32(v, 0xffffffffu, v); };
    uint32_t ab, cd;
    asm("prmt.b32 %0, %1, %2, 0xfb;" : "=r"(ab) : "r"(not_positive(a)), "r"(not_positive(b)));   // their signs, as bytes
    asm("prmt.b32 %0, %1, %2, 0xfb;" : "=r"(cd) : "r"(not_positive(c)), "r"(not_positive(d)));
    return __byte_perm(ab, cd, 0x5410u) | 0x01010101u;
}

}  // namespace dnb
