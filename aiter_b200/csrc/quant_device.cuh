// Device pieces of the 1x128 FP8 quantisation shared by the plain quantiser and the fused quantise-and-dispatch
// kernel of the expert-parallel exchange. Rounding sequence of the reference's torch oracle
// (aiter/ops/quant.py:64-94): amax -> scale = amax / 448 (IEEE division; 0 -> 1) -> code = RNE_e4m3(x / scale).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

namespace b200 {

// eight 16-bit floats (bf16 or fp16) of one 16-byte load -> fp32
template <bool F16>
__device__ __forceinline__ void unpack8(const uint4& raw, float (&v)[8]) {
    if (F16) {
        const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(h[i]);
            v[2 * i] = f.x;
            v[2 * i + 1] = f.y;
        }
    } else {
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(h[i]);
            v[2 * i] = f.x;
            v[2 * i + 1] = f.y;
        }
    }
}

// Correctly rounded a / b given rb = RN(1/b): two FMA residual corrections (the first makes the quotient faithful, the
// second then rounds it correctly), valid while nothing over- or underflows (P. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", 1990, theorem on quotient rounding).
__device__ __forceinline__ float div_rn_by(float a, float b, float rb) {
    float q = a * rb;
    q = fmaf(fmaf(-q, b, a), rb, q);
    return fmaf(fmaf(-q, b, a), rb, q);
}

// Scales for which div_rn_by stands in for the IEEE division. The residual a - q*b is a multiple of ulp(q) * ulp(b); for a
// quotient of at least 2^-10 (smaller ones are code 0) that is 2^-33 * ulp(b), which fp32 holds exactly, as a subnormal if
// need be, down to ulp(b) = 2^-116. 1e-24 (ulp 2^-103) leaves three decades; the upper limit keeps 1/b normal.
__device__ __forceinline__ bool scale_is_tame(float scale) { return scale > 1e-24f && scale < 1e30f; }

// Codes RNE_e4m3(v / scale) of eight values: five FMA-pipe operations per quotient from one reciprocal per scale instead of
// the ~4x longer division sequence, which bound the quantisers at 2.3 TB/s.
__device__ __forceinline__ uint2 quant_codes8(const float (&v)[8], float scale) {
    float d[8];
    if (scale_is_tame(scale)) {
        const float rs = __frcp_rn(scale);
#pragma unroll
        for (int i = 0; i < 8; ++i) d[i] = copysignf(div_rn_by(v[i], scale, rs), v[i]);   // the corrections lose the sign of -0
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) d[i] = __fdiv_rn(v[i], scale);
    }
    uint32_t w[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(d[4 * i], d[4 * i + 1]), __NV_SATFINITE, __NV_E4M3);
        const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(d[4 * i + 2], d[4 * i + 3]), __NV_SATFINITE, __NV_E4M3);
        w[i] = lo | (hi << 16);
    }
    return make_uint2(w[0], w[1]);
}

__device__ __forceinline__ float amax8(const float (&v)[8], float m = 0.f) {
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(v[i]));
    return m;
}

// 16 consecutive lanes of a warp (an aligned half-warp) hold one 128-element group, 8 elements each. Returns the
// group's scale (on all 16 lanes) and this lane's 8 codes. Must be called by the whole warp (shuffles).
template <bool F16>
__device__ __forceinline__ float quant_group16(const uint4& raw, uint2& codes) {
    float v[8];
    unpack8<F16>(raw, v);
    float amax = amax8(v);
#pragma unroll
    for (int d = 8; d >= 1; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
    float scale = __fdiv_rn(amax, 448.0f);
    if (scale == 0.f) scale = 1.f;
    codes = quant_codes8(v, scale);
    return scale;
}

}  // namespace b200
