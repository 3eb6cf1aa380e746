// Pieces the GEMM kernels of the fused-MoE layer share: activation functions, the promotion step, tensor maps.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "common.cuh"
#include "quant_device.cuh"
#include "sm100_ptx.cuh"

namespace b200 {
namespace {

// torch: silu(x) = x / (1 + exp(-x)) in fp32, then * up (aiter/fused_moe.py:3676).
// The quotient is formed from an approximate reciprocal and one FMA residual correction (error below
// one fp32 ulp, like the exp it depends on) instead of the ~4x longer IEEE division sequence.
__device__ __forceinline__ float silu_mul_fast(float g, float u) {   // valid for g >= -80
    const float d = 1.0f + expf(-g);
    const float y = ptx::rcp_approx(d);
    const float q = g * y;
    return fmaf(fmaf(-q, d, g), y, q) * u;
}
__device__ __forceinline__ float silu_mul_exact(float g, float u) { return __fdiv_rn(g, 1.0f + expf(-g)) * u; }

// torch: gelu(x) = 0.5 * x * (1 + erf(x / sqrt(2))) (the reference's get_torch_act(Gelu) = F.gelu), then * up
__device__ __forceinline__ float gelu_mul(float g, float u) {
    return 0.5f * g * (1.0f + erff(g * 0.70710678118654752440f)) * u;
}

// act(g) * u for N values. The SiLU fast path is straight-line code, so the N dependency chains (exp,
// reciprocal, two FMAs: ~150 clocks each) interleave; the exact path for exp(-g) near overflow sits behind
// ONE branch per group. With a branch per value every chain is a basic block of its own and the epilogue runs
// at the latency of one chain per value (measured: 9.5k of 11.6k clocks per tile).
template <int ACT, int N>
__device__ __forceinline__ void act_mul_n(const float (&g)[N], const float (&u)[N], float (&h)[N]) {
    if (ACT == 1) {
#pragma unroll
        for (int i = 0; i < N; ++i) h[i] = gelu_mul(g[i], u[i]);
        return;
    }
    float gmin = g[0];
#pragma unroll
    for (int i = 1; i < N; ++i) gmin = fminf(gmin, g[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) h[i] = silu_mul_fast(g[i], u[i]);
    if (gmin < -80.0f) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (g[i] < -80.0f) h[i] = silu_mul_exact(g[i], u[i]);
    }
}

// acc[0..7] += v[0..15] * s with packed fp32x2 FMAs (one instruction per column pair)
__device__ __forceinline__ void fold16(float2* acc, const uint32_t* v, float2 s) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
        acc[j] = __ffma2_rn(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), s, acc[j]);
}

// ------------------------------------------------------------------------------------- host
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                   CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                   CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        B200_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres));
        B200_CHECK(sym != nullptr && qres == cudaDriverEntryPointSuccess,
                   "cuTensorMapEncodeTiled is not available in this driver");
        fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

// 2-D view [rows, K] of an fp8 matrix (weights [E, n_rows, K] in boxes of 128 rows x 128 bytes, stage 2's activations in
// boxes of 32 rows), 128B swizzle. Encoding a map
// costs a few microseconds of host time, so the last maps are kept (per thread) and reused while pointer and shape
// repeat, as they do from layer call to layer call.
CUtensorMap make_map(const void* ptr, uint64_t rows, uint64_t K, uint32_t box_rows) {
    struct Entry {
        const void* ptr;
        uint64_t rows, K;
        uint32_t box_rows;
        CUtensorMap map;
    };
    constexpr int kEntries = 16;
    static thread_local Entry cache[kEntries];
    static thread_local int next = 0, used = 0;
    for (int i = 0; i < used; ++i)
        if (cache[i].ptr == ptr && cache[i].rows == rows && cache[i].K == K && cache[i].box_rows == box_rows) return cache[i].map;
    CUtensorMap m;
    cuuint64_t dims[2] = {K, rows};
    cuuint64_t strides[1] = {K};
    cuuint32_t box[2] = {128, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_tiled_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides,
                                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with code ", (int)r);
    cache[next] = Entry{ptr, rows, K, box_rows, m};
    next = (next + 1) % kEntries;
    if (used < kEntries) ++used;
    return m;
}

}  // namespace

// Settings of the wait self-test (b200_moe_debug_config), defined in moe_gemm.cu: the limit of every device-side wait in SM
// clocks, and whether the weight producer is stalled.
extern long long g_wait_limit;
extern int g_stall_producer;

}  // namespace b200
