// Per-row, per-128-column dynamic FP8 e4m3 quantisation (bandwidth kernel).
// Rounding sequence of the reference's torch oracle (aiter/ops/quant.py:64-94):
//   amax -> scale = amax / 448 (IEEE division; 0 -> 1) -> code = RNE_e4m3(x / scale), the quotient correctly
// rounded (quant_codes8), so the codes and scales are bit-identical to it.  The reference's HIP kernel multiplies by
// reciprocals instead (csrc/kernels/quant_kernels.cu:121,159-160), which is not.
//
// 16 lanes own one 128-element group (8 bf16 = one 16-byte load each), two groups per warp.
//
// What bounds these kernels: HBM, 3 bytes per element. That takes several loads in flight per thread and short
// arithmetic (quant_codes8); with one load per thread and eight IEEE divisions the 1x128 kernel ran at 2.3 TB/s.

#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "common.cuh"
#include "quant_device.cuh"

namespace b200 {
namespace {

constexpr int kQuantThreads = 256;

// num_rows (optional, device): only the first *num_rows * rows_factor rows are quantised. transposed: the scale of
// group (row, col-group) goes to scales[col-group * rows_used + row] instead of scales[row * groups_per_row + col-group]
// (the layout the reference's 1-stage path reads, csrc/kernels/quant_kernels.cu:143-146; rows_used = the dynamic
// row count when num_rows is given, as there).
// A CTA covers kQuantThreads * U consecutive 16-byte pieces, U loads in flight per thread.
// after_wait = false: this launch neither reads nor overwrites anything of the kernel before it on the stream, so it may
// run beside it (the layer's quantiser beside the sort); its completion still implies that kernel's.
template <bool F16, int U>
__global__ void __launch_bounds__(kQuantThreads) quant_1x128_kernel(
    const uint4* x, uint2* q, float* scales, int64_t groups, int groups_per_row, const int* num_rows, int rows_factor,
    int transposed, bool after_wait) {
    if (after_wait) pdl_wait();
    pdl_trigger();
    const int64_t p0 = (int64_t)blockIdx.x * (kQuantThreads * U) + threadIdx.x;
    int64_t rows_used = groups / groups_per_row;
    if (num_rows) rows_used = min(rows_used, (int64_t)*num_rows * rows_factor);
    const int64_t pieces = rows_used * groups_per_row * 16;
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        raw[u] = make_uint4(0, 0, 0, 0);
        if (p0 + u * kQuantThreads < pieces) raw[u] = x[p0 + u * kQuantThreads];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t p = p0 + u * kQuantThreads;
        uint2 codes;
        const float scale = quant_group16<F16>(raw[u], codes);
        if (p < pieces) {
            q[p] = codes;
            if ((threadIdx.x & 15) == 0) {
                const int64_t g = p >> 4;
                if (transposed) {
                    const int64_t row = g / groups_per_row, cg = g - row * groups_per_row;
                    scales[cg * rows_used + row] = scale;
                } else {
                    scales[g] = scale;
                }
            }
        }
    }
    if (!after_wait) pdl_wait();
}

// Per-row dynamic FP8 quantisation over the whole row (QuantType.per_Token): one CTA per row at a time; the row stays in
// registers (CACHE 16-byte pieces per thread) between the amax pass and the conversion pass; what does not fit there is
// read again (L1/L2). Same rounding sequence as above (aiter/ops/quant.py:64-94 over the last dimension). Rows at or past
// *row_limit * rows_factor (if given) are skipped: the grid is a few CTAs per SM that stride over the rows below it, so a
// sorted buffer's padded tail costs no CTAs. sorted_ids (if given; row_limit is then the sort's {rows, tokens} pair): rows of
// a sorted buffer that hold padding are skipped, neither read nor written (a decode batch has ~16 of them per live row).
__device__ __forceinline__ bool is_padding(const int* sorted_ids, const int* num_valid, int M, int64_t row) {
    return sorted_ids && (sorted_ids[row] & 0xFFFFFF) >= min(num_valid[1], M);
}
constexpr int kRowThreads = 256;
template <bool F16, int CACHE>
__global__ void __launch_bounds__(kRowThreads) quant_per_token_kernel(const uint4* x, uint2* q, float* scales, int64_t rows,
                                                                      int cols8, const int* row_limit, int rows_factor,
                                                                      const int* sorted_ids, int M, bool after_wait) {
    __shared__ float red[2][kRowThreads / 32];
    if (after_wait) pdl_wait();
    pdl_trigger();
    const int tid = threadIdx.x;
    if (row_limit) rows = min(rows, (int64_t)*row_limit * rows_factor);
    int par = 0;
    for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
        if (is_padding(sorted_ids, row_limit, M, row)) continue;
        const uint4* xr = x + row * cols8;
        uint4 raw[CACHE];
        float amax = 0.f, v[8];
#pragma unroll
        for (int k = 0; k < CACHE; ++k) {
            raw[k] = make_uint4(0, 0, 0, 0);
            if (k * kRowThreads + tid < cols8) raw[k] = xr[k * kRowThreads + tid];
        }
#pragma unroll
        for (int k = 0; k < CACHE; ++k) {
            unpack8<F16>(raw[k], v);
            amax = amax8(v, amax);
        }
        for (int i = CACHE * kRowThreads + tid; i < cols8; i += kRowThreads) {
            unpack8<F16>(xr[i], v);
            amax = amax8(v, amax);
        }
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
        if ((tid & 31) == 0) red[par][tid >> 5] = amax;
        // One barrier per row: the buffers alternate with the rows that pass it, skipped rows not counted, so a buffer is
        // written again only behind the barrier of the row in between, which every reader of this row has reached by then.
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kRowThreads / 32; ++k) amax = fmaxf(amax, red[par][k]);
        float scale = __fdiv_rn(amax, 448.0f);
        if (scale == 0.f) scale = 1.f;
#pragma unroll
        for (int k = 0; k < CACHE; ++k)
            if (k * kRowThreads + tid < cols8) {
                unpack8<F16>(raw[k], v);
                q[row * cols8 + k * kRowThreads + tid] = quant_codes8(v, scale);
            }
        for (int i = CACHE * kRowThreads + tid; i < cols8; i += kRowThreads) {
            unpack8<F16>(xr[i], v);
            q[row * cols8 + i] = quant_codes8(v, scale);
        }
        if (tid == 0) scales[row] = scale;
        par ^= 1;
    }
    if (!after_wait) pdl_wait();
}

// Per-tensor dynamic FP8 quantisation (QuantType.per_Tensor; torch twin per_tensor_quant, aiter/ops/quant.py:318-328:
// scale = max|x| / 448 and codes = RNE_e4m3(x / scale), both correctly rounded, no zero guard). Two passes:
// the maximum over the rows below *row_limit goes to amax[0] (non-negative floats order like their bit patterns,
// so an integer atomicMax does it), then every row is converted with the one scale, which is also written to
// scale[0] and, if asked, once per row to row_scales (the GEMM kernels take one activation scale per row).
template <bool F16>
__global__ void __launch_bounds__(256) amax_kernel(const uint4* x, int64_t rows, int cols8, const int* row_limit,
                                                   unsigned int* amax) {
    pdl_wait();
    pdl_trigger();
    const int64_t limit = row_limit ? min((int64_t)*row_limit, rows) : rows;
    const int64_t n = limit * cols8, step = (int64_t)gridDim.x * blockDim.x;
    float m = 0.f, v[8];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += 4 * step) {
        uint4 raw[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            raw[k] = make_uint4(0, 0, 0, 0);
            if (i + k * step < n) raw[k] = x[i + k * step];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            unpack8<F16>(raw[k], v);
            m = amax8(v, m);
        }
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(amax, __float_as_uint(m));
}

template <bool F16>
__global__ void __launch_bounds__(256) quant_per_tensor_kernel(const uint4* x, uint2* q, float* scale_out, float* row_scales,
                                                               int64_t rows, int cols8, const int* row_limit,
                                                               const int* sorted_ids, int M, const unsigned int* amax) {
    pdl_wait();
    pdl_trigger();
    const int64_t limit = row_limit ? min((int64_t)*row_limit, rows) : rows;
    const float scale = __fdiv_rn(__uint_as_float(*amax), 448.0f);
    if (blockIdx.x == 0 && threadIdx.x == 0) scale_out[0] = scale;
    if (sorted_ids) {   // a CTA takes whole rows, so that padding rows can be left out
        float v[8];
        for (int64_t row = blockIdx.x; row < limit; row += gridDim.x) {
            if (is_padding(sorted_ids, row_limit, M, row)) continue;
            for (int i = threadIdx.x; i < cols8; i += 256) {
                unpack8<F16>(x[row * cols8 + i], v);
                q[row * cols8 + i] = quant_codes8(v, scale);
            }
        }
        return;
    }
    const int64_t n = limit * cols8, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += 4 * step) {
        uint4 raw[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            raw[k] = make_uint4(0, 0, 0, 0);
            if (i + k * step < n) raw[k] = x[i + k * step];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float v[8];
            unpack8<F16>(raw[k], v);
            if (i + k * step < n) q[i + k * step] = quant_codes8(v, scale);
        }
    }
    if (row_scales)
        for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += step) row_scales[r] = scale;
}

}  // namespace

// input dtype of the three quantisers: bf16 or fp16 (the reference takes either, aiter/fused_moe.py:752-756)
static bool input_is_f16(const aiter_tensor_t* input) {
    B200_CHECK(input != nullptr, "input must not be NULL");
    B200_CHECK(input->dtype_ == AITER_DTYPE_bf16 || input->dtype_ == AITER_DTYPE_fp16,
               "input must be bf16 or fp16, got dtype code ", input->dtype_);
    return input->dtype_ == AITER_DTYPE_fp16;
}

void launch_quant_per_tensor(aiter_tensor_t* out, const aiter_tensor_t* input, aiter_tensor_t* scale, aiter_tensor_t* amax,
                             aiter_tensor_t* row_scales, const aiter_tensor_t* row_limit, bool amax_cleared, bool amax_done, const int* sorted_ids,
                             int M, cudaStream_t stream) {
    const bool f16 = input_is_f16(input);
    check_tensor(input, "input", -1, 2);
    check_tensor(out, "out", AITER_DTYPE_fp8, 2);
    check_tensor(scale, "scale", AITER_DTYPE_fp32, -1);
    check_tensor(amax, "amax", AITER_DTYPE_fp32, -1);
    const int64_t rows = input->shape[0], cols = input->shape[1];
    B200_CHECK(cols % 8 == 0 && cols >= 8, "row length must be a multiple of 8, got ", cols);
    B200_CHECK(out->shape[0] == rows && out->shape[1] == cols, "out must have the shape of input");
    B200_CHECK(scale->numel_ >= 1 && amax->numel_ >= 1, "scale and amax need one element each");
    B200_CHECK(((uintptr_t)input->ptr & 15) == 0 && ((uintptr_t)out->ptr & 7) == 0, "input must be 16-byte and out 8-byte aligned");
    if (row_scales) {
        check_tensor(row_scales, "row_scales", AITER_DTYPE_fp32, -1);
        B200_CHECK((int64_t)row_scales->numel_ >= rows, "row_scales needs one element per row");
    }
    if (row_limit) check_tensor(row_limit, "row_limit", AITER_DTYPE_i32, -1);
    if (!amax_cleared) B200_CUDA(cudaMemsetAsync(amax->ptr, 0, sizeof(float), stream));
    if (rows == 0) return;
    const int64_t n = sorted_ids ? rows * 256 : rows * (cols / 8);   // a CTA per row, or per 256 pieces
    const int grid = (int)std::min<int64_t>((n + 255) / 256, (int64_t)sm_count(input->device_id) * 8);
    const int* lim = row_limit ? (const int*)row_limit->ptr : nullptr;
    float* per_row = row_scales ? (float*)row_scales->ptr : nullptr;
    if (!amax_done)
        launch_pdl(f16 ? amax_kernel<true> : amax_kernel<false>, grid, 256, 0, stream, (const uint4*)input->ptr, rows, (int)(cols / 8),
               lim, (unsigned int*)amax->ptr);
    launch_pdl(f16 ? quant_per_tensor_kernel<true> : quant_per_tensor_kernel<false>, grid, 256, 0, stream, (const uint4*)input->ptr,
               (uint2*)out->ptr, (float*)scale->ptr, per_row, rows, (int)(cols / 8), lim, sorted_ids, M,
               (const unsigned int*)amax->ptr);
}

void launch_quant_per_token(aiter_tensor_t* out, const aiter_tensor_t* input, aiter_tensor_t* scales,
                            const aiter_tensor_t* row_limit, int rows_factor, bool after_wait, const int* sorted_ids, int M,
                            cudaStream_t stream) {
    const bool f16 = input_is_f16(input);
    check_tensor(input, "input", -1, 2);
    check_tensor(out, "out", AITER_DTYPE_fp8, 2);
    check_tensor(scales, "scales", AITER_DTYPE_fp32, -1);
    const int64_t rows = input->shape[0], cols = input->shape[1];
    B200_CHECK(cols % 8 == 0 && cols >= 8, "row length must be a multiple of 8, got ", cols);
    B200_CHECK(out->shape[0] == rows && out->shape[1] == cols, "out must have the shape of input");
    B200_CHECK((int64_t)scales->numel_ >= rows, "scales needs one element per row");
    B200_CHECK(((uintptr_t)input->ptr & 15) == 0 && ((uintptr_t)out->ptr & 7) == 0, "input must be 16-byte and out 8-byte aligned");
    B200_CHECK(rows_factor >= 1, "num_rows_factor must be >= 1, got ", rows_factor);
    if (row_limit) check_tensor(row_limit, "num_rows", AITER_DTYPE_i32, -1);
    if (rows == 0) return;
    const int* lim = row_limit ? (const int*)row_limit->ptr : nullptr;
    const int cols8 = (int)(cols / 8);
    const int grid = (int)std::min<int64_t>(rows, (int64_t)sm_count(input->device_id) * 8);
    // pieces a thread keeps: the whole row for rows up to 4096 / 16384 elements, 8 of them for longer ones
    auto go = [&](auto kernel) {
        launch_pdl(kernel, grid, kRowThreads, 0, stream, (const uint4*)input->ptr, (uint2*)out->ptr, (float*)scales->ptr, rows, cols8,
                   lim, rows_factor, sorted_ids, M, after_wait);
    };
    if (cols8 <= 2 * kRowThreads) f16 ? go(quant_per_token_kernel<true, 2>) : go(quant_per_token_kernel<false, 2>);
    else f16 ? go(quant_per_token_kernel<true, 8>) : go(quant_per_token_kernel<false, 8>);
}

void launch_quant_1x128(aiter_tensor_t* out, const aiter_tensor_t* input, aiter_tensor_t* scales,
                        const aiter_tensor_t* num_rows, int rows_factor, int transpose_scale, bool after_wait,
                        cudaStream_t stream) {
    const bool f16 = input_is_f16(input);
    check_tensor(input, "input", -1, -1);
    check_tensor(out, "out", AITER_DTYPE_fp8, -1);
    check_tensor(scales, "scales", AITER_DTYPE_fp32, -1);
    B200_CHECK(input->ndim >= 1, "input must have at least one dimension");
    const int64_t cols = input->shape[input->ndim - 1];
    B200_CHECK(cols % 128 == 0, "last dimension must be a multiple of 128, got ", cols);
    B200_CHECK(out->numel_ == input->numel_, "out must have as many elements as input");
    const int64_t groups = (int64_t)input->numel_ / 128;
    B200_CHECK((int64_t)scales->numel_ >= groups, "scales needs ", groups, " elements, has ",
               scales->numel_);
    B200_CHECK(((uintptr_t)input->ptr & 15) == 0 && ((uintptr_t)out->ptr & 7) == 0,
               "input must be 16-byte and out 8-byte aligned");
    B200_CHECK(rows_factor >= 1, "num_rows_factor must be >= 1, got ", rows_factor);
    if (num_rows) check_tensor(num_rows, "num_rows", AITER_DTYPE_i32, -1);
    if (groups == 0) return;
    const int* lim = num_rows ? (const int*)num_rows->ptr : nullptr;
    // four pieces per thread once that still gives every SM a few CTAs, one for small inputs (latency)
    const int64_t pieces = groups * 16, sms = sm_count(input->device_id);
    const int per_thread = pieces >= sms * 4 * kQuantThreads * 4 ? 4 : 1;
    const int64_t blocks = (pieces + kQuantThreads * per_thread - 1) / (kQuantThreads * per_thread);
    B200_CHECK(blocks < ((int64_t)1 << 31), "input too large");
    auto go = [&](auto kernel) {
        launch_pdl(kernel, (unsigned)blocks, kQuantThreads, 0, stream, (const uint4*)input->ptr, (uint2*)out->ptr, (float*)scales->ptr,
                   groups, (int)(cols / 128), lim, rows_factor, transpose_scale, after_wait);
    };
    if (per_thread == 4) f16 ? go(quant_1x128_kernel<true, 4>) : go(quant_1x128_kernel<false, 4>);
    else f16 ? go(quant_1x128_kernel<true, 1>) : go(quant_1x128_kernel<false, 1>);
}

}  // namespace b200
