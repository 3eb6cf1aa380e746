// Router kernels that feed moe_sorting / fused_moe: one warp per token, scores in registers.
//
//   biased_grouped_topk  DeepSeek-V3 style: sigmoid scores, + correction bias for the choice, groups ranked
//                        by the sum of their two best biased scores, top groups kept, top-k experts among
//                        them, weights = un-biased scores, renormalised, times routed_scaling_factor.
//                        Arithmetic of aiter/ops/topk.py:217-259 (biased_grouped_topk_torch); replaces the
//                        native op of aiter/ops/topk.py:89-99 / csrc/kernels/topk_softmax_kernels_group.cu:1219-1266.
//   topk_softmax         fp32 softmax, top-k, optional renormalisation (aiter/fused_moe.py:4058-4129,
//                        csrc/kernels/topk_softmax_kernels.cu:769).
//
// What bounds them: the latency of one token's chain of warp-wide reductions (a token's scores are 1-2 KB, a batch of
// 8192 fits the warps of one wave). So every reduction is one redux.sync on order-preserving integer keys instead of
// five (value, index) shuffle rounds, and the grouped router keeps a lane's experts contiguous, so that a routing group
// is a run of lanes and all groups are reduced at once. DeepSeek-V3 routing (E=256, 8 groups, top 8): 31 -> 4.6 us at 64
// tokens, 95 -> 17 us at 8192; the first version tested e / group_size against each group in turn.
// Selections break ties by the lower index, so the result does not depend on scheduling.

#include <cuda_bf16.h>
#include <math_constants.h>

#include <type_traits>

#include "common.cuh"

namespace b200 {
namespace {

constexpr int kWarpsPerBlock = 4;
#define kNegInf (-CUDART_INF_F)

template <typename T>
__device__ __forceinline__ float load_f(const T* p, int64_t i);
template <>
__device__ __forceinline__ float load_f<float>(const float* p, int64_t i) { return p[i]; }
template <>
__device__ __forceinline__ float load_f<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i) {
    return __bfloat162float(p[i]);
}

// VPL consecutive entries from index i on, those at or past n as 0. One 16-byte (fp32) or 8-byte (bf16) load per four
// entries where the rows keep that alignment (n a multiple of 4).
template <int VPL, typename T>
__device__ __forceinline__ void load_run(const T* row, int i, int n, bool aligned, float (&v)[VPL]) {
    if (VPL >= 4 && aligned) {
#pragma unroll
        for (int j = 0; j < VPL; j += 4) {
            float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i + j < n) {
                if constexpr (std::is_same<T, float>::value) {
                    f = *reinterpret_cast<const float4*>(row + i + j);
                } else {
                    const uint2 raw = *reinterpret_cast<const uint2*>(row + i + j);
                    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
                    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
                    f = make_float4(lo.x, lo.y, hi.x, hi.y);
                }
            }
            v[j] = f.x;
            if (j + 1 < VPL) v[j + 1] = f.y;
            if (j + 2 < VPL) v[j + 2] = f.z;
            if (j + 3 < VPL) v[j + 3] = f.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < VPL; ++j) v[j] = (i + j < n) ? load_f<T>(row, i + j) : 0.f;
    }
}

// Unsigned key with the order of the floats (-0 and +0 equal). NaN gets the lowest key: it is never preferred.
__device__ __forceinline__ uint32_t order_key(float v) {
    const uint32_t u = __float_as_uint(v + 0.f);
    return v != v ? 0u : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
}

// Picks the k largest of key[] (value, then lower index) one at a time; entry j of a lane is expert index(j), ascending in
// j; key 0 = not there, NaN or already taken. Lane i < k keeps pick i in (my_id, my_w), with the weight wsrc[] of the winning
// expert. Where nothing is left to pick the id is INT_MAX, which the sort drops, and the weight 0. Returns the sum of the k
// weights, added in the order of the picks.
template <int VPL, typename Index>
__device__ __forceinline__ float select_topk(uint32_t (&key)[VPL], const float (&wsrc)[VPL], int k, int lane, Index index,
                                             int& my_id, float& my_w) {
    float wsum = 0.f;
    for (int i = 0; i < k; ++i) {
        uint32_t best = key[0];
#pragma unroll
        for (int j = 1; j < VPL; ++j) best = max(best, key[j]);
        best = max(__reduce_max_sync(0xffffffffu, best), 1u);   // no score has key 1: at 0 nothing matches
        int mine = 0x7fffffff;
        float w = 0.f;
#pragma unroll
        for (int j = VPL - 1; j >= 0; --j)
            if (key[j] == best) {
                mine = index(j);
                w = wsrc[j];
            }
        const int win = __reduce_min_sync(0xffffffffu, mine);
        const unsigned owner = __ballot_sync(0xffffffffu, mine == win);
        w = __shfl_sync(0xffffffffu, w, __ffs(owner) - 1);
#pragma unroll
        for (int j = 0; j < VPL; ++j)
            if (index(j) == win) key[j] = 0u;   // retired
        wsum += w;
        if (lane == i) {
            my_id = win;
            my_w = w;
        }
    }
    return wsum;
}

// A score as it counts for its group: NaN counts for nothing (fmaxf returns the operand that is a number). The two largest of
// a run are merged by fminf / fmaxf, which would otherwise take the partner of a NaN twice.
__device__ __forceinline__ float in_group(float v) { return fmaxf(v, kNegInf); }

// Two largest of a run of values and of a second such pair (no NaN among them)
__device__ __forceinline__ void merge_top2(float& b1, float& b2, float o1, float o2) {
    b2 = fmaxf(fminf(b1, o1), fmaxf(b2, o2));
    b1 = fmaxf(b1, o1);
}

template <typename TG, typename TB, int VPL>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) biased_grouped_topk_kernel(
    const TG* gating, const TB* bias, float* out_w, int* out_id,
    int tokens, int E, int topk, int n_group, int topk_group, int renorm, float scale) {
    const int lane = threadIdx.x & 31;
    const int token = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    pdl_wait();
    pdl_trigger();
    if (token >= tokens) return;
    const int gsize = E / n_group;
    const int e0 = lane * VPL;      // this lane's experts: e0 .. e0 + VPL - 1
    float score[VPL], choice[VPL];
    load_run<VPL>(gating + (int64_t)token * E, e0, E, E % 4 == 0 && ((uintptr_t)gating & 15) == 0, score);
    load_run<VPL>(bias, e0, E, E % 4 == 0 && ((uintptr_t)bias & 15) == 0, choice);
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
        const bool there = e0 + j < E;
        score[j] = there ? __fdiv_rn(1.0f, 1.0f + expf(-score[j])) : 0.f;
        choice[j] = there ? score[j] + choice[j] : kNegInf;
    }
    // group score = sum of the two largest biased scores of the group; kept = the group is among the topk_group best
    uint32_t kept = 0;   // bit j: the group of expert e0 + j is kept
    const int span = gsize / VPL;   // lanes per group
    if (gsize % VPL == 0 && (span & (span - 1)) == 0) {
        // a group is a power-of-two run of lanes: all groups at once in log2(span) butterfly rounds
        float b1 = in_group(choice[0]), b2 = kNegInf;
#pragma unroll
        for (int j = 1; j < VPL; ++j) merge_top2(b1, b2, in_group(choice[j]), kNegInf);
        for (int d = 1; d < span; d <<= 1)
            merge_top2(b1, b2, __shfl_xor_sync(0xffffffffu, b1, d), __shfl_xor_sync(0xffffffffu, b2, d));
        const float gs = in_group((gsize >= 2) ? b1 + b2 : b1);   // inf - inf of two biases
        const int mine = lane / span;
        int better = 0;
        for (int g = 0; g < n_group; ++g) {
            const float o = __shfl_sync(0xffffffffu, gs, g * span);
            better += (o > gs || (o == gs && g < mine)) ? 1 : 0;
        }
        kept = better < topk_group ? 0xffffffffu : 0u;
    } else {
        // any other group size: one group at a time
        float gs_mine = kNegInf;   // lane g holds the score of group g (n_group <= 32)
        for (int g = 0; g < n_group; ++g) {
            float b1 = kNegInf, b2 = kNegInf;
#pragma unroll
            for (int j = 0; j < VPL; ++j)
                if (e0 + j >= g * gsize && e0 + j < (g + 1) * gsize) merge_top2(b1, b2, in_group(choice[j]), kNegInf);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1)
                merge_top2(b1, b2, __shfl_xor_sync(0xffffffffu, b1, d), __shfl_xor_sync(0xffffffffu, b2, d));
            if (lane == g) gs_mine = in_group((gsize >= 2) ? b1 + b2 : b1);
        }
        int better = 0;
        for (int g = 0; g < n_group; ++g) {
            const float o = __shfl_sync(0xffffffffu, gs_mine, g);
            better += (o > gs_mine || (o == gs_mine && g < lane)) ? 1 : 0;
        }
        const unsigned groups = __ballot_sync(0xffffffffu, lane < n_group && better < topk_group);
#pragma unroll
        for (int j = 0; j < VPL; ++j)
            if (e0 + j < E) kept |= ((groups >> ((e0 + j) / gsize)) & 1u) << j;
    }
    // experts of dropped groups compete with the value 0.0, as masked_fill(~mask, 0.0) does
    uint32_t key[VPL];
#pragma unroll
    for (int j = 0; j < VPL; ++j) key[j] = (e0 + j < E) ? order_key(((kept >> j) & 1u) ? choice[j] : 0.0f) : 0u;
    int my_id = 0;
    float my_w = 0.f;
    const float wsum = select_topk<VPL>(key, score, topk, lane, [&](int j) { return e0 + j; }, my_id, my_w);
    if (lane < topk) {
        float w = renorm ? __fdiv_rn(my_w, wsum) : my_w;
        out_w[(int64_t)token * topk + lane] = w * scale;
        out_id[(int64_t)token * topk + lane] = my_id;
    }
}

template <typename TG, int VPL>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) topk_softmax_kernel(
    const TG* gating, float* out_w, int* out_id, int* src_row,
    int tokens, int E, int topk, int renorm) {
    const int lane = threadIdx.x & 31;
    const int token = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    pdl_wait();
    pdl_trigger();
    if (token >= tokens) return;
    float x[VPL], prob[VPL];   // entry j of a lane is expert j * 32 + lane
    float mx = kNegInf;
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
        const int e = j * 32 + lane;
        x[j] = (e < E) ? load_f<TG>(gating, (int64_t)token * E + e) : kNegInf;
        mx = fmaxf(mx, x[j]);
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
        prob[j] = (j * 32 + lane < E) ? expf(x[j] - mx) : 0.f;
        sum += prob[j];
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    uint32_t key[VPL];
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
        prob[j] = __fdiv_rn(prob[j], sum);
        key[j] = (j * 32 + lane < E) ? order_key(prob[j]) : 0u;
    }
    int my_id = 0;
    float my_w = 0.f;
    const float wsum = select_topk<VPL>(key, prob, topk, lane, [&](int j) { return j * 32 + lane; }, my_id, my_w);
    if (lane < topk) {
        out_w[(int64_t)token * topk + lane] = renorm ? __fdiv_rn(my_w, wsum) : my_w;
        out_id[(int64_t)token * topk + lane] = my_id;
        if (src_row) src_row[(int64_t)token * topk + lane] = lane * tokens + token;
    }
}

template <typename F>
void dispatch_vpl(int E, F&& f) {
    const int need = (E + 31) / 32;
    if (need <= 1) f(std::integral_constant<int, 1>{});
    else if (need <= 2) f(std::integral_constant<int, 2>{});
    else if (need <= 4) f(std::integral_constant<int, 4>{});
    else if (need <= 8) f(std::integral_constant<int, 8>{});
    else if (need <= 16) f(std::integral_constant<int, 16>{});
    else f(std::integral_constant<int, 32>{});
}

void check_outputs(const aiter_tensor_t* gating, const aiter_tensor_t* w, const aiter_tensor_t* ids, int64_t& tokens,
                   int64_t& E, int64_t& topk) {
    check_tensor(gating, "gating_output", -1, 2);
    B200_CHECK(gating->dtype_ == AITER_DTYPE_fp32 || gating->dtype_ == AITER_DTYPE_bf16,
               "gating_output must be fp32 or bf16");
    check_tensor(w, "topk_weights", AITER_DTYPE_fp32, 2);
    check_tensor(ids, "topk_ids", AITER_DTYPE_i32, 2);
    tokens = gating->shape[0];
    E = gating->shape[1];
    topk = ids->shape[1];
    B200_CHECK(E >= 1 && E <= 1024, "number of experts must be in [1, 1024], got ", E);
    B200_CHECK(topk >= 1 && topk <= 32 && topk <= E, "topk must be in [1, min(32, experts)], got ", topk);
    B200_CHECK(w->shape[0] >= tokens && ids->shape[0] >= tokens && w->shape[1] == topk,
               "topk_weights / topk_ids must be [tokens, topk]");
}

}  // namespace

void launch_biased_grouped_topk(const aiter_tensor_t* gating, const aiter_tensor_t* bias, aiter_tensor_t* w,
                                aiter_tensor_t* ids, int n_group, int topk_group, int renorm, float scale,
                                cudaStream_t stream) {
    int64_t tokens, E, topk;
    check_outputs(gating, w, ids, tokens, E, topk);
    check_tensor(bias, "correction_bias", -1, 1);
    B200_CHECK(bias->dtype_ == AITER_DTYPE_fp32 || bias->dtype_ == AITER_DTYPE_bf16, "correction_bias must be fp32 or bf16");
    B200_CHECK((int64_t)bias->numel_ == E, "correction_bias must have one entry per expert");
    B200_CHECK(n_group >= 1 && n_group <= 32 && E % n_group == 0, "num_expert_group must divide the expert count and be <= 32");
    B200_CHECK(topk_group >= 1 && topk_group <= n_group, "topk_group must be in [1, num_expert_group]");
    if (tokens == 0) return;
    const unsigned grid = (unsigned)((tokens + kWarpsPerBlock - 1) / kWarpsPerBlock);
    dispatch_vpl((int)E, [&](auto vpl) {
        constexpr int V = decltype(vpl)::value;
        auto go = [&](auto* g, auto* b) {
            using TG = std::remove_cv_t<std::remove_pointer_t<decltype(g)>>;
            using TB = std::remove_cv_t<std::remove_pointer_t<decltype(b)>>;
            launch_pdl(biased_grouped_topk_kernel<TG, TB, V>, grid, kWarpsPerBlock * 32, 0, stream, g, b, (float*)w->ptr, (int*)ids->ptr, (int)tokens, (int)E, (int)topk, n_group, topk_group, renorm, scale);
        };
        const bool gf = gating->dtype_ == AITER_DTYPE_fp32, bf = bias->dtype_ == AITER_DTYPE_fp32;
        if (gf && bf) go((const float*)gating->ptr, (const float*)bias->ptr);
        else if (gf) go((const float*)gating->ptr, (const __nv_bfloat16*)bias->ptr);
        else if (bf) go((const __nv_bfloat16*)gating->ptr, (const float*)bias->ptr);
        else go((const __nv_bfloat16*)gating->ptr, (const __nv_bfloat16*)bias->ptr);
    });
}

void launch_topk_softmax(aiter_tensor_t* w, aiter_tensor_t* ids, aiter_tensor_t* src_row, const aiter_tensor_t* gating,
                         int renorm, cudaStream_t stream) {
    int64_t tokens, E, topk;
    check_outputs(gating, w, ids, tokens, E, topk);
    if (src_row) {
        check_tensor(src_row, "token_expert_indices", AITER_DTYPE_i32, 2);
        B200_CHECK(src_row->shape[0] >= tokens && src_row->shape[1] == topk, "token_expert_indices must be [tokens, topk]");
    }
    if (tokens == 0) return;
    const unsigned grid = (unsigned)((tokens + kWarpsPerBlock - 1) / kWarpsPerBlock);
    dispatch_vpl((int)E, [&](auto vpl) {
        constexpr int V = decltype(vpl)::value;
        if (gating->dtype_ == AITER_DTYPE_fp32)
            launch_pdl(topk_softmax_kernel<float, V>, grid, kWarpsPerBlock * 32, 0, stream, (const float*)gating->ptr, (float*)w->ptr, (int*)ids->ptr, src_row ? (int*)src_row->ptr : nullptr,
                (int)tokens, (int)E, (int)topk, renorm);
        else
            launch_pdl(topk_softmax_kernel<__nv_bfloat16, V>, grid, kWarpsPerBlock * 32, 0, stream, (const __nv_bfloat16*)gating->ptr, (float*)w->ptr, (int*)ids->ptr, src_row ? (int*)src_row->ptr : nullptr,
                (int)tokens, (int)E, (int)topk, renorm);
    });
}

}  // namespace b200
