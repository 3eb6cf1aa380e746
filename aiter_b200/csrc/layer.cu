// The layer as one host call (b200_fused_moe): the kernels of the separate entry points, enqueued back to back.
//
// What it is for: from Python every entry point costs 10-25 us of host time (argument marshalling, allocator, stream
// lookup), and a decode layer's kernels are over in 50 us: at M=1 the eager layer took 177 us of which the GPU worked 56.

#include <algorithm>

#include "common.cuh"

namespace b200 {

int64_t sorting_workspace_bytes(int tokens, int num_experts, int topk);
int sorting_launches(int64_t routes);
void launch_moe_sorting(const aiter_tensor_t*, const aiter_tensor_t*, aiter_tensor_t*, aiter_tensor_t*,
                        aiter_tensor_t*, aiter_tensor_t*, aiter_tensor_t*, int, int, const aiter_tensor_t*,
                        const aiter_tensor_t*, aiter_tensor_t*, aiter_tensor_t*, const BlockLists*, cudaStream_t);
void launch_quant_1x128(aiter_tensor_t*, const aiter_tensor_t*, aiter_tensor_t*, const aiter_tensor_t*, int, int, bool, cudaStream_t);
void launch_quant_per_token(aiter_tensor_t*, const aiter_tensor_t*, aiter_tensor_t*, const aiter_tensor_t*, int, bool,
                            const int*, int, cudaStream_t);
void launch_quant_per_tensor(aiter_tensor_t*, const aiter_tensor_t*, aiter_tensor_t*, aiter_tensor_t*, aiter_tensor_t*,
                             const aiter_tensor_t*, bool, bool, const int*, int, cudaStream_t);
void launch_moe_stage1(const aiter_tensor_t*, const aiter_tensor_t*, const aiter_tensor_t*, const aiter_tensor_t*,
                       const aiter_tensor_t*, const aiter_tensor_t*, const aiter_tensor_t*, aiter_tensor_t*,
                       aiter_tensor_t*, aiter_tensor_t*, int, const aiter_tensor_t*, int, bool, unsigned*, bool, SortedStage*, cudaStream_t);
void launch_moe_stage2(const aiter_tensor_t*, const aiter_tensor_t*, const aiter_tensor_t*, const aiter_tensor_t*,
                       const aiter_tensor_t*, const aiter_tensor_t*, const aiter_tensor_t*, const aiter_tensor_t*,
                       aiter_tensor_t*, aiter_tensor_t*, int, int, int, int, int, bool, SortedStage*, cudaStream_t);
void launch_gather_rows(const void*, const float*, void*, float*, const int*, const int*, int64_t, int64_t, int64_t, cudaStream_t);
void launch_finalize(aiter_tensor_t*, const aiter_tensor_t*, cudaStream_t);

namespace {

constexpr int kQuantPerTensor = 1, kQuantPerToken = 2;   // QuantType of the reference (csrc/include/aiter_enum.h:16-26)
constexpr int64_t kUnit = 128;                           // sort unit == row tile of the GEMM kernels

// What tests ask of the calls of their thread (b200_moe_debug_pairs): 0 the rule below, 1 pairs wherever there can be one, 2 none.
thread_local int t_debug_pairs = 0;

// Which layers work their row blocks in pairs (moe_gemm_sorted.cu). E: experts of this layer call, of global_E that are routed to.
// padded: how many of the M tokens are live stands on the device.
// Timed both ways in turn as graphs: 1132 block-scaled and 699 row-scaled layers, H 512 to 8192, I 1024 to 14336, 8 to 256 experts, 150
// to 1024 rows an expert, even and Zipf routing. Gain: time with one block a CTA / time in pairs, mean (least).
//  * Rows. Below 144 an expert most have one block. With three blocks each expert leaves one single, at the price of a pair: block
//    scales with 7 / 12 to 14 / 29 / 50 rounds of tiles 0.99 / 1.00 to 1.02 / 1.03 / 1.03 at 265 to 375 rows an expert; row scales with
//    I 4096 / 6144 / 8192 / 10880 / 14336 0.98 (0.96) / 1.00 (0.95) / 0.97 (0.92) / 1.01 / 1.01, and with I 4096 at five blocks 0.99
//    (0.97). Zipf routing, where the experts differ, gains 1.01 to 1.06 there, but the host does not see the routing.
//  * Block scales, stage 2 only: a second launch, 2 to 4 us, and tiles of twice the size want several rounds of tiles. By rounds of
//    128 x 256 tiles on all SMs below 1: 0.94 (0.88), 1-3: 0.98 (0.90), 3-6: 1.00 (0.95), 6-12: 1.02, 12-24: 1.03, above: 1.05.
//  * Row scales, both stages: three launches and a copy of the rows, 10 to 20 us, against a gain that grows with the rounds of
//    stage 1 and with I, less below H 4096. Three blocks aside, the 291 layers beyond the line 1.085 (0.986; with I 4096 / 6144 / 8192 /
//    14336 1.03 / 1.07 / 1.08 / 1.10), the 408 before it 1.00 (0.80).
//  * Padded batches. What pays for the pairs is rows that the host does not know to be there: with all / a half / a quarter / a 64th of
//    the tokens live, Mixtral-shaped 4097 tokens 1.16 / 1.04 / 1.06 / 0.95 (row scales) and 1.02 / 1.01 / 1.01 / 0.98, DeepSeek-V3-shaped
//    8193 tokens 1.05 / 1.02 / 0.99 / 0.97, a quarter of its experts and 6401 tokens 1.03 / 0.98 / 0.99 / 0.99 (block scales).
bool works_in_pairs(int64_t M, int64_t H, int64_t I, int64_t E, int64_t global_E, int64_t topk, bool rowwise, bool padded) {
    constexpr double kSms = 148;
    const int64_t routes = M * topk;
    if (t_debug_pairs) return t_debug_pairs == 1 && routes > kUnit;
    if (padded || global_E < 1 || routes < 144 * global_E || routes <= kUnit) return false;
    const int64_t rows = routes / global_E, blocks = (rows + kUnit - 8) / kUnit;     // an expert
    const int64_t odd = blocks % 2 && (rows + 8) / kUnit < blocks ? blocks : 0;      // most experts have this odd number of blocks
    const double here = (double)routes * std::min(E, global_E) / global_E / kUnit;   // blocks of rows in this call
    if (!rowwise) return I >= 1024 && here * H / 256 >= (odd == 3 ? 12 : 6) * kSms;
    if ((odd == 3 && I < 10240) || (odd == 5 && I < 6144)) return false;
    return I >= 4096 && H >= 2048 && here * I / 128 / kSms * I * std::min<int64_t>(H, 4096) >= 98304. * 4096;
}

// Workspace map: every buffer starts on a 256-byte boundary. Offsets depend on sizes only.
struct Layout {
    bool pairs;
    int64_t max_pairs, max_singles, lists, P, ld, sorted_ids, sorted_w, sorted_eids, num_valid, sort_ws, acc, a1, a1_scale, a2, a2_scale,
        a2_half, words, rows, rows_scale, total;
    Layout(int64_t M, int64_t H, int64_t I, int64_t E, int64_t topk, int qt, bool fp8_in, bool in_pairs) {
        const bool rowwise = qt == kQuantPerToken || qt == kQuantPerTensor;
        pairs = in_pairs;
        P = M * topk + E * kUnit - topk;
        ld = (P + 31) / 32 * 32;                 // row of a transposed scale array
        int64_t at = 0;
        auto take = [&](int64_t bytes) {
            const int64_t o = at;
            at += (bytes + 255) / 256 * 256;
            return o;
        };
        sorted_ids = take(P * 4);
        sorted_w = take(P * 4);
        sorted_eids = take((P + kUnit - 1) / kUnit * 4);
        num_valid = take(8);
        max_pairs = M * topk / (kUnit + 1);      // a pair needs more than one block's rows
        max_singles = std::min(E, M * topk);     // at most one per expert
        lists = take(pairs ? (2 + max_pairs + max_singles) * 4 : 0);
        sort_ws = take(sorting_workspace_bytes((int)M, (int)E, (int)topk));
        a1_scale = take(M * (rowwise ? 1 : H / 128) * 4);
        a2_scale = take(rowwise ? P * 4 : pairs ? ld * ((I + 511) / 512 * 4) * 4 : P * (I / 128) * 4);
        words = take(256);                       // per_Tensor: a maximum and a scale word per quantisation
        acc = take(M * H * 4);
        a1 = take(fp8_in ? 0 : M * H);
        a2 = take(P * I);
        a2_half = take(rowwise ? P * I * 2 : 0);  // stage-1 activation before the row requantisation
        rows_scale = take(pairs && rowwise ? P * 4 : 0);
        rows = take(pairs && rowwise ? P * H : 0);   // activation rows in sorted order
        total = at;
    }
};

aiter_tensor_t tensor(const void* ptr, int dtype, int dev, int64_t d0, int64_t d1 = -1, int64_t d2 = -1) {
    aiter_tensor_t t{};
    t.ptr = const_cast<void*>(ptr);
    t.dtype_ = dtype;
    t.device_id = dev;
    const int64_t d[3] = {d0, d1, d2};
    t.ndim = d2 >= 0 ? 3 : d1 >= 0 ? 2 : 1;
    int64_t n = 1;
    for (int i = t.ndim - 1; i >= 0; --i) {
        t.shape[i] = d[i];
        t.strides[i] = n;
        n *= d[i];
    }
    t.numel_ = (size_t)n;
    return t;
}

bool rowwise_quant(int qt) { return qt == kQuantPerToken || qt == kQuantPerTensor; }

}  // namespace

void set_debug_pairs(int mode) { t_debug_pairs = mode; }

// For every number of local experts and live tokens: with all of them here a layer is worked in pairs at the fewest tokens.
int64_t fused_moe_workspace_bytes(int64_t M, int64_t H, int64_t I, int64_t E, int64_t topk, int qt, int hidden_dtype) {
    return Layout(M, H, I, E, topk, qt, hidden_dtype == AITER_DTYPE_fp8, works_in_pairs(M, H, I, E, E, topk, rowwise_quant(qt), false)).total;
}

// Kernels that launch_fused_moe below enqueues for these sizes.
int fused_moe_launches(int64_t M, int64_t H, int64_t I, int64_t E, int64_t global_E, int64_t topk, int qt, int hidden_dtype,
                       bool padded) {
    const bool per_tensor = qt == kQuantPerTensor, rowwise = rowwise_quant(qt);
    const bool pairs = works_in_pairs(M, H, I, E, global_E, topk, rowwise, padded);
    int n = sorting_launches(M * topk);
    if (hidden_dtype != AITER_DTYPE_fp8) n += per_tensor ? 2 : 1;   // maximum, codes
    n += pairs && rowwise ? 3 : 1;                                  // stage 1: rows in order, pairs, single blocks
    n += rowwise ? 1 : 0;                                           // requantisation
    n += pairs ? 2 : 1;                                             // stage 2
    return n + 1;                                                   // final rounding
}

void launch_fused_moe(const b200_fused_moe_args& a, cudaStream_t stream) {
    const int dev = (int)a.device, qt = (int)a.quant_type;
    const int64_t M = a.M, H = a.H, I = a.I, E = a.E;
    const bool fp8_in = a.hidden_dtype == AITER_DTYPE_fp8;
    const bool per_tensor = qt == kQuantPerTensor, rowwise = rowwise_quant(qt);
    B200_CHECK(M >= 1 && H >= 1 && I >= 1 && E >= 1 && a.global_E >= 1 && a.topk >= 1, "sizes must be positive");
    B200_CHECK(a.workspace != nullptr && ((uintptr_t)a.workspace & 255) == 0, "workspace must be 256-byte aligned");
    Layout at(M, H, I, a.global_E, a.topk, qt, fp8_in, works_in_pairs(M, H, I, E, a.global_E, a.topk, rowwise, a.num_local_tokens != nullptr));
    if (at.pairs && a.workspace_bytes < at.total)   // no room for the pairs' lists and rows: one block a CTA asks for less
        at = Layout(M, H, I, a.global_E, a.topk, qt, fp8_in, false);
    B200_CHECK(a.workspace_bytes >= at.total, "workspace needs ", at.total, " bytes, has ", a.workspace_bytes);
    char* ws = (char*)a.workspace;
    const int F32 = AITER_DTYPE_fp32, I32 = AITER_DTYPE_i32, FP8 = AITER_DTYPE_fp8;

    aiter_tensor_t ids = tensor(a.topk_ids, I32, dev, M, a.topk), wts = tensor(a.topk_weight, F32, dev, M, a.topk);
    aiter_tensor_t s_ids = tensor(ws + at.sorted_ids, I32, dev, at.P), s_w = tensor(ws + at.sorted_w, F32, dev, at.P);
    aiter_tensor_t s_e = tensor(ws + at.sorted_eids, I32, dev, (at.P + kUnit - 1) / kUnit), nv = tensor(ws + at.num_valid, I32, dev, 2);
    aiter_tensor_t acc = tensor(ws + at.acc, F32, dev, M, H),
                   cleared = tensor(ws + at.words, F32, dev, 64 + M * H), status = tensor(a.status, I32, dev, 1);
    aiter_tensor_t mask = tensor(a.expert_mask, I32, dev, a.global_E), live = tensor(a.num_local_tokens, I32, dev, 1);
    const int64_t sort_bytes = sorting_workspace_bytes((int)M, (int)a.global_E, (int)a.topk);
    aiter_tensor_t sort_ws = tensor(ws + at.sort_ws, AITER_DTYPE_u8, dev, sort_bytes);
    BlockLists lists;
    lists.counts = (int*)(ws + at.lists);
    lists.pairs = lists.counts + 2;
    lists.singles = lists.pairs + at.max_pairs;
    lists.max_pairs = at.max_pairs;
    lists.max_singles = at.max_singles;
    launch_moe_sorting(&ids, &wts, &s_ids, &s_w, &s_e, &nv, &cleared, (int)a.global_E, (int)kUnit, a.expert_mask ? &mask : nullptr,
                       a.num_local_tokens ? &live : nullptr, sort_bytes ? &sort_ws : nullptr, nullptr, at.pairs ? &lists : nullptr, stream);

    aiter_tensor_t hidden = tensor(a.hidden, (int)a.hidden_dtype, dev, M, H);
    aiter_tensor_t a1 = hidden, a1_s = rowwise ? tensor(ws + at.a1_scale, F32, dev, M) : tensor(ws + at.a1_scale, F32, dev, M, H / 128);
    // the sort clears the accumulator and the words in front of it; the quantiser runs beside the sort
    aiter_tensor_t one = tensor(ws + at.words, F32, dev, 1), amax = tensor(ws + at.words + 64, F32, dev, 1);
    aiter_tensor_t one2 = tensor(ws + at.words + 128, F32, dev, 1), amax2 = tensor(ws + at.words + 192, F32, dev, 1);
    if (fp8_in) {
        B200_CHECK(a.a1_scale != nullptr, "fp8 hidden states need a1_scale");
        a1_s = tensor(a.a1_scale, F32, dev, a.a1_scale_numel);
    } else {
        a1 = tensor(ws + at.a1, FP8, dev, M, H);
        if (per_tensor) launch_quant_per_tensor(&a1, &hidden, &one, &amax, nullptr, nullptr, true, false, nullptr, 0, stream), a1_s = one;
        else if (rowwise) launch_quant_per_token(&a1, &hidden, &a1_s, nullptr, 1, false, nullptr, 0, stream);
        else launch_quant_1x128(&a1, &hidden, &a1_s, nullptr, 1, 0, false, stream);
    }

    aiter_tensor_t w1 = tensor(a.w1, FP8, dev, E, 2 * I, H), w1_s = tensor(a.w1_scale, F32, dev, a.w1_scale_numel);
    aiter_tensor_t w2 = tensor(a.w2, FP8, dev, E, H, I), w2_s = tensor(a.w2_scale, F32, dev, a.w2_scale_numel);
    aiter_tensor_t a2 = tensor(ws + at.a2, FP8, dev, at.P, I);
    aiter_tensor_t a2_s = rowwise ? tensor(ws + at.a2_scale, F32, dev, at.P) : tensor(ws + at.a2_scale, F32, dev, at.P, I / 128);
    const int gemm_qt = rowwise ? kQuantPerToken : qt;   // one scale per tensor runs through the row-scale kernels
    const aiter_tensor_t* w_stage1 = a.doweight_stage1 ? &s_w : nullptr;
    SortedStage stage{};
    SortedStage* in_order = at.pairs ? &stage : nullptr;
    if (at.pairs) {
        stage.sorted_ids = (const int*)s_ids.ptr;
        stage.sorted_w = (const float*)s_w.ptr;
        stage.sorted_eids = (const int*)s_e.ptr;
        stage.num_valid = (const int*)nv.ptr;
        stage.status = (int*)a.status;
        stage.lists = lists;
        stage.M = M, stage.H = H, stage.I = I, stage.E = E, stage.P = at.P, stage.ld = (int)at.ld;
        stage.device = dev;
        stage.rowwise = rowwise;
    }
    if (at.pairs && rowwise) {
        const bool per_row = (int64_t)a1_s.numel_ == M;   // else one for all
        float* scales = (float*)(ws + at.rows_scale);
        launch_gather_rows(a1.ptr, per_row ? (const float*)a1_s.ptr : nullptr, ws + at.rows, scales, stage.sorted_ids, stage.num_valid, M, H, at.P, stream);
        stage.rows = ws + at.rows;
        stage.a_scale = per_row ? scales : (const float*)a1_s.ptr;
        stage.a_scale_ld = per_row;
    }
    if (rowwise) {
        aiter_tensor_t half = tensor(ws + at.a2_half, AITER_DTYPE_bf16, dev, at.P, I);
        launch_moe_stage1(&a1, &a1_s, &w1, &w1_s, &s_ids, &s_e, &nv, &half, nullptr, &status, gemm_qt, w_stage1, (int)a.activation, true,
                          per_tensor ? (unsigned*)amax2.ptr : nullptr, per_tensor, in_order, stream);
        if (per_tensor) launch_quant_per_tensor(&a2, &half, &one2, &amax2, nullptr, &nv, true, true, (const int*)s_ids.ptr, (int)M, stream), a2_s = one2;
        else launch_quant_per_token(&a2, &half, &a2_s, &nv, 1, true, (const int*)s_ids.ptr, (int)M, stream);
    } else {
        launch_moe_stage1(&a1, &a1_s, &w1, &w1_s, &s_ids, &s_e, &nv, &a2, &a2_s, &status, gemm_qt, w_stage1, (int)a.activation, true, nullptr, false, in_order, stream);
    }
    launch_moe_stage2(&a2, &a2_s, &w2, &w2_s, &s_ids, &s_w, &s_e, &nv, &acc, &status, 0, 0, 0, gemm_qt, a.doweight_stage1 ? 0 : 1, per_tensor, in_order, stream);
    aiter_tensor_t out = tensor(a.out, (int)a.out_dtype, dev, M, H);
    launch_finalize(&out, &acc, stream);
}

}  // namespace b200
