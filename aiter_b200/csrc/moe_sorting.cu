// moe_sorting for sm_100a: stable counting sort of (token, slot) routes by expert, every
// expert padded to a multiple of unit_size.  Output contract of the reference's native sort
// (csrc/include/moe_sorting_opus.h:280-359) with the padding values of its torch oracle
// (op_tests/test_moe_sorting.py:45-99).
//
// Route r = token*topk + slot.  Within an expert routes keep ascending r, which is the order torch.where() yields in the
// oracle.  The position of a route is
//     base[expert] + (routes of that expert in earlier chunks) + (in earlier 32-route runs of its chunk)
//                  + (in lower lanes of its run)
// where the last term comes from __match_any_sync + popc and the third from one byte per (expert, run) that the run's
// leader lane writes: no atomics on the output side, the result is deterministic.
//
// Launch shapes (a chunk is 4096 routes, one CTA of 1024 threads):
//   routes <= kSingleMaxRoutes  one kernel; every CTA counts the other chunks' routes itself (a few shared-memory atomics
//                               per thread), which is cheaper than a grid-wide dependency;
//   more                        count per chunk -> scatter, whose CTAs each add up the per-chunk counts, with the counts in
//                               a caller-provided workspace. (A scan kernel in between, one CTA for all experts, was 9 us
//                               at 24 K routes and 50 us with the fill of a 235 MB moe_buf beside it.)
// What bounds it: latency, a handful of dependent phases of one CTA. Padding entries and block ids are written by warps,
// an expert each: a thread per expert wrote up to 127 pads one after the other, 12-27 us of decode layers.
// Measured (DeepSeek-V3 routing, unit 128): 64 tokens 26 -> 5 us, 3001 tokens (unit 32) 20 -> 11 us.
// Extra CTAs zero-fill moe_buf when the caller passes one.

#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace b200 {
namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kChunk = 4096;            // routes per sorting CTA
constexpr int kSingleMaxRoutes = 16384; // above this the two-kernel path is used
constexpr int kMaxExperts = 1024;

struct SortArgs {
    const int* ids;
    const float* weights;
    const int* mask;       // [E] or null
    const int* num_local;  // [1] or null
    int* sorted_ids;
    float* sorted_w;
    int* sorted_eids;
    int* num_valid;
    int* local_topk_ids;   // [M*topk] or null
    int* ws_cnt;           // [nchunks*E]   (two-kernel path only)
    uint4* zero_buf;       // moe_buf or null
    size_t zero_vec16;     // number of 16-byte words to clear
    unsigned char* zero_tail;
    int zero_tail_bytes;
    int M, topk, E, unit;
    int max_padded, max_blocks;
    int nchunks;           // CTAs that sort
    int runs;              // 32-route runs per chunk: 32 times the rounds of kThreads routes a CTA makes
};

// ... and lists the pairs and single blocks besides (BlockLists). A type of its own, so that the sorts of all other callers
// carry none of it: with the lists behind a branch of the one kernel a one-token layer took 49.7 us, without them 47.9.
struct SortArgsLists : SortArgs {
    int* counts;           // {pairs, singles}
    int* pairs;
    int* singles;
};

__device__ __forceinline__ int eff_tokens(const SortArgs& a) {
    int t = a.M;
    if (a.num_local) {
        int v = *a.num_local;
        v = v < 0 ? 0 : v;
        t = v < t ? v : t;
    }
    return t;
}

// Exclusive scans of two ints per thread over the whole CTA (kThreads threads).
__device__ __forceinline__ void block_scan2_excl(int& u, int& v, int2* warp_tot, int& total_v) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int iu = u, iv = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int nu = __shfl_up_sync(0xffffffffu, iu, d), nv = __shfl_up_sync(0xffffffffu, iv, d);
        if (lane >= d) {
            iu += nu;
            iv += nv;
        }
    }
    if (lane == 31) warp_tot[warp] = make_int2(iu, iv);
    __syncthreads();
    // every warp adds up the totals before it (no second round trip through shared memory)
    const int2 t = warp_tot[lane];
    const bool before = lane < warp;
    const int bu = __reduce_add_sync(0xffffffffu, before ? t.x : 0), bv = __reduce_add_sync(0xffffffffu, before ? t.y : 0);
    total_v = __reduce_add_sync(0xffffffffu, t.y);
    u = bu + iu - u;
    v = bv + iv - v;
}

__device__ __forceinline__ void zero_fill(const SortArgs& a, int part, int nparts) {
    const uint4 z = make_uint4(0, 0, 0, 0);
    for (size_t i = (size_t)part * kThreads + threadIdx.x; i < a.zero_vec16;
         i += (size_t)nparts * kThreads)
        a.zero_buf[i] = z;
    if (part == 0 && (int)threadIdx.x < a.zero_tail_bytes) a.zero_tail[threadIdx.x] = 0;
}

__device__ __forceinline__ int byte_sum(uint32_t w, int acc) { return __dp4a(w, 0x01010101u, (unsigned)acc); }

// Sum of the first n bytes of a 16-byte aligned row (n up to its length).
__device__ __forceinline__ int prefix_bytes(const unsigned char* row, int n) {
    const uint4* p = reinterpret_cast<const uint4*>(row);
    int s = 0;
    for (; n >= 16; n -= 16, ++p) {
        const uint4 x = *p;
        s = byte_sum(x.w, byte_sum(x.z, byte_sum(x.y, byte_sum(x.x, s))));
    }
    if (n > 0) {
        const uint4 x = *p;
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int nb = n - 4 * k;
            if (nb > 0) s = byte_sum(nb >= 4 ? w[k] : w[k] & ((1u << (8 * nb)) - 1u), s);
        }
    }
    return s;
}

extern __shared__ __align__(16) unsigned char smem_b[];
// smem of the sorting CTAs: run_cnt[E][row_bytes] | before[E] | after[E] | start[E] | base[E] | warp_tot[32]; with lists, behind it:
// warp_tot2[32] | pairs_at[E]
__host__ __device__ inline int row_bytes(int runs) { return runs + 16; }   // + 16: rows start in different banks
inline size_t sort_smem(int E, int runs, bool with_lists) {
    return (size_t)E * row_bytes(runs) + 4 * (size_t)E * sizeof(int) + 32 * sizeof(int2) + (with_lists ? 32 * sizeof(int2) + (size_t)E * sizeof(int) : 0);
}

// FROM_WS: the routes of the other chunks come from the counts in the workspace; else they are counted here.
template <bool FROM_WS, typename Args>
__global__ void __launch_bounds__(kThreads, 1) sort_kernel(Args a) {
    constexpr bool kLists = std::is_same<Args, SortArgsLists>::value;
    if ((int)blockIdx.x >= a.nchunks) {
        // the fill beside the two-kernel sort starts at once: the kernel before it is the count, which does not touch moe_buf
        if (!FROM_WS) pdl_wait();
        pdl_trigger();
        zero_fill(a, blockIdx.x - a.nchunks, gridDim.x - a.nchunks);
        if (FROM_WS) pdl_wait();
        return;
    }
    const int rb = row_bytes(a.runs), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned char* run_cnt = smem_b;
    int* before = reinterpret_cast<int*>(smem_b + (size_t)a.E * rb);   // routes of e in earlier chunks
    int* after = before + a.E;                                         // ... in later chunks
    int* start = after + a.E;    // position of this chunk's first route of e, -1: expert dropped
    int* base = start + a.E;     // first position of e
    int2* warp_tot = reinterpret_cast<int2*>(base + a.E);
    int* pairs_at = reinterpret_cast<int*>(warp_tot + 64);   // pairs of blocks of the experts before e
    for (int i = tid; i < a.E * rb / 16; i += kThreads) reinterpret_cast<uint4*>(run_cnt)[i] = make_uint4(0, 0, 0, 0);
    for (int i = tid; i < a.E; i += kThreads) before[i] = after[i] = 0;
    pdl_wait();
    pdl_trigger();
    const int tokens = eff_tokens(a);
    const int routes = tokens * a.topk;
    const int c = blockIdx.x, r0 = min(c * kChunk, routes), r1 = min(r0 + kChunk, routes);
    // this chunk's ids and weights, kept in registers
    const int rounds = a.runs / kWarps;
    int e[kChunk / kThreads], rank[kChunk / kThreads];
    float w[kChunk / kThreads];
#pragma unroll
    for (int q = 0; q < kChunk / kThreads; ++q) {
        const int i = r0 + q * kThreads + tid;
        const bool in = q < rounds && i < r1;
        e[q] = in ? a.ids[i] : -1;
        w[q] = in ? a.weights[i] : 0.f;
        if (e[q] >= a.E) e[q] = -1;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kChunk / kThreads; ++q) {
        if (q >= rounds) break;
        const bool live = e[q] >= 0;
        const unsigned grp = __match_any_sync(0xffffffffu, live ? e[q] : a.E + lane);   // lanes without a route: a key each
        rank[q] = __popc(grp & ((1u << lane) - 1u));
        if (live && rank[q] == 0) run_cnt[e[q] * rb + q * kWarps + warp] = (unsigned char)__popc(grp);
    }
    if (FROM_WS) {
        // thread (part, expert): parts of the chunks in parallel, eight loads in flight each
        const int parts = kThreads / a.E;   // E <= kThreads
        const int ex = tid % a.E, part = tid / a.E;
        if (part < parts) {
            int b = 0, f = 0;
            for (int k0 = part; k0 < a.nchunks; k0 += 8 * parts) {
                int v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int ch = k0 + k * parts;
                    v[k] = ch < a.nchunks ? __ldcg(a.ws_cnt + (size_t)ch * a.E + ex) : 0;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int ch = k0 + k * parts;
                    b += ch < c ? v[k] : 0;
                    f += ch > c ? v[k] : 0;
                }
            }
            if (b) atomicAdd(before + ex, b);
            if (f) atomicAdd(after + ex, f);
        }
    } else {
        for (int i = tid; i < routes; i += kThreads)
            if (i < r0 || i >= r1) {
                const int x = a.ids[i];
                if (x >= 0 && x < a.E) atomicAdd((i < r0 ? before : after) + x, 1);
            }
    }
    __syncthreads();
    // layout: thread e owns expert e
    int cnt = 0, lid = 0, at = 0, total;
    bool keep = false;
    if (tid < a.E) {
        keep = a.mask ? a.mask[tid] != 0 : true;
        cnt = before[tid] + after[tid] + prefix_bytes(run_cnt + tid * rb, a.runs);
    }
    const int padded = keep ? (cnt + a.unit - 1) / a.unit * a.unit : 0;
    lid = keep ? 1 : 0;
    at = padded;
    block_scan2_excl(lid, at, warp_tot, total);   // local expert id, first position
    if constexpr (kLists) {
        int np = padded / a.unit / 2, ns = padded / a.unit & 1, singles;
        const int mine = np;
        block_scan2_excl(np, ns, warp_tot + 32, singles);
        if (tid < a.E) pairs_at[tid] = np;
        if (c == 0 && tid == a.E - 1) {
            a.counts[0] = np + mine;
            a.counts[1] = singles;
        }
    }
    if (tid < a.E) {
        start[tid] = keep ? at + before[tid] : -1;
        base[tid] = keep ? at : -1;
        after[tid] = cnt;       // from here on: routes of e in all chunks
        before[tid] = lid;      // ... and the local id
    }
    if (c == 0 && tid == 0) {
        a.num_valid[0] = total;
        a.num_valid[1] = tokens;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kChunk / kThreads; ++q) {
        if (q >= rounds) break;
        const int i = r0 + q * kThreads + tid;
        const int s = e[q] >= 0 ? start[e[q]] : -1;
        if (i < r1 && a.local_topk_ids) a.local_topk_ids[i] = s >= 0 ? before[e[q]] : -1;
        if (s >= 0) {
            const int pos = s + prefix_bytes(run_cnt + e[q] * rb, q * kWarps + warp) + rank[q];
            const int token = i / a.topk;
            a.sorted_ids[pos] = ((i - token * a.topk) << 24) | token;
            a.sorted_w[pos] = w[q];
        }
    }
    // expert ids of the blocks and pad entries: a warp per expert; then the tail past the padded total
    const int pad_id = (a.topk << 24) | a.M;
    for (int x = c * kWarps + warp; x < a.E; x += a.nchunks * kWarps) {
        const int n = after[x], b = base[x];
        if (b < 0 || n == 0) continue;
        const int end = b + (n + a.unit - 1) / a.unit * a.unit;
        for (int k = b / a.unit + lane; k < end / a.unit; k += 32) a.sorted_eids[k] = before[x];
        if constexpr (kLists) {
            const int first = b / a.unit, blocks = (end - b) / a.unit, at = pairs_at[x];
            for (int k = lane; k < blocks / 2; k += 32) a.pairs[at + k] = first + 2 * k;
            if ((blocks & 1) && lane == 0) a.singles[first - 2 * at] = first + blocks - 1;   // blocks before, less those in pairs
        }
        for (int p = b + n + lane; p < end; p += 32) {
            a.sorted_ids[p] = pad_id;
            a.sorted_w[p] = 0.f;
        }
    }
    const int part = c * kThreads + tid, nparts = a.nchunks * kThreads;
    for (int k = total / a.unit + part; k < a.max_blocks; k += nparts) a.sorted_eids[k] = -1;
    for (int p = total + part; p < a.max_padded; p += nparts) {
        a.sorted_ids[p] = pad_id;
        a.sorted_w[p] = 0.f;
    }
    if (a.local_topk_ids)
        for (int i = routes + part; i < a.M * a.topk; i += nparts) a.local_topk_ids[i] = -1;
}

// Routes per (chunk, expert) for the two-kernel path.
__global__ void __launch_bounds__(kThreads, 1) sort_count_kernel(SortArgs a) {
    int* hist = reinterpret_cast<int*>(smem_b);
    for (int i = threadIdx.x; i < a.E; i += kThreads) hist[i] = 0;
    pdl_wait();
    pdl_trigger();
    const int routes = eff_tokens(a) * a.topk;
    const int r0 = min((int)blockIdx.x * kChunk, routes), r1 = min(r0 + kChunk, routes);
    int e[kChunk / kThreads];
#pragma unroll
    for (int q = 0; q < kChunk / kThreads; ++q) {
        const int i = r0 + q * kThreads + threadIdx.x;
        e[q] = i < r1 ? a.ids[i] : -1;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kChunk / kThreads; ++q)
        if (e[q] >= 0 && e[q] < a.E) atomicAdd(hist + e[q], 1);
    __syncthreads();
    for (int i = threadIdx.x; i < a.E; i += kThreads) a.ws_cnt[(size_t)blockIdx.x * a.E + i] = hist[i];
}

inline int num_chunks(int64_t routes) { return (int)((routes + kChunk - 1) / kChunk); }

}  // namespace

// One counter per chunk and expert, and one more row that nothing uses: the size is part of the ABI (callers may have stored
// it, and the static scratch below is stated in bytes).
int64_t sorting_workspace_bytes(int tokens, int num_experts, int topk) {
    int64_t routes = (int64_t)tokens * topk;
    if (routes <= kSingleMaxRoutes) return 0;
    return ((int64_t)num_chunks(routes) * num_experts + num_experts) * (int64_t)sizeof(int);
}

int sorting_launches(int64_t routes) { return routes <= kSingleMaxRoutes ? 1 : 2; }

void launch_moe_sorting(const aiter_tensor_t* topk_ids, const aiter_tensor_t* topk_weights,
                        aiter_tensor_t* sorted_ids, aiter_tensor_t* sorted_w,
                        aiter_tensor_t* sorted_eids, aiter_tensor_t* num_valid,
                        aiter_tensor_t* moe_buf, int E, int unit, const aiter_tensor_t* mask,
                        const aiter_tensor_t* num_local, aiter_tensor_t* workspace,
                        aiter_tensor_t* local_topk_ids, const BlockLists* lists, cudaStream_t stream) {
    check_tensor(topk_ids, "topk_ids", AITER_DTYPE_i32, 2);
    check_tensor(topk_weights, "topk_weights", -1, 2);
    B200_CHECK(topk_weights->dtype_ == AITER_DTYPE_fp32, "topk_weights must be FP32 (float32)");
    check_tensor(sorted_ids, "sorted_token_ids", AITER_DTYPE_i32, 1);
    check_tensor(sorted_w, "sorted_weights", AITER_DTYPE_fp32, 1);
    check_tensor(sorted_eids, "sorted_expert_ids", AITER_DTYPE_i32, 1);
    check_tensor(num_valid, "num_valid_ids", AITER_DTYPE_i32, 1);
    const int64_t M = topk_ids->shape[0], topk = topk_ids->shape[1];
    B200_CHECK(topk_weights->shape[0] == M && topk_weights->shape[1] == topk,
               "topk_weights must have the [tokens, topk] shape of topk_ids");
    B200_CHECK(E >= 1 && E <= kMaxExperts, "num_experts must be in [1, ", kMaxExperts, "], got ", E);
    B200_CHECK(unit >= 1, "unit_size must be positive, got ", unit);
    // ids pack the token in 24 bits and the slot in 8 (csrc/include/moe_sorting_opus.h:273-274)
    B200_CHECK(M < (1 << 24), "tokens must be < 2^24, got ", M);
    B200_CHECK(topk >= 1 && topk < 256, "topk must be in [1, 255], got ", topk);
    const int64_t max_padded = M * topk + (int64_t)E * unit - topk;
    B200_CHECK(max_padded < (int64_t)1 << 31, "problem too large");
    const int64_t max_blocks = (max_padded + unit - 1) / unit;
    B200_CHECK((int64_t)sorted_ids->numel_ >= max_padded, "sorted_token_ids needs ", max_padded,
               " elements, has ", sorted_ids->numel_);
    B200_CHECK((int64_t)sorted_w->numel_ >= max_padded, "sorted_weights needs ", max_padded,
               " elements, has ", sorted_w->numel_);
    B200_CHECK((int64_t)sorted_eids->numel_ >= max_blocks, "sorted_expert_ids needs ", max_blocks,
               " elements, has ", sorted_eids->numel_);
    B200_CHECK(num_valid->numel_ >= 2, "num_valid_ids needs 2 elements");
    if (mask) {
        check_tensor(mask, "local_expert_mask", AITER_DTYPE_i32, 1);
        B200_CHECK((int64_t)mask->numel_ == E, "local_expert_mask must have num_experts entries");
    }
    if (num_local) {
        check_tensor(num_local, "num_local_tokens", AITER_DTYPE_i32, -1);
        B200_CHECK(num_local->numel_ >= 1, "num_local_tokens is empty");
    }
    if (local_topk_ids) {
        check_tensor(local_topk_ids, "local_topk_ids", AITER_DTYPE_i32, 2);
        B200_CHECK(local_topk_ids->shape[0] == M && local_topk_ids->shape[1] == topk,
                   "local_topk_ids must have the same [tokens, topk] shape as topk_ids");
    }

    SortArgsLists a{};
    a.ids = (const int*)topk_ids->ptr;
    a.weights = (const float*)topk_weights->ptr;
    a.mask = mask ? (const int*)mask->ptr : nullptr;
    a.num_local = num_local ? (const int*)num_local->ptr : nullptr;
    a.sorted_ids = (int*)sorted_ids->ptr;
    a.sorted_w = (float*)sorted_w->ptr;
    a.sorted_eids = (int*)sorted_eids->ptr;
    a.num_valid = (int*)num_valid->ptr;
    a.local_topk_ids = local_topk_ids ? (int*)local_topk_ids->ptr : nullptr;
    a.M = (int)M;
    a.topk = (int)topk;
    a.E = E;
    a.unit = unit;
    a.max_padded = (int)max_padded;
    a.max_blocks = (int)max_blocks;
    if (lists) {
        a.counts = lists->counts;
        a.pairs = lists->pairs;
        a.singles = lists->singles;
    }

    int zero_ctas = 0;
    if (moe_buf && moe_buf->numel_ > 0) {
        check_tensor(moe_buf, "moe_buf", -1, -1);
        size_t esz = (moe_buf->dtype_ == AITER_DTYPE_fp32 || moe_buf->dtype_ == AITER_DTYPE_i32 ||
                      moe_buf->dtype_ == AITER_DTYPE_u32) ? 4
                   : (moe_buf->dtype_ == AITER_DTYPE_bf16 || moe_buf->dtype_ == AITER_DTYPE_fp16 ||
                      moe_buf->dtype_ == AITER_DTYPE_i16) ? 2
                   : (moe_buf->dtype_ == AITER_DTYPE_i64 || moe_buf->dtype_ == AITER_DTYPE_u64) ? 8 : 1;
        size_t bytes = moe_buf->numel_ * esz;
        B200_CHECK(((uintptr_t)moe_buf->ptr & 15) == 0, "moe_buf must be 16-byte aligned");
        a.zero_buf = (uint4*)moe_buf->ptr;
        a.zero_vec16 = bytes / 16;
        a.zero_tail = (unsigned char*)moe_buf->ptr + a.zero_vec16 * 16;
        a.zero_tail_bytes = (int)(bytes % 16);
        size_t want = (a.zero_vec16 + kThreads * 8 - 1) / (kThreads * 8);
        int cap = 2 * sm_count(topk_ids->device_id);
        zero_ctas = (int)(want < 1 ? 1 : (want > (size_t)cap ? (size_t)cap : want));
    }

    const int64_t routes = M * topk;
    a.nchunks = std::max(1, num_chunks(routes));
    a.runs = kWarps * (int)((std::min<int64_t>(routes, kChunk) + kThreads - 1) / kThreads);
    if (a.runs < kWarps) a.runs = kWarps;
    const size_t smem = sort_smem(E, a.runs, lists != nullptr);
    static bool attr_set[64] = {false};
    const int dev = topk_ids->device_id;
    if (dev >= 64 || !attr_set[dev]) {
        const int most = (int)sort_smem(kMaxExperts, kChunk / 32, false), most_lists = (int)sort_smem(kMaxExperts, kChunk / 32, true);
        B200_CUDA(cudaFuncSetAttribute(sort_kernel<false, SortArgs>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        B200_CUDA(cudaFuncSetAttribute(sort_kernel<true, SortArgs>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        B200_CUDA(cudaFuncSetAttribute(sort_kernel<false, SortArgsLists>, cudaFuncAttributeMaxDynamicSharedMemorySize, most_lists));
        B200_CUDA(cudaFuncSetAttribute(sort_kernel<true, SortArgsLists>, cudaFuncAttributeMaxDynamicSharedMemorySize, most_lists));
        if (dev < 64) attr_set[dev] = true;
    }
    if (routes <= kSingleMaxRoutes) {
        if (lists) launch_pdl(sort_kernel<false, SortArgsLists>, a.nchunks + zero_ctas, kThreads, smem, stream, a);
        else launch_pdl(sort_kernel<false, SortArgs>, a.nchunks + zero_ctas, kThreads, smem, stream, a);
    } else {
        const int64_t need = sorting_workspace_bytes((int)M, E, (int)topk);
        B200_CHECK(workspace != nullptr && workspace->ptr != nullptr,
                   "workspace of ", need, " bytes is required for this problem size");
        check_tensor(workspace, "workspace", -1, -1);
        B200_CHECK(((uintptr_t)workspace->ptr & 3) == 0, "workspace must be 4-byte aligned");
        size_t ws_esz = (workspace->dtype_ == AITER_DTYPE_u8 || workspace->dtype_ == AITER_DTYPE_i8) ? 1 : 4;
        B200_CHECK((int64_t)(workspace->numel_ * ws_esz) >= need, "workspace needs ", need, " bytes");
        a.ws_cnt = (int*)workspace->ptr;
        launch_pdl(sort_count_kernel, a.nchunks, kThreads, (size_t)E * sizeof(int), stream, a);
        if (lists) launch_pdl(sort_kernel<true, SortArgsLists>, a.nchunks + zero_ctas, kThreads, smem, stream, a);
        else launch_pdl(sort_kernel<true, SortArgs>, a.nchunks + zero_ctas, kThreads, smem, stream, a);
    }
}

// ------------------------------------------------------------------------------------------------
// Sorting without any allocation by anybody.
//
// Some callers have no way to hand over a workspace: a host runtime that reaches this library over
// an FFI and owns no device allocator of its own, a serving loop whose memory pool is frozen after
// start-up, or code that must not trigger the implicit device synchronisation of cudaMalloc/cudaFree
// in the middle of its steady state.  For them the multi-CTA sort keeps its per-chunk counters in a
// fixed array that is part of the loaded module.  Every GPU that loads the library holds these
// kStaticScratchInts * 4 bytes until the process exits.
//
// The name g_sort_scratch is only a host-side handle: the kernels get the real device address from
// cudaGetSymbolAddress, looked up once per device with that device current.
constexpr int kStaticMaxChunks = 64;                       // 64 chunks x 4096 routes = 262144 routes
constexpr int kStaticScratchInts = kStaticMaxChunks * kMaxExperts + kMaxExperts;   // 260 KiB
static __device__ __align__(256) int g_sort_scratch[kStaticScratchInts];

int64_t static_scratch_bytes() { return (int64_t)kStaticScratchInts * (int64_t)sizeof(int); }

// Device address of the scratch array on `dev` (which must be the current device).
static int* static_scratch_ptr(int dev) {
    static int* cached[64] = {nullptr};
    if (dev >= 0 && dev < 64 && cached[dev]) return cached[dev];
    void* ptr = nullptr;
    B200_CUDA(cudaGetSymbolAddress(&ptr, g_sort_scratch));
    B200_CHECK(ptr != nullptr, "cudaGetSymbolAddress returned a null scratch address");
    if (dev >= 0 && dev < 64) cached[dev] = (int*)ptr;
    return (int*)ptr;
}

void launch_moe_sorting_noalloc(const aiter_tensor_t* topk_ids, const aiter_tensor_t* topk_weights,
                                aiter_tensor_t* sorted_ids, aiter_tensor_t* sorted_w,
                                aiter_tensor_t* sorted_eids, aiter_tensor_t* num_valid,
                                aiter_tensor_t* moe_buf, int E, int unit, const aiter_tensor_t* mask,
                                const aiter_tensor_t* num_local, aiter_tensor_t* local_topk_ids,
                                cudaStream_t stream) {
    check_tensor(topk_ids, "topk_ids", AITER_DTYPE_i32, 2);
    const int64_t M = topk_ids->shape[0], topk = topk_ids->shape[1];
    B200_CHECK(E >= 1 && E <= kMaxExperts, "num_experts must be in [1, ", kMaxExperts, "], got ", E);
    const int64_t need = sorting_workspace_bytes((int)M, E, (int)topk);
    // stated limit: 262144 routes (tokens*topk); with that and E <= 1024 the scratch always suffices
    B200_CHECK(M * topk <= (int64_t)kStaticMaxChunks * kChunk && need <= static_scratch_bytes(),
               "problem too large for the built-in scratch: ", M * topk, " routes (tokens*topk), the limit is ",
               (int64_t)kStaticMaxChunks * kChunk, " with up to ", kMaxExperts, " experts (", static_scratch_bytes(),
               " bytes held by the library); use b200_moe_sorting_fwd with a caller-provided workspace instead");
    // Nothing in the scratch has to start at zero: the count kernel writes every counter before the
    // scatter kernel reads it.
    aiter_tensor_t ws{};
    ws.ptr = static_scratch_ptr(topk_ids->device_id);
    ws.numel_ = (size_t)static_scratch_bytes();
    ws.ndim = 1;
    ws.shape[0] = (int64_t)ws.numel_;
    ws.strides[0] = 1;
    ws.dtype_ = AITER_DTYPE_u8;
    ws.device_id = topk_ids->device_id;
    launch_moe_sorting(topk_ids, topk_weights, sorted_ids, sorted_w, sorted_eids, num_valid, moe_buf, E, unit,
                       mask, num_local, need > 0 ? &ws : nullptr, local_topk_ids, nullptr, stream);
}

}  // namespace b200
