// GEMM stages of the fused-MoE layer for batches with many rows per expert: the activation rows lie in sorted order, so both
// operands arrive by TMA, and two CTAs work on one tile (tcgen05 cta_group::2).
//
//   stage 1 (row scales only):  [gate|up] = A1 . W1_e^T, act(gate)*up -> bf16; gather_rows below puts the rows in order
//   stage 2:                    [rows x 256] = A2 . W2_e^T, times the route weight, added into fp32 acc[token]
//
// Same arithmetic, element by element, as moe_gemm.cu, which gathers its rows itself and serves small batches, stage 1 with block
// scales and the separate entry points.
//
// What bounds the stages of a large batch, and what this does about it:
//  * The shared-memory port. A tile of 128 x 256 moves 48 KB per K step of 128 into shared memory and the UMMAs read 48 KB
//    back: 768 clocks at 128 B/clock, where the tensor pipe needs 512. In a pair each CTA loads and reads half of the weight box
//    (32 + 32 KB, 512 clocks). Pairs are two neighbouring row blocks of one expert (BlockLists); an expert's odd block is worked
//    by a single CTA (PAIR = false), in a launch of its own that fills the SMs as the pairs run out.
//  * The gather of stage 1 by cp.async: 963 clocks a step in a pair with it, 738 with rows in order and TMA (per_Token; the copy
//    that puts them in order is 21 us of 1540 for 8192 rows of 4096).
//  * The reductions of stage 2: see the reducer. K step of the 16384-token Qwen3-shaped layer 1745 clocks in moe_gemm.cu,
//    1230 here.
// Measured, layers in turn with the same layers worked one block a CTA, on three boxes, in us: Mixtral-shaped, 4096 tokens, 2056..2108 ->
// 1804..1825; Qwen3-shaped, 16384 tokens, 4132..4169 -> 3928..3955; DeepSeek-V3-shaped, 8192 tokens, 5328..5426 -> 5218..5278 (the clock
// falls as the work gets denser: these run at the power limit). Stage 2 of the last two, in one call: 1.48 -> 1.24 and 1.93 -> 1.65 ms.
// Stage 1 with block scales was built here as well and gained nothing (Qwen3-shaped: 2.29 ms one block a CTA, 2.19 and 2.30 in two
// builds of pairs, and 0.15 for putting the rows in order): its promotion is the serial chain, whose every access to shared memory,
// barriers included, takes 100 to 300 clocks while the UMMAs read their operands. Which layers gain and which lose: works_in_pairs
// (layer.cu). ptxas spills 40 to 100 bytes of the 96 registers the CTA is launched with; 3.2 % of the instructions of stage 2's pairs
// are reloads of them, whose cost was not measured by itself.

#include <algorithm>

#include "moe_gemm_device.cuh"

namespace b200 {
namespace {

constexpr int BM = 128;            // rows of a CTA's tile (== sort unit); a pair works on 256
constexpr int BK = 128;            // K elements (bytes) per pipeline step == scale block
constexpr int BN = 256;            // UMMA N: 128 gate + 128 up columns, or 256 output columns
constexpr int kABytes = BM * BK;   // 16 KB
constexpr int kPromoWarp0 = 4, kPromoWarps = 16;
constexpr int kThreads = 32 * (kPromoWarp0 + kPromoWarps);
constexpr int kTmemCols = 512;     // 2 stages x 256 fp32 columns
// Registers per thread of each role after setmaxnreg; see moe_gemm.cu for why the sum is checked.
constexpr int kRegsLaunch = 65536 / kThreads / 8 * 8, kRegsLoad = 32, kRegsPromo = 112;
constexpr int kRegDemand = 32 * (kPromoWarp0 * kRegsLoad + kPromoWarps * kRegsPromo);
static_assert(kRegDemand <= kThreads * kRegsLaunch, "setmaxnreg: the roles ask for more registers than the CTA is launched with");
constexpr int kPromoSleepNs = 20;   // back-off of the promotion warps while the UMMAs run

// Stage 2 of a pair: a warp of its own (the reducer) hands the staged rows to the copy engine. A row is staged whole (block
// scales) or in two rounds of 128 columns (PT, whose tiles are long enough to hide them and whose fill needs the stages).
template <int STAGE, bool PT, bool PAIR>
struct Smem {
    static constexpr bool kReducer = STAGE == 2 && PAIR;
    static constexpr int kRounds = PT ? 2 : 1;                  // kReducer: rounds of a tile
    static constexpr int kStages = STAGE == 1 ? (PAIR ? 6 : 4) : PAIR && PT ? 5 : 3;
    static constexpr int kB = (PAIR ? BN / 2 : BN) * BK;        // weight bytes of a stage in this CTA
    static constexpr int kPiece = 32;                           // stage 2 without reducer: columns a thread stages at a time
    static constexpr int kRowPitch = (kReducer ? BN / kRounds : 4 * kPiece) * 4 + 16;   // bytes of a staged row (+ 16: lanes in different banks)
    static constexpr int kOffA = 0;
    static constexpr int kOffB = kOffA + kStages * kABytes;
    static constexpr int kOffOut = kOffB + kStages * kB;        // stage 2: staged rows
    static constexpr int kOffBar = kOffOut + (STAGE == 1 ? 0 : BM * kRowPitch);
    // barriers: full, empty [kStages], TMEM full, empty [2], staged rows [4], free rows [kRounds][4]
    static constexpr int kBarStaged = 2 * kStages + 4;
    static constexpr int kNumBars = kBarStaged + (kReducer ? 4 + 4 * kRounds : 0);
    static constexpr int kOffTmemSlot = kOffBar + kNumBars * 8;
    static constexpr int kOffAbort = kOffTmemSlot + 4;
    static constexpr int kBytes = kOffAbort + 4;
    static_assert(kBytes <= 232448, "shared memory of a CTA");
};

struct SortedGemmParams {
    const float* a_scale;    // [ceil(K/512)][a_scale_ld][4]: four K steps of a sorted row together; PT: [rows], or [1] (a_scale_ld 0)
    const float* w_scale;    // [E, n_rows/128, K/128]; PT: [E, n_rows], or [E] (w_scale_by_expert)
    int a_scale_ld;
    int w_scale_by_expert;
    const int* sorted_ids;
    const float* sorted_w;
    const int* sorted_eids;
    const int* num_valid;    // {padded total, tokens}
    const int* blocks;       // row blocks this launch covers (PAIR: the first of each pair)
    const int* num_blocks;   // how many (device)
    int M;                   // static token count
    int KB;                  // K/128
    int n_tiles;             // stage 1 I/128; stage 2 ceil(H/256)
    int n_rows;              // weight rows per expert: 2I (stage 1) or H (stage 2)
    int inter;               // I
    __nv_bfloat16* half;     // stage 1 out [P, I]
    float* acc;              // stage 2 out [M, H] fp32
    int* status;
    unsigned* amax;          // stage 1: maximum magnitude written, as fp32 bits, or null
    int beside;              // may run beside the kernel before it on the stream (which covers other blocks of the same stage)
    int use_weight;          // multiply this stage's GEMM result by the route weight
    long long wait_limit;
    int stall_producer;
};

template <int STAGE, bool PT, int ACT, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
sorted_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a, const SortedGemmParams p) {
    static_assert(STAGE == 2 || PT, "stage 1 with block scales is moe_gemm.cu's");
    using S = Smem<STAGE, PT, PAIR>;
    constexpr int kStages = S::kStages, kB = S::kB;
    constexpr int kPromoArrivals = (PAIR ? 2 : 1) * kPromoWarps;   // promotion warps that read a TMEM stage
    constexpr uint32_t kIdesc = ptx::make_idesc_e4m3_f32(PAIR ? 2 * BM : BM, BN);
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = ptx::smem_u32(smem);
    if (sbase & 1023u) {   // the swizzle of the operand tiles counts on it (the launch gives no static shared memory)
        if (threadIdx.x == 0) atomicExch(p.status, 1);
        return;
    }
    const uint32_t sA = sbase + S::kOffA, sB = sbase + S::kOffB;
    const uint32_t bar0 = sbase + S::kOffBar;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (kStages + s); };
    auto tfull_bar = [&](int s) { return bar0 + 8u * (2 * kStages + s); };
    auto tempty_bar = [&](int s) { return bar0 + 8u * (2 * kStages + 2 + s); };   // PT only, see the issuer
    auto staged_bar = [&](int q) { return bar0 + 8u * (S::kBarStaged + q); };
    auto free_bar = [&](int q) { return bar0 + 8u * (S::kBarStaged + 4 + q); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + S::kOffTmemSlot);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + S::kOffAbort);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int rank = PAIR ? (int)ptx::cluster_rank() : 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            // the two loading threads (PAIR: of the first CTA, for both), and the promotion warps (see the issuer)
            ptx::mbar_init(full_bar(s), 2 + (PT ? 0 : kPromoArrivals));
            ptx::mbar_init(empty_bar(s), 1);   // one tcgen05.commit
        }
        for (int s = 0; s < 2; ++s) {
            ptx::mbar_init(tfull_bar(s), 1);                              // one tcgen05.commit
            ptx::mbar_init(tempty_bar(s), kPromoArrivals);                // one arrive per promotion warp
        }
        if (S::kReducer)
            for (int q = 0; q < 4; ++q) {
                ptx::mbar_init(staged_bar(q), 4 / S::kRounds);   // the warps that write a round of 32 rows
                for (int g = 0; g < S::kRounds; ++g) ptx::mbar_init(free_bar(4 * g + q), 1);   // a barrier per round: its
            }                                                                                // warps wait once a tile
        *abort_flag = 0;
        ptx::fence_mbar_init();
        ptx::prefetch_tensormap(&tmap_w);
        ptx::prefetch_tensormap(&tmap_a);
    }
    if (warp == 2) {
        ptx::tmem_alloc<PAIR>(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemCols);
        ptx::tmem_relinquish<PAIR>();
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (PAIR) ptx::cluster_sync();   // the other CTA's barriers are initialised before anything arrives on them
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (!p.beside) pdl_wait();       // everything above overlaps the kernels before this one
    pdl_trigger();

    const int tokens = min(p.num_valid[1], p.M);
    const int total_tiles = *p.num_blocks * p.n_tiles;
    const int t_first = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, t_step = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    auto block_of = [&](int t) { return p.blocks[t / p.n_tiles] + rank; };   // row block of tile t

    if (warp < kPromoWarp0) {
        ptx::setmaxnreg_dec<kRegsLoad>();
        int s = 0;
        uint32_t ph = 0;   // phase of the stage's barriers
        bool ok = true;
        auto next_stage = [&]() {
            if (++s == kStages) s = 0, ph ^= 1u;
        };
        if (warp == 0 && lane == 0) {
            // ---------------------------------------------------------------- weight TMA producer
            const uint32_t lead = PAIR ? ptx::map_to_rank(bar0, 0) : bar0;   // the pair reports to its first CTA's barriers
            ok = !p.stall_producer;   // self-test: issue nothing; the other roles' waits then run out
            for (int t = t_first; ok && t < total_tiles; t += t_step) {
                const int nt = t % p.n_tiles, e = p.sorted_eids[block_of(t)];
                int r0, r1;
                if (STAGE == 1) {
                    r0 = e * p.n_rows + nt * 128;   // gate rows
                    r1 = r0 + p.inter;              // up rows
                } else {
                    r0 = e * p.n_rows + nt * 256;
                    r1 = (nt * 256 + 128 < p.n_rows) ? r0 + 128 : r0;
                }
                if (PAIR && rank == 1) r0 = r1;     // each CTA loads one of the tile's two weight boxes
                for (int kb = 0; kb < p.KB; ++kb) {
                    if (!(ok = ptx::mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, p.wait_limit))) break;
                    if (rank == 0) ptx::mbar_arrive_expect_tx(full_bar(s), BN * BK);
                    if (PAIR) {
                        ptx::tma_load_2d_pair(sB + s * kB, &tmap_w, kb * BK, r0, lead + 8u * s);
                    } else {
                        ptx::tma_load_2d(sB + s * kB, &tmap_w, kb * BK, r0, full_bar(s));
                        ptx::tma_load_2d(sB + s * kB + kB / 2, &tmap_w, kb * BK, r1, full_bar(s));
                    }
                    next_stage();
                }
            }
            if (PAIR)   // the commits that free the last stages have arrived before this CTA may leave
                for (int i = 0; ok && i < kStages; ++i) {
                    ok = ptx::mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, p.wait_limit);
                    next_stage();
                }
        } else if (warp == 1 && lane == 0 && rank == 0) {
            // ---------------------------------------------------------------- UMMA issuer
            // Block scales (PT = false): every K block's partial sums go to the TMEM stage of that step's parity
            // and are promoted in registers. Row/channel scales (PT = true) do not depend on K: the whole K loop
            // accumulates in one TMEM stage, stages alternate per TILE, and the epilogue of a tile overlaps the
            // MMAs of the next.
            // With block scales a step's TMEM stage is free when the promotion of the step two before is over; its warps then
            // arrive on the full barrier of this step's operands, so that one wait covers both (a second wait behind a burst of
            // MMAs costs ~150 clocks of the step).
            uint32_t tcount = 0;   // what the TMEM stage ring counts
            for (int t = t_first; ok && t < total_tiles; t += t_step) {
                for (int kb = 0; kb < p.KB; ++kb) {
                    const int ts = tcount & 1;
                    if (PT && kb == 0)
                        if (!(ok = ptx::mbar_wait(tempty_bar(ts), ((tcount >> 1) & 1u) ^ 1u, abort_flag, p.wait_limit))) break;
                    if (!(ok = ptx::mbar_wait(full_bar(s), ph, abort_flag, p.wait_limit))) break;
                    ptx::tc_fence_after();
                    const uint64_t da = ptx::make_kmajor_sw128_desc(sA + s * kABytes);
                    const uint64_t db = ptx::make_kmajor_sw128_desc(sB + s * kB);
                    const uint32_t d = tmem_base + ts * BN;
#pragma unroll
                    for (int k = 0; k < BK / 32; ++k)   // 32 bytes of K per UMMA: +2 in 16-byte units
                        ptx::umma_f8<PAIR>(d, da + 2u * k, db + 2u * k, kIdesc, (k > 0 || (PT && kb > 0)) ? 1u : 0u);
                    ptx::umma_commit<PAIR>(empty_bar(s));
                    if (!PT || kb == p.KB - 1) {
                        ptx::umma_commit<PAIR>(tfull_bar(ts));
                        ++tcount;
                    }
                    next_stage();
                }
            }
        } else if (warp == 2) {
            // ---------------------------------------------------------------- activation TMA producer
            if (PAIR) {
                // whole blocks (what lies in the padding rows of a pair's second block is multiplied too, but belongs to TMEM
                // lanes that nobody reads)
                const uint32_t lead = ptx::map_to_rank(bar0, 0);
                if (lane == 0)
                    for (int t = t_first; ok && t < total_tiles; t += t_step) {
                        const int row0 = block_of(t) * BM;
                        for (int kb = 0; kb < p.KB; ++kb) {
                            if (!(ok = ptx::mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, p.wait_limit))) break;
                            if (rank == 0) ptx::mbar_arrive_expect_tx(full_bar(s), 2 * kABytes);
                            ptx::tma_load_2d_pair(sA + s * kABytes, &tmap_a, kb * BK, row0, lead + 8u * s);
                            next_stage();
                        }
                    }
            } else {
                // 32 rows a box; the boxes that hold padding only are left out
                int ids[4] = {0, 0, 0, 0};   // sorted ids of the next tile's rows (one per quarter and lane)
                auto fetch = [&](int t) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) ids[q] = p.sorted_ids[block_of(t) * BM + q * 32 + lane];
                };
                if (t_first < total_tiles) fetch(t_first);
                for (int t = t_first; ok && t < total_tiles; t += t_step) {
                    const int row0 = block_of(t) * BM;
                    uint32_t live = 0;
#pragma unroll
                    for (int q = 0; q < 4; ++q) live |= (__any_sync(0xffffffffu, (ids[q] & 0xFFFFFF) < tokens) ? 1u : 0u) << q;
                    if (t + t_step < total_tiles) fetch(t + t_step);
                    if (lane == 0) {
                        for (int kb = 0; kb < p.KB; ++kb) {
                            if (!(ok = ptx::mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, p.wait_limit))) break;
                            ptx::mbar_arrive_expect_tx(full_bar(s), __popc(live) * (kABytes / 4));
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                if ((live >> q) & 1u)
                                    ptx::tma_load_2d(sA + s * kABytes + q * (kABytes / 4), &tmap_a, kb * BK, row0 + q * 32, full_bar(s));
                            next_stage();
                        }
                    }
                    ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
                }
            }
        }
        else if (S::kReducer && warp == 3) {
            // ---------------------------------------------------------------- reducer: staged rows -> acc
            // out[token] += row (aiter/fused_moe.py:3802-3811) as fp32 reductions in L2, one asynchronous bulk reduce-add per row.
            // An SM's port takes ~20 B/clock of them, 6.5k clocks a tile, during which an issuing thread is held up: with a warp
            // of its own to wait, the promotion of the next tile goes on.
            uint32_t uses = 0;   // bit q: parity of the quarter's next use
            int id[4] = {0, 0, 0, 0};
            auto fetch = [&](int t) {
#pragma unroll
                for (int q = 0; q < 4; ++q) id[q] = p.sorted_ids[block_of(t) * BM + q * 32 + lane] & 0xFFFFFF;
            };
            if (t_first < total_tiles) fetch(t_first);
            for (int t = t_first; ok && t < total_tiles; t += t_step) {
                const int nt = t % p.n_tiles;
                int tok[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) tok[q] = id[q];
                if (t + t_step < total_tiles) fetch(t + t_step);
#pragma unroll
                for (int g = 0; g < S::kRounds; ++g) {
                    const int c0 = nt * BN + g * (BN / S::kRounds);
                    const int bytes = min(BN / S::kRounds, p.n_rows - c0) * 4;
                    uint32_t live = 0;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const bool valid = tok[q] < tokens;
                        if (!ok || !__any_sync(0xffffffffu, valid)) continue;
                        live |= 1u << q;
                        ok = ptx::mbar_wait<100>(staged_bar(q), (uses >> q) & 1u, abort_flag, p.wait_limit);
                        if (ok && valid && bytes > 0) {
                            float* to = p.acc + (size_t)tok[q] * p.n_rows + c0;
                            const uint32_t from = sbase + S::kOffOut + (uint32_t)(q * 32 + lane) * S::kRowPitch;
                            ptx::bulk_reduce_add_f32(to, from, bytes);
                        }
                        ptx::bulk_commit();
                        ok = __all_sync(0xffffffffu, ok) != 0;
                    }
                    if (!ok) break;
                    ptx::bulk_wait_read_all();
                    __syncwarp();
                    if (lane < 4 && ((live >> lane) & 1u)) ptx::mbar_arrive(free_bar((g + 1) % S::kRounds * 4 + lane));
                    uses ^= live;
                }
            }
            ptx::bulk_wait_all();   // nothing of this warp is in flight when the CTA winds down
        }
    } else {
        // -------------------------------------------------------------------- promotion + epilogue
        ptx::setmaxnreg_inc<kRegsPromo>();
        const int q = warp & 3;                         // TMEM lane quarter this warp may read
        const int part = (warp - kPromoWarp0) >> 2;     // stage 1: 32 of the 128 channels; stage 2: 64 of the 256 columns
        const int r = q * 32 + lane;                    // row of the tile == TMEM lane
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + part * (STAGE == 1 ? 32 : 64);
        const uint32_t lead = PAIR ? ptx::map_to_rank(bar0, 0) : bar0;
        const int groups = p.n_rows / 128;
        uint32_t it = 0;
        uint32_t par = 0;      // parity of the staged rows' next use
        int s_free = 2 % kStages;   // operand stage of the step after the next
        bool ok = true;
        // Row info and the first two K steps' scales of the next tile are fetched ahead, so their latency is off the path
        // between two tiles (where the MMA warp can only run two K steps ahead of these warps)
        int prow_next = 0, tok_next = 0, eid = 0;
        float wgt_next = 0.f;
        // PT = false: the scales of the next four K steps, of this thread's row and of its columns
        float4 a_next = make_float4(0.f, 0.f, 0.f, 0.f), w_next = a_next;
        float a_row = 0.f;                                  // PT: the row's scale
        auto row_info = [&](int t) {
            const int blk = block_of(t);
            prow_next = blk * BM + r;
            tok_next = p.sorted_ids[prow_next] & 0xFFFFFF;
            eid = p.sorted_eids[blk];
            if (p.use_weight) wgt_next = p.sorted_w[prow_next];
        };
        const bool quads = p.KB % 4 == 0 && ((uintptr_t)p.w_scale & 15) == 0;   // rows of weight scales keep 16-byte alignment
        auto quad = [&](const float* at, int left) {
            if (quads) return __ldg(reinterpret_cast<const float4*>(at));
            return make_float4(__ldg(at), left > 1 ? __ldg(at + 1) : 0.f, left > 2 ? __ldg(at + 2) : 0.f, left > 3 ? __ldg(at + 3) : 0.f);
        };
        auto load_scales = [&](int kb, int at_row, int expert, int nt) {   // of K steps kb .. kb + 3
            a_next = __ldg(reinterpret_cast<const float4*>(p.a_scale) + (size_t)(kb >> 2) * p.a_scale_ld + at_row);
            w_next = quad(p.w_scale + (size_t)(expert * groups + min(nt * 2 + (part >> 1), groups - 1)) * p.KB + kb, p.KB - kb);
        };
        auto first_scales = [&](int t) {
            if (PT) {
                a_row = __ldg(p.a_scale + (size_t)prow_next * p.a_scale_ld);
                if (p.w_scale_by_expert) a_row *= __ldg(p.w_scale + eid);   // per_Tensor: the expert's scale rides on the row scale
            } else {
                load_scales(0, prow_next, eid, t % p.n_tiles);
            }
        };
        auto release = [&](int at) {   // lane 0: this warp has read the TMEM stage that the step with barrier `at` waits for
            if (PAIR) ptx::mbar_arrive_cluster(lead + 8u * at);
            else ptx::mbar_arrive(bar0 + 8u * at);
        };
        if (!PT && lane == 0) {        // both TMEM stages are free at the start
            release(0);
            release(1);
        }
        if (t_first < total_tiles) {
            row_info(t_first);
            first_scales(t_first);
        }
        for (int t = t_first; ok && t < total_tiles; t += t_step) {
            const int nt = t % p.n_tiles;
            const int row = prow_next, tok = tok_next, e = eid;
            const bool valid = tok < tokens;
            // the route weight (stage 2, or stage 1 with doweight_stage1) rides on the per-step scales
            const float wgt = p.use_weight ? (valid ? wgt_next : 0.f) : 1.f;
            const bool more = t + t_step < total_tiles;
            if (PT && more) row_info(t + t_step);
            // a warp whose 32 rows are all padding leaves its accumulators at 0
            const bool warp_live = __any_sync(0xffffffffu, valid);

            // stage 1: acc[j] holds channels (2j, 2j+1) of this thread's 32, gate for j < 16, up from 16 on; stage 2: columns
            float2 acc[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[j] = make_float2(0.f, 0.f);

            // Four K steps a round, their scales (products of the row's and the columns') loaded a round ahead. Loads, shuffles and
            // shared memory alike take 100 to 300 clocks while the UMMAs read their operands: one a step, however early it is
            // issued, costs 10 to 20 % of it.
            float4 sq = make_float4(a_row * wgt, 0.f, 0.f, 0.f);   // PT: the first word; wgt is exactly 1 when the stage does not weight
            for (int kb = PT ? p.KB - 1 : 0; kb < p.KB; ++kb, ++it) {   // PT: one pass over the finished accumulators per tile
                if (!PT && (kb & 3) == 0) {
                    sq = make_float4(a_next.x * wgt * w_next.x, a_next.y * wgt * w_next.y, a_next.z * wgt * w_next.z, a_next.w * wgt * w_next.w);
                    if (kb + 4 < p.KB) load_scales(kb + 4, row, e, nt);
                    else if (more) row_info(t + t_step);
                }
                const int ts = it & 1;
                if (!(ok = ptx::mbar_wait<kPromoSleepNs>(tfull_bar(ts), (it >> 1) & 1u, abort_flag, p.wait_limit))) break;
                ptx::tc_fence_after();
                const float f = PT ? sq.x : (kb & 2) ? ((kb & 1) ? sq.w : sq.z) : ((kb & 1) ? sq.y : sq.x);
                const float2 f2 = make_float2(f, f);
                const uint32_t ta = lane_addr + ts * BN;
                uint32_t v[16];
                if (warp_live) {
                    ptx::tmem_ld_x16_sync(ta, v);
                    fold16(acc, v, f2);
                    ptx::tmem_ld_x16_sync(ta + 16, v);
                    fold16(acc + 8, v, f2);
                    ptx::tmem_ld_x16_sync(ta + (STAGE == 1 ? 128 : 32), v);
                    fold16(acc + 16, v, f2);
                    ptx::tmem_ld_x16_sync(ta + (STAGE == 1 ? 128 : 32) + 16, v);
                }
                // all reads of this TMEM stage are done: hand it back to the MMA warp
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) release(PT ? 2 * kStages + 2 + ts : s_free);
                if (!PT && ++s_free == kStages) s_free = 0;
                if (warp_live) fold16(acc + 24, v, f2);
            }
            if (!ok) break;
            if (more) first_scales(t + t_step);

            if (!warp_live) continue;   // rows of padding are not written (nothing reads them)
            if (PT && !p.w_scale_by_expert) {
                // weight scales per output channel (all lanes read the same addresses)
                const int c0 = STAGE == 1 ? nt * 128 + part * 32 : min(nt * 256 + part * 64, p.n_rows - 64);
                const float4* c_w0 = reinterpret_cast<const float4*>(p.w_scale + (size_t)e * p.n_rows + c0);
                const float4* c_w1 = STAGE == 1 ? reinterpret_cast<const float4*>(p.w_scale + (size_t)e * p.n_rows + c0 + p.inter) : c_w0 + 8;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 a = __ldg(c_w0 + j), b = __ldg(c_w1 + j);
                    acc[2 * j] = make_float2(acc[2 * j].x * a.x, acc[2 * j].y * a.y);
                    acc[2 * j + 1] = make_float2(acc[2 * j + 1].x * a.z, acc[2 * j + 1].y * a.w);
                    acc[16 + 2 * j] = make_float2(acc[16 + 2 * j].x * b.x, acc[16 + 2 * j].y * b.y);
                    acc[16 + 2 * j + 1] = make_float2(acc[16 + 2 * j + 1].x * b.z, acc[16 + 2 * j + 1].y * b.w);
                }
            }

            if (STAGE == 1) {
                // act(gate) * up in fp32 -> bf16 (RNE), as the oracle does: aiter/fused_moe.py:3668-3681; the row-wise requantisation
                // needs the whole row and is a kernel of its own
                uint32_t hb[16];
                __nv_bfloat162 m2 = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
                for (int j0 = 0; j0 < 16; j0 += 2) {   // four values at a time: with eight the 112 registers do not suffice
                    const float g[4] = {acc[j0].x, acc[j0].y, acc[j0 + 1].x, acc[j0 + 1].y};
                    const float u[4] = {acc[16 + j0].x, acc[16 + j0].y, acc[17 + j0].x, acc[17 + j0].y};
                    float h[4];
                    act_mul_n<ACT, 4>(g, u, h);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const __nv_bfloat162 b2 = __floats2bfloat162_rn(h[2 * i], h[2 * i + 1]);
                        hb[j0 + i] = *reinterpret_cast<const uint32_t*>(&b2);
                        m2 = __hmax2(m2, __habs2(b2));   // skips NaN, as fmaxf does
                    }
                }
                if (p.amax) {
                    // per_Tensor requantisation: the maximum is taken here, where the values are in registers
                    const float amax = valid ? fmaxf(__low2float(m2), __high2float(m2)) : 0.f;
                    const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
                    if (lane == 0 && top != 0u) atomicMax(p.amax, top);
                }
                uint4* dst = reinterpret_cast<uint4*>(p.half + (size_t)row * p.inter + nt * 128 + part * 32);
                if (valid) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) dst[j] = make_uint4(hb[4 * j], hb[4 * j + 1], hb[4 * j + 2], hb[4 * j + 3]);
                }
            } else if (S::kReducer) {
                // to the staged row, whose previous contents the copy engine has read; the weight is already in the accumulators
                const int g = part * S::kRounds / 4;   // this warp's round
                if (!(ok = ptx::mbar_wait<kPromoSleepNs>(free_bar(4 * g + q), g == 0 ? par ^ 1u : par, abort_flag, p.wait_limit))) break;
                par ^= 1u;
                const uint32_t srow = sbase + S::kOffOut + (uint32_t)r * S::kRowPitch + (part * 64 - g * (BN / S::kRounds)) * 4;
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    ptx::st_shared_v4(srow + j * 16, acc[2 * j].x, acc[2 * j].y, acc[2 * j + 1].x, acc[2 * j + 1].y);
                ptx::fence_proxy_async();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(staged_bar(q));
            } else if (valid && nt * 256 + part * 64 < p.n_rows) {
                // as the reducer does, by the thread itself, in pieces for which there is room
                const uint32_t srow = sbase + S::kOffOut + (uint32_t)r * S::kRowPitch + part * S::kPiece * 4;
                float* orow = p.acc + (size_t)tok * p.n_rows + nt * 256 + part * 64;
                constexpr int kQuads = S::kPiece / 4;
#pragma unroll
                for (int g = 0; g < 16 / kQuads; ++g) {
                    ptx::bulk_wait_read_all();   // the copy engine has read this row's previous contents
#pragma unroll
                    for (int j = 0; j < kQuads; ++j) {
                        const float2 x = acc[2 * (g * kQuads + j)], y = acc[2 * (g * kQuads + j) + 1];
                        ptx::st_shared_v4(srow + j * 16, x.x, x.y, y.x, y.y);
                    }
                    ptx::fence_proxy_async();
                    ptx::bulk_reduce_add_f32(orow + g * S::kPiece, srow, S::kPiece * 4);
                    ptx::bulk_commit();
                }
            }
        }
        ptx::bulk_wait_all();   // nothing of this thread is in flight when the CTA winds down
    }

    // ------------------------------------------------------------------------ tail
    ptx::tc_fence_before();
    __syncthreads();
    const bool gave_up = *abort_flag != 0;
    if (gave_up && threadIdx.x == 0) atomicExch(p.status, 1);
    if (warp == 2 && gave_up) {
        // give copies / MMAs still in flight a bounded time to land before TMEM is released
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {
        }
    }
    if (p.beside) pdl_wait();        // this launch is not over before the one beside it
    if (PAIR) ptx::cluster_sync();   // nothing of this CTA is still read, written or signalled by the other one
    if (warp == 2) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc<PAIR>(tmem_base, kTmemCols);
    }
}

// a1 rows [M, H] and, if given, their scales into sorted order; rows of padding are not written. A CTA takes 32 sorted rows.
constexpr int kGatherThreads = 256;
__global__ void __launch_bounds__(kGatherThreads) gather_rows_kernel(const uint4* a1, const float* a1_scale, uint4* rows, float* scales,
                                                                    const int* sorted_ids, const int* num_valid, int M, int pieces) {
    pdl_wait();
    pdl_trigger();
    const int row0 = blockIdx.x * 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (row0 >= num_valid[0]) return;
    const int tokens = min(num_valid[1], M);
    const int tok = sorted_ids[row0 + lane] & 0xFFFFFF;
    for (int i = warp; i < 32; i += kGatherThreads / 32) {
        const int src = __shfl_sync(0xffffffffu, tok, i);
        if (src >= tokens) continue;
        const uint4* from = a1 + (size_t)src * pieces;
        uint4* to = rows + (size_t)(row0 + i) * pieces;
        for (int c = lane; c < pieces; c += 128) {
            uint4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (c + 32 * k < pieces) v[k] = from[c + 32 * k];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (c + 32 * k < pieces) to[c + 32 * k] = v[k];
        }
    }
    if (a1_scale && warp == 0 && tok < tokens) scales[row0 + lane] = a1_scale[tok];
}

template <int STAGE, bool PT, int ACT, bool PAIR>
void launch_blocks(const CUtensorMap& tmap_w, const CUtensorMap& tmap_a, SortedGemmParams p, int64_t max_blocks, int dev, cudaStream_t stream) {
    using S = Smem<STAGE, PT, PAIR>;
    auto* kernel = sorted_gemm_kernel<STAGE, PT, ACT, PAIR>;
    static bool attr_set[64] = {false};
    if (dev >= 64 || !attr_set[dev]) {
        B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kBytes));
        cudaFuncAttributes fa;
        B200_CUDA(cudaFuncGetAttributes(&fa, kernel));
        B200_CHECK((int64_t)fa.numRegs * kThreads >= kRegDemand, "GEMM kernel was compiled with ", fa.numRegs,
                   " registers per thread: its roles' setmaxnreg requests (", kRegDemand, " per CTA) could never be met");
        if (dev < 64) attr_set[dev] = true;
    }
    const int64_t max_tiles = max_blocks * p.n_tiles, sms = sm_count(dev);
    const int64_t grid = PAIR ? std::min(sms / 2, max_tiles) * 2 : std::min(sms, max_tiles);
    if (grid < 1) return;
    p.wait_limit = g_wait_limit;
    p.stall_producer = g_stall_producer;
    p.beside = PAIR ? 0 : 1;
    launch_kernel(true, kernel, (unsigned)grid, kThreads, S::kBytes, stream, PAIR ? 2 : 1, tmap_w, tmap_a, p);
}

// the pairs by the pair kernel, and the single blocks beside its last tiles
template <int STAGE, bool PT, int ACT = 0>
void launch_lists(const void* w, int64_t w_rows, const void* a, int64_t a_rows, int64_t K, SortedGemmParams p, const BlockLists& lists,
                  int dev, cudaStream_t stream) {
    // the launch over the single blocks starts without a wait of its own: there has to be one over pairs in front of it
    B200_CHECK(lists.max_pairs >= 1 && p.n_tiles >= 1, "row blocks cannot be worked in pairs");
    const CUtensorMap tmap_w = make_map(w, (uint64_t)w_rows, (uint64_t)K, 128);
    p.blocks = lists.pairs;
    p.num_blocks = lists.counts;
    launch_blocks<STAGE, PT, ACT, true>(tmap_w, make_map(a, (uint64_t)a_rows, (uint64_t)K, 128), p, lists.max_pairs, dev, stream);
    p.blocks = lists.singles;
    p.num_blocks = lists.counts + 1;
    launch_blocks<STAGE, PT, ACT, false>(tmap_w, make_map(a, (uint64_t)a_rows, (uint64_t)K, 32), p, lists.max_singles, dev, stream);
}

}  // namespace

void launch_gather_rows(const void* a1, const float* a1_scale, void* rows, float* scales, const int* sorted_ids, const int* num_valid,
                        int64_t M, int64_t H, int64_t P, cudaStream_t stream) {
    B200_CHECK(H % 16 == 0 && ((uintptr_t)a1 & 15) == 0 && ((uintptr_t)rows & 15) == 0, "rows must be 16-byte aligned");
    launch_pdl(gather_rows_kernel, (unsigned)(P / 32), kGatherThreads, 0, stream, (const uint4*)a1, a1_scale, (uint4*)rows, scales,
               sorted_ids, num_valid, (int)M, (int)(H / 16));
}

static SortedGemmParams common_params(const SortedStage& a) {
    SortedGemmParams p{};
    p.a_scale = a.a_scale;
    p.a_scale_ld = a.a_scale_ld;
    p.w_scale = a.w_scale;
    p.w_scale_by_expert = a.w_scale_by_expert;
    p.sorted_ids = a.sorted_ids;
    p.sorted_w = a.sorted_w;
    p.sorted_eids = a.sorted_eids;
    p.num_valid = a.num_valid;
    p.use_weight = a.use_weight;
    p.M = (int)a.M;
    p.inter = (int)a.I;
    p.status = a.status;
    return p;
}

void launch_sorted_stage1(const SortedStage& a, cudaStream_t stream) {
    SortedGemmParams p = common_params(a);
    p.KB = (int)(a.H / 128);
    p.n_tiles = (int)(a.I / 128);
    p.n_rows = (int)(2 * a.I);
    p.half = (__nv_bfloat16*)a.out;
    p.amax = a.amax;
    auto go = [&](auto launch) { launch(a.w, a.E * 2 * a.I, a.rows, a.P, a.H, p, a.lists, a.device, stream); };
    a.activation == 1 ? go(launch_lists<1, true, 1>) : go(launch_lists<1, true, 0>);
}

void launch_sorted_stage2(const SortedStage& a, cudaStream_t stream) {
    SortedGemmParams p = common_params(a);
    p.KB = (int)(a.I / 128);
    p.n_tiles = (int)((a.H + 255) / 256);
    p.n_rows = (int)a.H;
    p.acc = (float*)a.out;
    auto go = [&](auto launch) { launch(a.w, a.E * a.H, a.rows, a.P, a.I, p, a.lists, a.device, stream); };
    a.rowwise ? go(launch_lists<2, true>) : go(launch_lists<2, false>);
}

}  // namespace b200
