// Grouped GEMM of the expert layer with the WEIGHTS as the tensor cores' M operand and the tokens as N:
//
//   out[t, :] = epilogue( W[e(t)] @ A[t, :]^T )^T      for the rows t of every expert's range.
//
// Why this way round: an expert's row count is whatever the router made it.  With tokens as M a pair of CTAs works on
// 256 rows whether they exist or not (32 experts of 1024 +- 32 rows: 1152 rows of MMA work on average, and 128 for the 16
// rows of a decode step); as N a tile takes any multiple of 32 tokens up to 256, so an expert's rows are split into equal
// tiles that end within 31 rows of the last real one, and a decode step moves little besides its weights.
//
// A cluster of two CTAs computes 256 weight rows x N tokens (tcgen05.mma.cta_group::2): each CTA loads its 128 weight rows
// and half of the token rows by TMA, the leader issues the MMAs, each CTA holds the accumulator of its own 128 weight rows
// in its own TMEM (two buffers, so that the epilogue of a tile runs under the next tile's MMAs).  SwiGLU interleaves 16
// gate rows with their 16 up rows, which puts both factors of an output into the same registers of the same thread.
// The accumulator is transposed on its way out: fragments (16 x 256-bit TMEM loads) go through stmatrix.trans into 32
// staged token rows of shared memory per epilogue group, and whole token rows leave in 128-byte (SwiGLU) or 256-byte pieces
// to the output or, in the scatter mode, straight into the source rank's return partition (peer memory over NVLink, or local).
//
// What bounds it.  Few tokens: the weights' way from memory (32 experts of 7168 x 2048, 16 rows each: up 320 -> 283 us = 6.6
// TB/s, down 185 -> 154 us, tokens as M -> as N).  Many tokens: in a burst the SM's ingress (16 KB of weights and up to 16 KB of
// tokens per 512 cycles of MMA against 64 B a cycle; 54 B measured, tensor pipe 88 % active at N = 256 and 80 % at 224), in a
// long run the card's power limit: 990 W at 1.1 GHz, 32 experts of ~1024 rows up 1706 -> 1620 us, down 880 -> 800 us.  Two weight
// tiles per token tile (a quarter less ingress, one accumulator each) ran at 1.3 GHz and the same power: up 1707, down 823 us.
// In between, 4662 rows over 32 experts of 4096 x 1536: up 209 -> 163 us, down 121 -> 86 us.
//
// Who computes what.  The grid holds a cluster for every unit (one weight tile x one token tile) that the offsets allow (see
// unit_places for where it holds fewer); the clusters that run take over the places of those that have not started (cluster launch control), in order, one or two
// units ahead.  With a fixed share of the units per cluster, clusters that share a weight tile drift apart by more than
// L2 keeps it (small differences add up over units of 100 us) and fetch it again: the up-projection of 32 experts of 1024
// rows read 4.0-5.3 GB from memory instead of the 2.35 GB that there are, now 2.5-2.7 GB, and at the power limit every byte costs
// clock.  us, fixed share -> taken over: 32 x 1024 rows up 1325 -> 1260, 0.8 s in a row 1533 -> 1480, down 660 -> 648, 785 -> 770; 32 x (1024
// +- 32) up 1410 -> 1345, 0.8 s in a row 1650 -> 1566, down 692 -> 686; 4662 uneven rows (4096 x 1536) up 165 -> 158, down 91 -> 85.  The readers of a unit
// acknowledge it without a fence: a releasing arrival waits for the thread's bulk loads in flight and drained the
// operand pipeline at every unit (tensor pipe 98 -> 93 % active up, 96 -> 80 % down).  Which unit comes when is hand_out_units
// (unit_queue.hpp): every unit taken over is computed, whatever the order of the answers.  A launch with a cap on its CTAs keeps fixed shares.
//
// All waits are bounded; on expiry a CTA records a code in `status`, stops issuing work, and both CTAs still meet at the
// final cluster barrier and free their TMEM.
#include "grouped_gemm_sm100.hpp"
#include "unit_queue.hpp"

#include <cuda_bf16.h>

#include <atomic>

#include "tc_prim.cuh"

namespace nep {
namespace gemm {
namespace {

using namespace tc;

constexpr int BW = 256, BK = 64;             // weight rows of a pair tile, K per stage
constexpr int kWBytes = BW / 2 * BK * 2;     // 16 KB: this CTA's weight rows
constexpr int kGroups = 2;                   // epilogue groups of four warps
constexpr int kEpiThreads = kGroups * 128;
constexpr int kThreads = 64 + kEpiThreads;
constexpr int kTmemCols = 512, kAccCols = 256;
constexpr int kMaxExperts = 1024;
constexpr int kMaxStages = 10;
constexpr int kChunk = 32;                   // token rows staged at a time by a group
constexpr int kMaxTokens = 256;              // largest N
constexpr int kUnitReaders = 5;              // readers of a handed-out unit: two producers, the MMA issuer, two epilogues

template <int kMode>
struct Out {
    static constexpr int kFeatures = kMode == kSwiGLU ? 64 : 128;  // output columns of one CTA's tile
    static constexpr int kRowBytes = kFeatures * 2;
    static constexpr int kPitch = kRowBytes + 16;  // 8 staged rows hit all banks once
    static constexpr int kBufBytes = kChunk * kPitch;
};

struct Shared {
    alignas(16) uint32_t cancelled[4];  // answer to a request for the next cluster's place (CTA 1)
    uint64_t full[kMaxStages], empty[kMaxStages], tmem_full[2], tmem_empty[2];
    uint64_t cancel_done, unit_full[kUnitSlots], unit_empty[kUnitSlots];
    uint32_t tmem_base;
    int abort;
    int go[2];
    int next_unit[kUnitSlots];  // handed out by the scheduler, -1: none
    int epi_unit[2];   // the epilogue's unit, by parity of the item
    int offsets[kMaxExperts + 1];       // first row
    int rows[kMaxExperts];              // rows to compute
    int first_tile[kMaxExperts + 1];    // exclusive prefix of token tiles
    float scale[kMaxTokens];            // epilogue: per token of the current tile
    void* dst[kMaxTokens];              // scatter: destination row or null
};

// Shape of a launch's pipeline: small token tiles leave room for more stages.
constexpr int kSmemLimit = 232448;
template <int kMode, int kTileTokens>
struct Pipe {
    static constexpr int kStageBytes = kWBytes + kTileTokens / 2 * BK * 2;
    static constexpr int kFixedBytes = kGroups * Out<kMode>::kBufBytes + int(sizeof(Shared));
    static constexpr int kFit = (kSmemLimit - kFixedBytes) / kStageBytes;
    static constexpr int kStages = kFit < kMaxStages ? kFit : kMaxStages;
    static constexpr size_t kSmemBytes = size_t(kStages) * kStageBytes + kFixedBytes;
    static_assert(kStages >= 6 && kStageBytes % 1024 == 0 && Out<kMode>::kBufBytes % 16 == 0, "stage layout");
};

__device__ __forceinline__ int round32(int v) { return (v + 31) & ~31; }
// tokens per tile of an expert with n rows: equal tiles, a multiple of 32
__device__ __forceinline__ int tile_tokens(int n, int largest) {
    const int tiles = (n + largest - 1) / largest;
    return round32((n + tiles - 1) / tiles);
}

struct Tile {
    int expert, row0, tokens;  // tokens: N of the MMA (multiple of 32)
    int wt;                    // weight tile
};

// Unit -> tile.  The token tiles of an expert that share a weight tile are neighbours and go to clusters that start together,
// so that the weights come from memory once and from L2 afterwards (with the weight tiles as neighbours: 754 us instead
// of 729 for 16 experts of 1030 rows).
__device__ __forceinline__ Tile locate(const Shared& sh, int experts, int weight_tiles, int unit, int largest) {
    const int at = unit / weight_tiles;
    int lo = 0, hi = experts;  // first_tile[lo] <= at < first_tile[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (sh.first_tile[mid] <= at) lo = mid; else hi = mid;
    }
    const int tiles = sh.first_tile[lo + 1] - sh.first_tile[lo], j = unit - sh.first_tile[lo] * weight_tiles;
    const int n = sh.rows[lo], tn = tile_tokens(n, largest), start = j % tiles * tn;
    return Tile{lo, sh.offsets[lo] + start, min(tn, round32(n - start)), j / tiles};
}

__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar_cluster_addr) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(map), "r"(bar_cluster_addr), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
// Takes over the place of a cluster of this grid that has not started: 16 bytes of answer, counted in on `bar`.
__device__ __forceinline__ void request_cluster(void* answer, uint64_t* bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(smem_u32(answer)),
                 "r"(smem_u32(bar))
                 : "memory");
}
// First CTA of the cluster taken over, or -1 when none was left.
__device__ __forceinline__ int cancelled_cta(const void* answer) {
    uint32_t taken, x;
    asm volatile(
        "{\n .reg .b128 r;\n .reg .pred p;\n mov.b32 %1, 0;\n ld.shared.b128 r, [%2];\n"
        " clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n selp.u32 %0, 1, 0, p;\n"
        " @p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, _, _, _}, r;\n}"
        : "=&r"(taken), "=&r"(x)
        : "r"(smem_u32(answer))
        : "memory");
    return taken ? int(x) : -1;
}
__device__ __forceinline__ void st_cluster(uint32_t cluster_addr, int v) {
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
// Arrival behind the read that gave `unit`, without the fence of a releasing one.  The barrier's address is computed from the value
// (units lie between -1 and 2^31 - 2, so the added term is 0, which the compiler does not know), so the arrival cannot be on its
// way before the value is there.  Whoever rewrites the slot waits for the arrival first: a read that returned the rewritten
// value would be its own cause, through a chain of dependencies.
__device__ __forceinline__ void arrive_behind(uint32_t cluster_addr, int unit) {
    const uint32_t zero = (uint32_t(unit) + 1u) >> 31;
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr + 8u * zero) : "memory");
}
// Bounded wait that also orders what the other CTA of the pair wrote before its arrival.
__device__ __forceinline__ bool mbar_wait_pair(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
    const uint64_t start = timer_ns();
    uint32_t spins = 0;
    for (;;) {
        uint32_t done;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done)
                     : "r"(smem_u32(bar)), "r"(parity)
                     : "memory");
        if (done) return true;
        if ((++spins & 1023u) == 0u && timer_ns() - start > limit_ns) return false;
    }
}
__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory"); }
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(2 + group) : "memory"); }

template <int kMode, int kTileTokens>
__global__ void __launch_bounds__(kThreads, 1) expert_gemm_kernel(const __grid_constant__ ExpertMaps maps, const __grid_constant__ Args args) {
    using P = Pipe<kMode, kTileTokens>;
    using O = Out<kMode>;
    constexpr int kStages = P::kStages;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* stage_out = smem + kStages * P::kStageBytes;
    Shared& sh = *reinterpret_cast<Shared*>(stage_out + kGroups * O::kBufBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t cta = cluster_ctarank();
    const bool leader = cta == 0;
    const uint64_t limit_ns = args.timeout_ns;

    allow_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&sh.full[s], 1);   // leader: one expect_tx arrival covering both CTAs' bytes
            mbar_init(&sh.empty[s], 1);  // one commit from the leader's MMA thread
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&sh.tmem_full[a], 1);
            mbar_init(&sh.tmem_empty[a], 2 * kEpiThreads / 32);  // leader: the epilogue warps of both CTAs
        }
        mbar_init(&sh.cancel_done, 1);
        for (int u = 0; u < kUnitSlots; ++u) {
            mbar_init(&sh.unit_full[u], 1);
            mbar_init(&sh.unit_empty[u], kUnitReaders);
        }
        sh.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    for (int i = threadIdx.x; i <= args.num_experts; i += kThreads) {
        const int64_t off = args.expert_offsets[i];
        sh.offsets[i] = int(off);
        // one expert per 128-row block: offsets must be multiples of 128, start at 0, not fall, and end at the row count (or in front of it)
        const bool falls = i > 0 && off < args.expert_offsets[i - 1];
        if ((off & 127) != 0 || falls || (i == 0 && off != 0) || (i == args.num_experts && (args.rows_bound ? off > args.rows : off != args.rows))) {
            sh.abort = 1;
            if (atomicCAS(args.status, 0u, uint32_t(kGemmBadOffsets)) == 0u) args.status[1] = uint32_t(i);
        }
    }
    if (warp == 1) tmem_alloc_pair(&sh.tmem_base, kTmemCols);
    __syncthreads();
    if (warp == 0) {
        int carry = 0;
        for (int base = 0; base < args.num_experts; base += 32) {
            const int e = base + lane;
            int n = 0, tiles = 0;
            if (e < args.num_experts && !sh.abort) {
                n = sh.offsets[e + 1] - sh.offsets[e];
                if (args.expert_counts != nullptr) {
                    const int64_t real = args.expert_counts[e];
                    n = int(real < 0 ? 0 : real < n ? real : n);
                }
                if (n > 0) {
                    const int tn = tile_tokens(n, kTileTokens);
                    tiles = (n + tn - 1) / tn;
                }
            }
            int incl = tiles;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += v;
            }
            if (e < args.num_experts) {
                sh.rows[e] = n;
                sh.first_tile[e] = carry + incl - tiles;
            }
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) sh.first_tile[args.num_experts] = carry;
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs have initialised their barriers before anyone signals across
    tc_fence_after();
    const uint32_t tmem_base = sh.tmem_base;

    const int k_blocks = args.k_blocks;
    const int cluster_id = blockIdx.x >> 1, num_clusters = gridDim.x >> 1;
    const int units = sh.first_tile[args.num_experts] * args.n_tiles;  // none after bad offsets
    volatile int* abort_flag = &sh.abort;
    auto fail = [&](uint32_t code) {
        *abort_flag = 1;
        if (atomicCAS(args.status, 0u, code) == 0u) args.status[1] = blockIdx.x;
    };

    // The unit that a reader (one thread) computes behind `unit`, its `item`-th; -1 at the end.  A cluster without a unit of its own
    // asks for its first one as well.
    const bool own_unit = cluster_id < units;
    auto next_unit = [&](int unit, int item) -> int {
        if (*abort_flag) return -1;
        if (!args.dynamic) return unit + num_clusters < units ? unit + num_clusters : -1;
        const int handed = own_unit ? item : item + 1, slot = handed % kUnitSlots;
        if (!mbar_wait_pair(&sh.unit_full[slot], uint32_t(handed / kUnitSlots) & 1u, limit_ns)) {
            fail(kGemmPipeTimeout);
            return -1;
        }
        const int next = *(volatile int*)&sh.next_unit[slot];
        arrive_behind(map_to_cta(smem_u32(&sh.unit_empty[slot]), 1), next);
        return next;
    };
    auto first_unit = [&]() { return own_unit ? cluster_id : args.dynamic ? next_unit(-1, -1) : -1; };

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (both CTAs)
        if (elect_one()) {
            int stage = 0, item = 0;
            uint32_t phase = 0;
            for (int i = first_unit(); i >= 0 && !*abort_flag; i = next_unit(i, item++)) {
                const Tile t = locate(sh, args.num_experts, args.n_tiles, i, kTileTokens);
                const int half = t.tokens / 2, t_row = t.row0 + int(cta) * half;  // this CTA's token rows
                const uint32_t bytes = uint32_t(2 * (kWBytes + half * BK * 2));    // of a stage, in both CTAs
                auto load_weights = [&](int kb, int s) {
                    uint8_t* dst = smem + s * P::kStageBytes;
                    const uint32_t bar = map_to_cta(smem_u32(&sh.full[s]), 0);
                    if (leader) mbar_expect_tx(&sh.full[s], bytes);
                    if (kMode == kSwiGLU) {
                        // 16 gate rows followed by their 16 up rows, four times: 64 output features of this CTA
                        const int f0 = t.wt * 128 + int(cta) * 64;
#pragma unroll
                        for (int q = 0; q < 4; ++q) tma_load_3d_pair(dst + q * 4096, &maps.weights, kb * BK, f0 + 16 * q, 2 * t.expert, bar);
                    } else {
                        tma_load_2d_pair(dst, &maps.weights, kb * BK, t.expert * args.b_rows_per_expert + t.wt * BW + int(cta) * (BW / 2), bar);
                    }
                };
                auto load_tokens = [&](int kb, int s) {
                    uint8_t* dst = smem + s * P::kStageBytes + kWBytes;
                    const uint32_t bar = map_to_cta(smem_u32(&sh.full[s]), 0);
                    // boxes of 128, 64, 32 and 16 rows make up any multiple of 16
                    int at = 0;
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        const int box = 128 >> b;
                        if (half & box) {
                            tma_load_2d_pair(dst + at * BK * 2, &maps.tokens[b], kb * BK, t_row + at, bar);
                            at += box;
                        }
                    }
                };
                int early = 0;  // k-blocks whose weights are on their way already
                if (item == 0) {
                    // The ring is empty: fill it with weights while the kernel in front, which writes the token rows, ends.  (A layer of
                    // 64 tokens, 32 experts of 7168 x 2048, with a cached handle 446 -> 437.7 us; of 777 tokens, 4096 x 1536, 289 -> 284.)
                    early = min(kStages, k_blocks);
                    for (int kb = 0; kb < early; ++kb) load_weights(kb, kb);
                    wait_for_previous();
                }
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (kb >= early) {
                        if (!mbar_wait(&sh.empty[stage], phase ^ 1u, limit_ns)) {
                            fail(kGemmPipeTimeout);
                            break;
                        }
                        load_weights(kb, stage);
                    }
                    load_tokens(kb, stage);
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (leader CTA only)
        if (leader && elect_one()) {
            int stage = 0, item = 0;
            uint32_t phase = 0;
            wait_for_previous();  // the time limits below are this kernel's, not those of a pull that waits for its peers in front of it
            for (int i = first_unit(); i >= 0 && !*abort_flag; i = next_unit(i, item++)) {
                const Tile t = locate(sh, args.num_experts, args.n_tiles, i, kTileTokens);
                const uint32_t idesc = instr_desc_bf16(BW, t.tokens);
                const int acc = item & 1;
                if (!mbar_wait(&sh.tmem_empty[acc], (uint32_t(item >> 1) & 1u) ^ 1u, limit_ns)) {
                    fail(kGemmPipeTimeout);
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + uint32_t(acc * kAccCols);
                auto commit = [&](uint64_t* bar) {  // in both CTAs, once the MMAs so far have been done
                    tc_commit_pair(map_to_cta(smem_u32(bar), 0));
                    tc_commit_pair(map_to_cta(smem_u32(bar), 1));
                };
                bool ok = true;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_wait(&sh.full[stage], phase, limit_ns)) {
                        fail(kGemmPipeTimeout);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint8_t* w_tile = smem + stage * P::kStageBytes;
                    const uint64_t w_desc = smem_desc_sw128(w_tile);
                    const uint64_t t_desc = smem_desc_sw128(w_tile + kWBytes);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        tc_mma_pair(d_tmem, w_desc + uint64_t(k * 2), t_desc + uint64_t(k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
                    commit(&sh.empty[stage]);
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (!ok) break;
                commit(&sh.tmem_full[acc]);
            }
        }
        // ------------------------------------------------------------------ scheduler (the other CTA)
        if (!leader && args.dynamic && elect_one()) {
            struct {
                Shared& sh;
                uint64_t limit_ns;
                int answers;
                __device__ bool wait_read(int n) {
                    if (n == kUnitSlots) wait_for_previous();  // as the readers do
                    return mbar_wait_pair(&sh.unit_empty[n % kUnitSlots], uint32_t(n / kUnitSlots - 1) & 1u, limit_ns);
                }
                __device__ bool request(int& place) {
                    mbar_expect_tx(&sh.cancel_done, 16);
                    request_cluster(sh.cancelled, &sh.cancel_done);
                    if (!mbar_wait(&sh.cancel_done, uint32_t(answers++) & 1u, limit_ns)) return false;
                    const int cta_taken = cancelled_cta(sh.cancelled);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the next answer comes behind this read
                    place = cta_taken < 0 ? -1 : cta_taken >> 1;
                    return true;
                }
                __device__ void hand_out(int n, int unit) {
                    const int at = n % kUnitSlots;
                    *(volatile int*)&sh.next_unit[at] = unit;
                    st_cluster(map_to_cta(smem_u32(&sh.next_unit[at]), 0), unit);
                    mbar_arrive_cluster(map_to_cta(smem_u32(&sh.unit_full[at]), 1));
                    mbar_arrive_cluster(map_to_cta(smem_u32(&sh.unit_full[at]), 0));
                }
            } io{sh, limit_ns, 0};
            if (!hand_out_units(io, units, num_clusters, cluster_id)) fail(kGemmPipeTimeout);
        }
    } else {
        // ------------------------------------------------------------------ epilogue (both CTAs)
        const int quarter = warp & 3;             // TMEM lanes [32 * quarter, +32) belong to this warp
        const int group = (warp - 2) >> 2;        // every second chunk of token rows
        const int tid = threadIdx.x - 64, gtid = tid & 127;
        const int tok_of = 2 * (lane & 3);
        // stmatrix: matrix m = lane / 8 holds token group m / 2 and feature half m % 2; this lane addresses its row lane % 8
        const int st_tok = (lane >> 4) * 8 + (lane & 7), st_feat = ((lane >> 3) & 1) * 8;
        uint8_t* buf = stage_out + group * O::kBufBytes;
        // Rows, scales and destinations are the work of kernels in front; no CTA ends before those have.
        wait_for_previous();
        int unit = -1;  // warp 2, lane 0
        for (int item = 0;; ++item) {
            if (warp == 2) {
                if (lane == 0) {
                    unit = item > 0 ? next_unit(unit, item - 1) : first_unit();
                    *(volatile int*)&sh.epi_unit[item & 1] = unit;
                }
                __syncwarp();
            }
            epilogue_sync();  // and the previous unit's destinations have been used
            const int i = *(volatile int*)&sh.epi_unit[item & 1];
            if (i < 0) break;
            const Tile t = locate(sh, args.num_experts, args.n_tiles, i, kTileTokens);
            if (kMode != kSwiGLU) {
                for (int r = tid; r < t.tokens; r += kEpiThreads) {
                    const int row = t.row0 + r;
                    float scale = 1.f;
                    if (kMode == kScatter) {
                        char* dst = nullptr;
                        const int a = args.slot_map[row];
                        if (a >= 0) {
                            const int recv_row = a / args.topk, k = a % args.topk;
                            const int* meta = args.recv_metadata + int64_t(recv_row) * (args.topk + 2);
                            const bool inside = recv_row < args.recv_rows;
                            const int src = inside ? meta[0] : -1, tok = inside ? meta[1] : -1;
                            if (src < 0 || src >= args.ranks || tok < 0 || tok >= args.max_tokens) {
                                // impossible provenance: skip the row and report it, as the push kernel does
                                if (atomicCAS(args.status, 0u, uint32_t(kGemmBadMetadata)) == 0u) args.status[1] = uint32_t(row);
                            } else {
                                if (args.slot_weights != nullptr) scale = args.slot_weights[row];
                                dst = static_cast<char*>(args.peers[src]) + args.ret_offset + (int64_t(k) * args.max_tokens + tok) * int64_t(args.ldo) * 2;
                            }
                        }
                        sh.dst[r] = dst;
                    } else if (args.row_scale != nullptr) {
                        scale = args.row_scale[row];
                    }
                    sh.scale[r] = scale;
                }
            }
            const int acc = item & 1;
            // one warp waits and decides for all: they share the staging buffers and their barriers
            if (warp == 2) {
                bool ok = !*abort_flag && mbar_wait(&sh.tmem_full[acc], uint32_t(item >> 1) & 1u, limit_ns);
                ok = __all_sync(0xffffffffu, ok);
                if (lane == 0) {
                    if (!ok) fail(kGemmPipeTimeout);
                    *(volatile int*)&sh.go[acc] = ok;
                }
            }
            epilogue_sync();
            if (!*(volatile int*)&sh.go[acc]) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + (uint32_t(quarter * 32) << 16) + uint32_t(acc * kAccCols);
            const int col0 = t.wt * 2 * O::kFeatures + int(cta) * O::kFeatures;  // first output column of this CTA
            auto drained = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&sh.tmem_empty[acc]), 0));
            };
            if (group * kChunk >= t.tokens) drained();
            for (int c0 = group * kChunk; c0 < t.tokens; c0 += kGroups * kChunk) {
                uint32_t lo[16], hi[16];  // lanes 0..15 and 16..31 of the quarter
                tmem_ld_16x32(taddr + uint32_t(c0), lo);
                tmem_ld_16x32(taddr + (16u << 16) + uint32_t(c0), hi);
                tmem_ld_wait();
                if (c0 + kGroups * kChunk >= t.tokens) drained();
                group_sync(group);  // the rows staged before have been read
#pragma unroll
                for (int j = 0; j < 4; j += 2) {  // token groups j and j + 1 (8 tokens each)
                    if (kMode == kSwiGLU) {
                        uint32_t o[4];
#pragma unroll
                        for (int m = 0; m < 4; ++m) {
                            const int r = 4 * (j + (m >> 1)) + 2 * (m & 1);
                            o[m] = pack_bf16(silu(__uint_as_float(lo[r])) * __uint_as_float(hi[r]),
                                             silu(__uint_as_float(lo[r + 1])) * __uint_as_float(hi[r + 1]));
                        }
                        st_matrix_x4_trans(buf + (8 * j + st_tok) * O::kPitch + (16 * quarter + st_feat) * 2, o[0], o[1], o[2], o[3]);
                    } else {
                        float f[4];  // tokens of groups j and j + 1
#pragma unroll
                        for (int m = 0; m < 4; ++m) f[m] = sh.scale[c0 + 8 * (j + (m >> 1)) + tok_of + (m & 1)];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t o[4];
#pragma unroll
                            for (int m = 0; m < 4; ++m) {
                                const int r = 4 * (j + (m >> 1)) + 2 * (m & 1);
                                const uint32_t a = h ? hi[r] : lo[r], b = h ? hi[r + 1] : lo[r + 1];
                                o[m] = pack_bf16(__uint_as_float(a) * f[m & 2], __uint_as_float(b) * f[(m & 2) + 1]);
                            }
                            st_matrix_x4_trans(buf + (8 * j + st_tok) * O::kPitch + (32 * quarter + 16 * h + st_feat) * 2, o[0], o[1], o[2], o[3]);
                        }
                    }
                }
                group_sync(group);
                // whole token rows leave, 16 bytes per thread
                constexpr int kVecs = O::kRowBytes / 16;
#pragma unroll
                for (int v = gtid; v < kChunk * kVecs; v += 128) {
                    const int r = v / kVecs, c = v % kVecs;
                    const int4 d = *reinterpret_cast<const int4*>(buf + r * O::kPitch + c * 16);
                    char* row = kMode == kScatter ? static_cast<char*>(sh.dst[c0 + r])
                                                  : reinterpret_cast<char*>(args.out + int64_t(t.row0 + c0 + r) * args.ldo);
                    if (kMode != kScatter || row != nullptr) *reinterpret_cast<int4*>(row + col0 * 2 + c * 16) = d;
                }
            }
        }
        if (kMode == kScatter) __threadfence_system();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the peer may still be reading this CTA's operands / signalling its barriers
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

template <int kMode, int kTileTokens>
cudaError_t launch_tile(const ExpertMaps& maps, const Args& args, int grid, bool early, cudaStream_t stream) {
    auto* fn = expert_gemm_kernel<kMode, kTileTokens>;
    using P = Pipe<kMode, kTileTokens>;
    // The limit is the same for every launch of this kernel: raised once per device (a second thread may do it again).
    static std::atomic<uint64_t> raised{0};
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const uint64_t bit = device < 64 ? uint64_t(1) << device : 0;
    if ((raised.load(std::memory_order_acquire) & bit) == 0) {
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(P::kSmemBytes));
        if (e != cudaSuccess) return e;
        raised.fetch_or(bit, std::memory_order_release);
    }
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(unsigned(grid));
    config.blockDim = dim3(kThreads);
    config.dynamicSmemBytes = P::kSmemBytes;
    config.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attr;
    config.numAttrs = early ? 2 : 1;
    return cudaLaunchKernelEx(&config, fn, maps, args);
}

template <int kMode>
cudaError_t launch_mode(const ExpertMaps& maps, const Args& args, int tile_tokens, int grid, bool early, cudaStream_t stream) {
    if (tile_tokens <= 64) return launch_tile<kMode, 64>(maps, args, grid, early, stream);
    if (tile_tokens <= 128) return launch_tile<kMode, 128>(maps, args, grid, early, stream);
    return launch_tile<kMode, 256>(maps, args, grid, early, stream);
}

}  // namespace

cudaError_t launch_expert(const ExpertMaps& maps, const Args& args, int mode, int tile_tokens, int grid, bool early, cudaStream_t stream) {
    if (args.num_experts > kMaxExperts) return cudaErrorInvalidValue;
    grid &= ~1;
    if (grid < 2) return cudaErrorInvalidValue;
    if (mode == kPlain) return launch_mode<kPlain>(maps, args, tile_tokens, grid, early, stream);
    if (mode == kSwiGLU) return launch_mode<kSwiGLU>(maps, args, tile_tokens, grid, early, stream);
    if (mode == kScatter) return launch_mode<kScatter>(maps, args, tile_tokens, grid, early, stream);
    return cudaErrorInvalidValue;
}

}  // namespace gemm
}  // namespace nep
