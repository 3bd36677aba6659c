// Dispatch / combine kernels for sm_100a: stage, plan, pull, push, reduce, barrier.
// See ep_kernels.hpp for the protocol.  All waits are bounded (prim.cuh); nothing traps.
#include "ep_kernels.hpp"

#include <map>
#include <mutex>
#include <utility>

#include "flag_queue.hpp"
#include "prim.cuh"

namespace nep {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kStageThreads = 512;
constexpr int kPlanThreads = 256;
constexpr int kLocalPlanThreads = 512;
constexpr int kLocalPlanCtas = 8;  // largest cluster every GPU of this architecture accepts
constexpr int kLocalPlanChunks = kLocalPlanMaxTokens / 32 / kLocalPlanCtas;
constexpr int kRowSumThreads = 256, kRowSumBlocks = 2, kRowCopyBlocks = 5;  // blocks: resident per SM
constexpr int kZeroBytes = 2048;  // smallest zero source of the padding rows
constexpr int kTagStage = 1, kTagPlan = 2, kTagPull = 3, kTagPush = 4, kTagReduce = 5, kTagBarrier = 6;

__device__ __forceinline__ char* window(const CommonParams& c, int r) { return static_cast<char*>(c.peers[r]); }
__device__ __forceinline__ int* ctrl_words(const CommonParams& c) {
    return reinterpret_cast<int*>(window(c, c.rank) + c.layout.ctrl_offset);
}
__device__ __forceinline__ StatusRef status_of(const CommonParams& c) { return StatusRef{c.status_dev, c.status_host}; }
__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// The block that takes the last ticket runs the tail of a kernel; the counter is reset by it.  One thread's fences stand for
// the block's: what the other threads wrote is ordered before them by the block barrier, and what other blocks wrote before
// their tickets is ordered for the other threads by the second one.
__device__ __forceinline__ int take_ticket(int* ticket) {
    __shared__ int number;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        number = atomicAdd(ticket, 1);
        __threadfence();
    }
    __syncthreads();
    return number;
}
__device__ __forceinline__ bool take_last_ticket(int* ticket) { return take_ticket(ticket) == int(gridDim.x) - 1; }

// Single-launch paths: the block that took the last ticket runs the peer barrier and then tells the other
// blocks of its rank the outcome through one word: +tag = go, -tag = failed (tag derives from the epoch, never 0).
__device__ __forceinline__ int go_tag(uint64_t epoch) { return int(epoch & 0x3fffffff) | 0x40000000; }

__device__ __forceinline__ void publish_go(int* ctrl, uint64_t epoch, bool ok, int word = WindowLayout::kGoWord) {
    const int want = go_tag(epoch);
    __threadfence();
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(ctrl + word), "r"(ok ? want : -want) : "memory");
}

// Called by every thread of a block; thread 0 polls (bounded), the block gets the outcome.
__device__ bool wait_go(int* ctrl, uint64_t epoch, uint64_t timeout_ns, StatusRef status, uint32_t tag, int word = WindowLayout::kGoWord) {
    __shared__ int s_go;
    if (threadIdx.x == 0) {
        const int want = go_tag(epoch);
        const uint64_t start = global_timer_ns();
        int seen = 0;
        for (;;) {
            seen = ld_acquire_gpu(ctrl + word);
            if (seen == want || seen == -want) break;
            __nanosleep(32);
            if (global_timer_ns() - start > 2 * timeout_ns) {
                report(status, kBarrierTimeout, 0xffffu, tag);
                seen = -want;
                break;
            }
        }
        s_go = seen == want;
    }
    __syncthreads();
    return s_go != 0;
}

// Receive counts to the host, which returns from the dispatch with them.  Later kernels of this stream see everything else
// that this kernel writes, so no fence stands here in general.  A gated dispatch is the exception: its consumer runs on
// another stream and reads expert_offsets and expert_counts as soon as the host has the counts, ordered behind nothing but
// the mailbox (`ordered`).  Called by the thread that has observed (block or warp barrier) all of the block's writes to those two.
__device__ __forceinline__ void publish_counts(volatile int64_t* mailbox, int64_t rows, int64_t capacity, bool ordered) {
    if (ordered) __threadfence_system();
    mailbox[1] = capacity;
    mailbox[0] = rows;
}

// ------------------------------------------------------------------------------------------
// stage: copy this rank's tokens (x + gate weights) into its own window, snapshot and count the
// routing, send the per-destination counts to the peers, peer barrier, derive N / C / offsets.
// ------------------------------------------------------------------------------------------
// Returns true when the peer barrier succeeded (only meaningful to every block in fused mode).
__device__ bool stage_body(const StageParams& p) {
    extern __shared__ int s_counts[];  // [R + E]
    const WindowLayout& L = p.c.layout;
    const int R = L.ranks, K = L.topk, H = L.hidden, Le = L.local_experts;
    const int E = int(L.num_experts);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wpb = blockDim.x >> 5;
    const int gw = blockIdx.x * wpb + warp, GW = gridDim.x * wpb;
    char* win = window(p.c, p.c.rank);
    int* ctrl = ctrl_words(p.c);
    int* count_acc = ctrl + L.ctrl_count_acc();
    const StatusRef status = status_of(p.c);

    if (p.fresh) {
        for (int i = tid; i < R + E; i += blockDim.x) s_counts[i] = 0;
        __syncthreads();
    }
    char* rows = win + L.stage_rows_offset + int64_t(p.parity) * L.stage_rows_stride;
    // this rank's slice of every receiver's routing table
    const int64_t routing_slice = L.routing_in_offset + int64_t(p.parity) * L.routing_in_stride + int64_t(p.c.rank) * L.max_tokens * K * 4;
    const int64_t rb = L.row_bytes();
    const int vecs = H / 8;  // 16-byte chunks per row

    auto stamp = [&](int slot) {
        if (p.trace != nullptr && tid == 0) atomicMax(p.trace + slot, global_timer_ns());
    };
    if (p.trace != nullptr && tid == 0) atomicMin(p.trace, global_timer_ns());

    // ---- fresh dispatch, step 1: snapshot, validate, publish and count the routing (one warp per token).  The
    // counts are what every rank and the host wait for, so they go first; the rows follow underneath the exchange.
    bool runs_tail = false;
    int share = int(blockIdx.x), shares = int(gridDim.x);  // this block's share of the rows to copy
    if (p.fresh) {
        for (int t = gw; t < p.tokens; t += GW) {
            int e = -1;
            bool valid = false;
            if (lane < K) {
                const int64_t raw = p.topk[int64_t(t) * K + lane];
                p.snapshot[int64_t(t) * K + lane] = raw;
                if (raw >= 0 && raw < E) {
                    e = int(raw);
                    valid = true;
                } else if (raw != -1) {
                    report(status, kBadExpertId, uint32_t(t), kTagStage);
                }
                // Publish the routing to every rank (itself included): receivers plan from local memory.
                for (int d = 0; d < R; ++d) reinterpret_cast<int*>(window(p.c, d) + routing_slice)[int64_t(t) * K + lane] = e;
            }
            const unsigned vmask = __ballot_sync(kFull, valid);
            const int d = valid ? e / Le : -1;
            if (valid) {
                atomicAdd(&s_counts[R + e], 1);
                const unsigned same = __match_any_sync(vmask, d);
                if (lane == __ffs(same) - 1) atomicAdd(&s_counts[d], 1);
            }
            const unsigned dmask = __reduce_or_sync(kFull, valid ? (1u << d) : 0u);
            if (lane < R) {
                const bool goes = (dmask >> lane) & 1u;
                p.dst_slots[int64_t(t) * R + lane] = goes ? int64_t(t) : int64_t(-1);
                // rows this rank sends to destination `lane` out of the token's chunk of 32: the receivers turn these
                // into row offsets, so that receive rows are ordered by (source rank, source token)
                if (goes) atomicAdd(ctrl + L.ctrl_chunk_acc() + int64_t(lane) * L.chunks_per_rank() + (t >> 5), 1);
            }
        }
        __syncthreads();
        for (int i = tid; i < R + E; i += blockDim.x)
            if (s_counts[i] != 0) atomicAdd(&count_acc[i], s_counts[i]);
        share = take_ticket(ctrl + WindowLayout::kTicketStage);
        runs_tail = share == shares - 1;
        if (shares > 1) --shares;  // the block that runs the tail copies nothing where there are others
        stamp(1);
    }

    __shared__ int s_ok;
    __shared__ int s_rows;  // receive rows of this rank

    auto copy_rows = [&]() {
        // ---- rows: x and gate weights into this rank's staging area.  Work item = one quarter of a token row, so that
        // even a few thousand tokens spread over the whole grid and every lane keeps up to eight 16-byte loads in flight.
        if (!p.skip_copy) {
            constexpr int kParts = 4;
            const int per_part = (vecs + kParts - 1) / kParts;
            for (int item = share * wpb + warp; item < p.tokens * kParts; item += shares * wpb) {
                const int t = item / kParts, q = item % kParts;
                const int4* src = reinterpret_cast<const int4*>(p.x + int64_t(t) * H);
                int4* dst = reinterpret_cast<int4*>(rows + int64_t(t) * rb);
                const int end = min(vecs, (q + 1) * per_part);
                for (int i = q * per_part + lane; i < end; i += 256) {
                    int4 v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (i + j * 32 < end) v[j] = ld_nc_v4(src + i + j * 32);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (i + j * 32 < end) dst[i + j * 32] = v[j];
                }
                if (q == 0 && lane < K) {
                    const float w = p.weights != nullptr ? p.weights[int64_t(t) * K + lane] : 0.f;
                    reinterpret_cast<float*>(rows + int64_t(t) * rb + wire_weights_offset(H))[lane] = w;
                }
            }
        }
    };

    // The tail: run by ONE block per rank (the one that took the last ticket of the counting step, or of the copy in a
    // cached dispatch).  Returns whether the peer barrier succeeded.
    auto tail = [&]() -> bool {
        // ---- tail: one block per rank
        const int msg = int(L.msg_ints());
        if (p.fresh) {
            for (int i = tid; i < R * msg; i += blockDim.x) {
                const int d = i / msg, j = i % msg;
                const int v = j == 0 ? __ldcg(count_acc + d) : j == 1 ? p.tokens : __ldcg(count_acc + R + d * Le + (j - 2));
                int* remote =
                    reinterpret_cast<int*>(window(p.c, d) + L.counts_in_offset + int64_t(p.parity) * L.counts_in_stride) + p.c.rank * msg + j;
                st_relaxed_sys(remote, v);
            }
            for (int d = tid; d < R; d += blockDim.x) p.send_counts[d] = __ldcg(count_acc + d);
            // per-chunk row counts go to their destination (the accumulators are cleared for the next dispatch)
            const int cps = int(L.chunks_per_rank()), my_chunks = (p.tokens + 31) / 32;
            int* chunk_acc = ctrl + L.ctrl_chunk_acc();
            for (int i = tid; i < R * my_chunks; i += blockDim.x) {
                const int d = i / my_chunks, c = i % my_chunks;
                int* remote = reinterpret_cast<int*>(window(p.c, d) + L.chunks_in_offset + int64_t(p.parity) * L.chunks_in_stride) + p.c.rank * cps + c;
                st_relaxed_sys(remote, __ldcg(chunk_acc + d * cps + c));
                chunk_acc[d * cps + c] = 0;
            }
            __syncthreads();
            for (int i = tid; i < R + E; i += blockDim.x) count_acc[i] = 0;
        }
        if (tid == 0) ctrl[WindowLayout::kTicketStage] = 0;
        if (R > 1) {
            __threadfence_system();
            __syncthreads();
            if (warp == 0) {
                const bool ok = peer_barrier_warp(p.c.peers, p.c.rank, R, L.signal_offset, p.epoch, p.c.timeout_ns, status, kTagStage);
                if (lane == 0) s_ok = ok;
            }
        } else {
            // a single-rank group has nobody to wait for: its own messages are ordered by the block barrier below
            __threadfence();
            if (tid == 0) s_ok = 1;
        }
        __syncthreads();
        stamp(3);
        if (p.fused && !p.fresh) {
            if (tid == 0) publish_go(ctrl, p.epoch, s_ok != 0);
            return s_ok != 0;
        }
        if (!p.fresh) return s_ok != 0;
        if (!s_ok) {
            if (tid == 0) {
                __threadfence_system();
                p.mailbox[1] = -2;
                p.mailbox[0] = -2;
                if (p.fused) publish_go(ctrl, p.epoch, false);
            }
            return false;
        }
        const int* in = reinterpret_cast<const int*>(win + L.counts_in_offset + int64_t(p.parity) * L.counts_in_stride);
        // The host waits for what follows: loads are issued in groups, not one behind the other, and the mailbox is written
        // before the chunk prefixes.  Eight ranks of 16 tokens: counts in the mailbox 20 -> 14 us after the kernel's start.
        // Phase 1 (all threads): per local expert, sum the sources' counts and round up to the alignment.
        // The padded sizes reuse the dynamic shared array (R + E ints >= L ints).
        int* s_padded = s_counts;
        for (int l = tid; l < Le; l += blockDim.x) {
            int cnt = 0;
            for (int src0 = 0; src0 < R; src0 += 8) {
                int v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = src0 + j < R ? ld_relaxed_sys(in + (src0 + j) * msg + 2 + l) : 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) cnt += v[j];
            }
            p.expert_counts[l] = cnt;
            ctrl[L.ctrl_expert_counts() + l] = cnt;
            ctrl[L.ctrl_expert_cursor() + l] = 0;
            s_padded[l] = (cnt + p.alignment - 1) / p.alignment * p.alignment;
        }
        // receive rows by source: inclusive prefix (R <= 32)
        if (warp == 0) {
            const int n = lane < R ? ld_relaxed_sys(in + lane * msg) : 0;
            const int tokens = lane < R ? ld_relaxed_sys(in + lane * msg + 1) : 0;
            const int incl = warp_inclusive_sum(n);
            if (lane < R) {
                p.recv_rank_prefix[lane] = incl;
                ctrl[L.ctrl_recv_prefix() + lane] = incl - n;
                ctrl[L.ctrl_src_tokens() + lane] = tokens;
            }
            if (lane == R - 1) {
                ctrl[L.ctrl_recv_prefix() + R] = incl;
                s_rows = incl;
            }
        }
        __syncthreads();
        if (warp == 0) {
            // Phase 2: exclusive scan of the padded sizes in waves of 32 (shared memory only)
            int carry = 0;
            for (int base = 0; base < Le; base += 32) {
                const int l = base + lane;
                const int padded = l < Le ? s_padded[l] : 0;
                const int incl = warp_inclusive_sum(padded);
                if (l < Le) {
                    const int off = carry + incl - padded;
                    p.expert_offsets[l] = off;
                    ctrl[L.ctrl_expert_offsets() + l] = off;
                }
                carry += __shfl_sync(kFull, incl, 31);
            }
            if (lane == 0) {
                p.expert_offsets[Le] = carry;
                ctrl[L.ctrl_expert_offsets() + Le] = carry;
            }
            __syncwarp();  // the other lanes' offsets; the counts are behind the block barrier above
            // reports of invalid ids reach the host before the counts do (a group has passed the system fence of its
            // peer barrier): the call after this one raises them
            if (lane == 0) publish_counts(p.mailbox, s_rows, carry, p.gated != 0 || R == 1);
        }
        // Every source's per-chunk row counts become exclusive prefixes: chunk c of source s starts at receive row
        // recv_prefix[s] + chunk_prefix[s][c].  The total must equal the source's announced row count.
        {
            const int cps = int(L.chunks_per_rank());
            int* chunks = reinterpret_cast<int*>(win + L.chunks_in_offset + int64_t(p.parity) * L.chunks_in_stride);
            for (int s = wpb - 1 - warp; s < R; s += wpb) {  // warp 0 comes last: it has the scan above
                const int tokens = ld_relaxed_sys(in + s * msg + 1), announced = ld_relaxed_sys(in + s * msg);
                const int n_chunks = (tokens + 31) / 32;
                int carry = 0;
                for (int base = 0; base < n_chunks; base += 32) {
                    const int c = base + lane;
                    const int v = c < n_chunks ? ld_relaxed_sys(chunks + s * cps + c) : 0;
                    const int incl = warp_inclusive_sum(v);
                    if (c < n_chunks) chunks[s * cps + c] = carry + incl - v;
                    carry += __shfl_sync(kFull, incl, 31);
                }
                if (lane == 0 && carry != announced) report(status, kSlotOverflow, uint32_t(s), kTagStage);
            }
        }
        __syncthreads();
        // the other blocks of a single-launch dispatch go on to plan
        if (tid == 0 && p.fused) publish_go(ctrl, p.epoch, true);
        stamp(4);
        return true;
    };

    if (p.fresh) {
        // The count exchange comes first: every rank and the host wait for it.  The rows are staged underneath it by all
        // the other blocks; the tail block copies only where it is alone.  (With a share of its own behind the tail it was the
        // last to finish.  Without it, with one system fence per signal and two blocks per SM, the kernel alone with cold caches: eight ranks
        // of 16 tokens 46 -> 26 us, of 512 tokens 62 -> 32; four skewed ranks of 1000 tokens 54 -> 26.)
        bool ok = true;
        if (runs_tail) ok = tail();
        if (share < shares) {
            copy_rows();
            // The block that finishes its rows last tells every peer that this rank's rows are staged; the receivers'
            // pull waits for these signals, nobody waits here.
            if (take_ticket(ctrl + WindowLayout::kTicketCopy) == shares - 1) {
                if (tid == 0) ctrl[WindowLayout::kTicketCopy] = 0;
                // a single-rank group stages nothing and its pull waits for no signal
                if (R > 1 && warp == 0) peer_signal_warp(p.c.peers, p.c.rank, R, L.data_signal_offset, p.epoch);
            }
        }
        stamp(2);
        if (runs_tail) return ok;
        // single-launch fresh dispatch: wait for the tail block's prefixes before planning
        if (!p.fused) return false;
        return wait_go(ctrl, p.epoch, p.c.timeout_ns, status, kTagStage);
    }
    copy_rows();
    if (!take_last_ticket(ctrl + WindowLayout::kTicketStage)) {
        if (!p.fused) return false;
        return wait_go(ctrl, p.epoch, p.c.timeout_ns, status, kTagStage);
    }
    return tail();
}

// ------------------------------------------------------------------------------------------
// local_plan (fresh dispatch of a single-rank group): counts, offsets, receive rows and slots in ONE launch.
//
// Bound by latency, not by bytes: 4096 tokens x top-8 read 256 KB and write 0.9 MB.  With nobody to exchange counts with,
// a cluster of up to eight CTAs replaces the stage and plan kernels with their grid-wide tickets and global atomics:
// each CTA counts a contiguous range of tokens in shared memory, the CTAs read one another's counts through distributed
// shared memory, and every CTA derives the same offsets and its own first slots from them.  Metadata goes straight to
// the handle's tensors, and N and C reach the host before the rows are assigned.
// Against stage + plan, top-8 of 256 experts: 1 token 22 -> 6.6 us, 256 tokens 14.6 -> 8.1 us, 4096 tokens 25 -> 14 us;
// the pull of a call whose output bound is modest no longer waits for the host: 1 token and its combine 59 -> 52 us.
// A chain of latencies throughout, so: all threads scan the experts instead of one warp in waves, the other CTAs' counts and the
// slots of eight choices are asked for at once, and a warp keeps the choices of its only chunk.  The kernel alone with cold
// caches: 1 token 8.0 -> 6.7 us, 256 tokens 10.5 -> 9.2, 4096 tokens 15.2 -> 13.3.  (In a call, which the host bounds, half a
// microsecond of 36 to 40, no more than runs of one side differ.)
// ------------------------------------------------------------------------------------------
__device__ void local_plan_body(const LocalPlanParams& p) {
    extern __shared__ int s_plan[];
    const WindowLayout& L = p.c.layout;
    const int K = L.topk, E = int(L.num_experts);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kWarps = kLocalPlanThreads / 32;
    const int cta = int(cluster_rank()), ctas = int(cluster_size());
    const StatusRef status = status_of(p.c);
    int* s_count = s_plan;          // [E] choices of this CTA's tokens per expert (read by the other CTAs)
    int* s_cursor = s_count + E;    // [E] next slot
    int* s_padded = s_cursor + E;   // [E] padded size, then offset
    int* s_real = s_padded + E;     // [E] choices of all CTAs
    int* s_rows = s_real + E;       // [kLocalPlanChunks] rows of this CTA's chunks of 32 tokens, then their prefix
    int* mine = s_rows + kLocalPlanChunks + warp * 32 * K;  // [32 * K] experts of the warp's chunk
    __shared__ int s_total;         // rows of this CTA (read by the other CTAs)
    __shared__ int s_invalid;       // a token of this CTA names an expert that does not exist (read by the other CTAs)
    __shared__ int s_first, s_all, s_any_invalid;
    __shared__ int s_warp[kWarps];
    allow_dependents();
    wait_for_previous();
    const int chunks = (p.tokens + 31) / 32, per_cta = (chunks + ctas - 1) / ctas;
    const int first_chunk = cta * per_cta, my_chunks = max(0, min(per_cta, chunks - first_chunk));
    for (int i = tid; i < E; i += kLocalPlanThreads) s_count[i] = 0;
    if (tid == 0) s_invalid = 0;
    __syncthreads();

    // experts of a chunk into the warp's buffer; `first` also snapshots, validates and counts them
    auto load_chunk = [&](int chunk, bool first) -> int {
        const int tok0 = chunk * 32, n_tok = min(32, p.tokens - tok0), n = n_tok * K;
        const int64_t base = int64_t(tok0) * K;
        __syncwarp();
        for (int i0 = 0; i0 < n; i0 += 256) {
            int64_t raw[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int i = i0 + 32 * j + lane;
                raw[j] = i < n ? p.topk[base + i] : -1;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int i = i0 + 32 * j + lane;
                if (i >= n) break;
                const bool valid = raw[j] >= 0 && raw[j] < E;
                mine[i] = valid ? int(raw[j]) : -1;
                if (first) {
                    p.snapshot[base + i] = raw[j];
                    if (valid) {
                        atomicAdd(&s_count[int(raw[j])], 1);
                    } else if (raw[j] != -1) {
                        report(status, kBadExpertId, uint32_t(tok0 + i / K), kTagStage);
                        s_invalid = 1;
                    }
                }
            }
        }
        __syncwarp();
        bool has = false;
        if (lane < n_tok)
            for (int k = 0; k < K; ++k) has |= mine[lane * K + k] >= 0;
        if (first && lane < n_tok) p.dst_slots[tok0 + lane] = has ? tok0 + lane : -1;
        return has;
    };

    // ---- count
    bool kept = false;  // whether the lane's token of the chunk loaded last has a row
    for (int ch = warp; ch < my_chunks; ch += kWarps) {
        kept = load_chunk(first_chunk + ch, true) != 0;
        const unsigned hm = __ballot_sync(kFull, kept);
        if (lane == 0) s_rows[ch] = __popc(hm);
    }
    __syncthreads();
    if (warp == 0) {
        int carry = 0;
        for (int b = 0; b < my_chunks; b += 32) {
            const int v = b + lane < my_chunks ? s_rows[b + lane] : 0;
            const int incl = warp_inclusive_sum(v);
            if (b + lane < my_chunks) s_rows[b + lane] = carry + incl - v;
            carry += __shfl_sync(kFull, incl, 31);
        }
        if (lane == 0) s_total = carry;
    }
    cluster_arrive();
    cluster_wait();
    // ---- combine the CTAs' counts
    if (warp == kWarps - 1) {
        const int v = lane < ctas ? ld_cluster_smem(&s_total, uint32_t(lane)) : 0;
        const int incl = warp_inclusive_sum(v);
        if (lane == cta) s_first = incl - v;
        const bool any = __any_sync(kFull, lane < ctas && ld_cluster_smem(&s_invalid, uint32_t(lane)) != 0);
        if (lane == 31) {
            s_all = incl;
            s_any_invalid = any;
        }
    }
    int capacity = 0;  // padded rows of the experts so far; every thread ends with all of them
    for (int e0 = 0; e0 < E; e0 += kLocalPlanThreads) {
        const int e = e0 + tid;
        int before = 0, all = 0;
        if (e < E) {
            int v[kLocalPlanCtas];  // all CTAs' counts are on their way before the first is used
#pragma unroll
            for (int c = 0; c < kLocalPlanCtas; ++c) v[c] = c < ctas ? ld_cluster_smem(s_count + e, uint32_t(c)) : 0;
#pragma unroll
            for (int c = 0; c < kLocalPlanCtas; ++c) {
                before += c < cta ? v[c] : 0;
                all += v[c];
            }
        }
        const int padded = (all + p.alignment - 1) / p.alignment * p.alignment;
        const int incl = warp_inclusive_sum(padded);
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        const int sums = warp_inclusive_sum(lane < kWarps ? s_warp[lane] : 0);
        const int lower = __shfl_sync(kFull, sums, warp > 0 ? warp - 1 : 0);
        const int off = capacity + (warp > 0 ? lower : 0) + incl - padded;
        if (e < E) {
            s_real[e] = all;
            s_padded[e] = off;
            s_cursor[e] = off + before;
            if (cta == 0) {
                p.expert_counts[e] = all;
                p.expert_offsets[e] = off;
            }
        }
        capacity += __shfl_sync(kFull, sums, 31);
        if (e0 + kLocalPlanThreads < E) __syncthreads();  // s_warp is written again
    }
    if (cta == 0 && tid == 0) {
        p.expert_offsets[E] = capacity;
        p.recv_rank_prefix[0] = s_all;
        p.send_counts[0] = s_all;
    }
    __syncthreads();
    if (warp == 0) {
        __syncwarp();  // everybody's offsets and counts are behind the block barrier above
        // the report of an invalid id reaches the host before the counts do: the call after this one raises it
        if (lane == 0 && cta == 0) publish_counts(p.mailbox, s_all, capacity, p.gated != 0 || s_any_invalid != 0);
    }
    cluster_arrive();  // this CTA has read the others' counts; they may exit once everybody has
    // ---- assign rows and slots
    for (int ch = warp; ch < my_chunks; ch += kWarps) {
        const int tok0 = (first_chunk + ch) * 32;
        const bool has = my_chunks <= kWarps ? kept : load_chunk(first_chunk + ch, false) != 0;  // the buffer still holds the warp's only chunk
        const unsigned hm = __ballot_sync(kFull, has);
        if (!has) continue;
        const int row = s_first + s_rows[ch] + __popc(hm & lanemask_lt());
        int* m = p.meta + int64_t(row) * (K + 2);
        m[0] = 0;
        m[1] = tok0 + lane;
        for (int k0 = 0; k0 < K; k0 += 8) {  // the slots of eight choices are taken before the first is used
            int v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] = k0 + j < K ? mine[lane * K + k0 + j] : -1;
                if (p.expand && v[j] >= 0) v[j] = atomicAdd(&s_cursor[v[j]], 1);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (k0 + j >= K) break;
                if (p.expand && v[j] >= 0) p.slot_map[v[j]] = row * K + k0 + j;
                m[2 + k0 + j] = v[j];
            }
        }
    }
    if (p.expand && p.alignment > 1) {
        // alignment gaps hold no row
        for (int e = cta * kWarps + warp; e < E; e += ctas * kWarps) {
            const int next = e + 1 < E ? s_padded[e + 1] : capacity;
            for (int slot = s_padded[e] + s_real[e] + lane; slot < next; slot += 32) p.slot_map[slot] = -1;
        }
    }
    cluster_wait();
}

// ------------------------------------------------------------------------------------------
// plan (fresh dispatch): every receiver scans the routing all sources wrote into its window, 32 tokens at a time,
// keeps the tokens that chose one of its experts, and assigns a receive row (grouped by source
// rank) and, in the expert-major layout, one slot per local choice.
// ------------------------------------------------------------------------------------------
__device__ void plan_body(const PlanParams& p) {
    extern __shared__ int s_chunk[];  // [warps][32*K]
    const WindowLayout& L = p.c.layout;
    const int R = L.ranks, K = L.topk, Le = L.local_experts;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const int gw = blockIdx.x * wpb + warp, GW = gridDim.x * wpb;
    int* ctrl = ctrl_words(p.c);
    const int* prefix = ctrl + L.ctrl_recv_prefix();
    const int* src_tokens = ctrl + L.ctrl_src_tokens();
    const int* eoff = ctrl + L.ctrl_expert_offsets();
    int* expert_cursor = ctrl + L.ctrl_expert_cursor();
    const int* chunk_prefix = reinterpret_cast<const int*>(window(p.c, p.c.rank) + L.chunks_in_offset + int64_t(p.parity) * L.chunks_in_stride);
    int* meta = reinterpret_cast<int*>(window(p.c, p.c.rank) + L.meta_scratch_offset);
    int* mine = s_chunk + warp * 32 * K;
    const StatusRef status = status_of(p.c);
    const int cps = int((L.max_tokens + 31) / 32);
    const int lo = p.c.rank * Le;
    int* slot_scratch = reinterpret_cast<int*>(window(p.c, p.c.rank) + L.slot_scratch_offset);
    if (p.expand) {
        // alignment gaps of the expert-major layout hold no row
        const int* ecnt = ctrl + L.ctrl_expert_counts();
        for (int l = gw; l < Le; l += GW)
            for (int slot = eoff[l] + ecnt[l] + lane; slot < eoff[l + 1]; slot += 32)
                if (slot < L.slot_scratch_ints) slot_scratch[slot] = -1;
    }

    for (int c = gw; c < R * cps; c += GW) {
        const int s = c / cps, tok0 = (c % cps) * 32;
        const int Ts = src_tokens[s];
        if (tok0 >= Ts) continue;
        const int n_tok = min(32, Ts - tok0);
        const int n = n_tok * K;
        const int* remote = reinterpret_cast<const int*>(window(p.c, p.c.rank) + L.routing_in_offset + int64_t(p.parity) * L.routing_in_stride) +
                            (int64_t(s) * L.max_tokens + tok0) * K;
        __syncwarp();
        for (int base = 0; base < n; base += 256) {
            int v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int i = base + j * 32 + lane;
                v[j] = i < n ? ld_relaxed_sys(remote + i) : -1;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int i = base + j * 32 + lane;
                if (i < n) mine[i] = v[j];
            }
        }
        __syncwarp();
        bool has = false;
        if (lane < n_tok)
            for (int k = 0; k < K; ++k) {
                const int e = mine[lane * K + k];
                has |= (e >= lo && e < lo + Le);
            }
        const unsigned hm = __ballot_sync(kFull, has);
        if (hm == 0) continue;
        // rows of a source are ordered by token: the chunk's first row comes from the prefix the stage kernel built
        const int base_row = chunk_prefix[s * cps + (tok0 >> 5)];
        if (has) {
            const int row = prefix[s] + base_row + __popc(hm & lanemask_lt());
            if (row >= prefix[s + 1]) {
                report(status, kSlotOverflow, uint32_t(row), kTagPlan);
            } else {
                int* m = meta + int64_t(row) * (K + 2);
                m[0] = s;
                m[1] = tok0 + lane;
                // Eight choices at a time: all slot atomics of a group are issued before any result
                // is consumed, so their latencies overlap.
                for (int k0 = 0; k0 < K; k0 += 8) {
                    int le[8], got[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int e = k0 + j < K ? mine[lane * K + k0 + j] : -1;
                        le[j] = (e >= lo && e < lo + Le) ? e - lo : -1;
                        got[j] = (p.expand && le[j] >= 0) ? atomicAdd(&expert_cursor[le[j]], 1) : 0;
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (k0 + j >= K) break;
                        int v = -1;
                        if (le[j] >= 0) {
                            v = p.expand ? eoff[le[j]] + got[j] : le[j];
                            if (p.expand && v >= eoff[le[j] + 1]) {
                                report(status, kSlotOverflow, uint32_t(v), kTagPlan);
                                v = -1;
                            }
                            if (p.expand && v >= 0 && v < L.slot_scratch_ints) slot_scratch[v] = row * K + k0 + j;
                        }
                        m[2 + k0 + j] = v;
                    }
                }
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// Ring of row buffers private to one warp, filled by bulk loads that complete on mbarriers.
// ------------------------------------------------------------------------------------------
struct Ring {
    char* buf;
    uint64_t* bars;
    int stages;
    int64_t pitch;
    uint32_t parity;  // bit s = parity of the next phase to wait for on stage s
    __device__ __forceinline__ char* slot(int i) const { return buf + int64_t(i % stages) * pitch; }
    __device__ __forceinline__ uint64_t* bar(int i) const { return bars + (i % stages); }
    // Wait for the load issued into item i's stage.  Only stages that really received a load may be
    // waited on: the parity advances per completed wait, not per item, so skipped items are harmless.
    __device__ __forceinline__ bool wait(int i, uint64_t timeout_ns) {
        const int s = i % stages;
        bool ok = mbar_wait(bars + s, (parity >> s) & 1u, timeout_ns);
        ok = __all_sync(0xffffffffu, ok);
        parity ^= 1u << s;
        return ok;
    }
};

__device__ __forceinline__ Ring make_ring(char* smem, int warps, int stages, int64_t row_bytes) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t pitch = align_up(row_bytes, 128);
    Ring r;
    r.buf = smem + int64_t(warp) * stages * pitch;
    r.bars = reinterpret_cast<uint64_t*>(smem + int64_t(warps) * stages * pitch) + warp * stages;
    r.stages = stages;
    r.pitch = pitch;
    r.parity = 0;
    if (lane == 0) {
        for (int s = 0; s < stages; ++s) mbar_init(r.bars + s, 1);
        mbar_init_fence();
        fence_proxy_async_smem();
    }
    __syncwarp();
    return r;
}


// Receive rows are stored grouped by source rank.  Walking them in storage order would make every
// receiver talk to the same source at the same time (one GPU's NVLink port serving all others).
// Instead item v visits the sources round-robin, starting after the own rank:
//   source s = (rank + 1 + v % R) % R,  j = v / R,  row = first_row(s) + j   (skipped when j >= rows(s)).
struct SourceWalk {
    int first, count;  // lane s: first receive row and row count of source s
    int items;         // R * max_s count
    int rank, ranks;
    __device__ __forceinline__ bool locate(int v, int& row) const {
        const int s = (rank + 1 + v % ranks) % ranks;
        const int j = v / ranks;
        const int f = __shfl_sync(0xffffffffu, first, s);
        const int c = __shfl_sync(0xffffffffu, count, s);
        row = f + j;
        return j < c;
    }
};
__device__ __forceinline__ SourceWalk make_walk(const int64_t* inclusive_prefix, int rank, int ranks) {
    const int lane = threadIdx.x & 31;
    SourceWalk w;
    const int incl = lane < ranks ? int(inclusive_prefix[lane]) : 0;
    const int prev = lane > 0 && lane < ranks ? int(inclusive_prefix[lane - 1]) : 0;
    w.first = prev;
    w.count = lane < ranks ? incl - prev : 0;
    int mx = w.count;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    w.items = mx * ranks;
    w.rank = rank;
    w.ranks = ranks;
    return w;
}

// ------------------------------------------------------------------------------------------
// pull: for every receive row, bulk-load the staged row from its source rank (NVLink or local)
// into shared memory and bulk-store it to its final place(s): row r (compact) or every
// expert-major slot of the row (expanded).  Gaps of the expert-major layout are zero-filled here.
// ------------------------------------------------------------------------------------------
__device__ void pull_body(const PullParams& p) {
    extern __shared__ __align__(128) char s_ring[];
    const WindowLayout& L = p.c.layout;
    const int R = L.ranks, K = L.topk, H = L.hidden, Le = L.local_experts;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    // neighbouring rows go to different SMs: 32 rows to eight slots each leave through 32 of them instead of 7 (12.5 -> 5.2 us,
    // 64 rows 18.3 -> 11.3, 4096 rows 131-136 -> 129)
    const int gw = warp * gridDim.x + blockIdx.x, GW = gridDim.x * wpb;
    const int64_t rb = L.row_bytes();
    const StatusRef status = status_of(p.c);
    const int MW = K + 2;
    Ring ring = make_ring(s_ring, wpb, p.stages, rb);
    const int S = p.stages;
    wait_for_previous();
    if (p.dependents) allow_dependents();  // behind the wait: what a dependent reads before its own has been written by then (offsets, counts)
    if (p.data_epoch != 0) {
        // A fresh dispatch stages its rows underneath the count exchange: every source signals when its rows are in place.
        __shared__ int s_staged;
        if (warp == 0) {
            const bool ok = peer_wait_warp(p.c.peers, p.c.rank, R, L.data_signal_offset, p.data_epoch, p.c.timeout_ns, status, kTagPull);
            if (lane == 0) s_staged = ok;
        }
        __syncthreads();
        if (!s_staged) return;
        fence_proxy_async();
    }
    const SourceWalk walk = make_walk(p.recv_rank_prefix, p.c.rank, R);
    const bool slot_order = p.slot_src != nullptr;
    const int n_items = slot_order ? p.capacity : walk.items;
    const int n_my = n_items > gw ? (n_items - gw + GW - 1) / GW : 0;
    // The metadata of an item is requested three items before its turn and stays in registers (lane j holds word j, and
    // word 32 + j of a row with more choices than that): neither the load of a row nor its stores wait for it.  With one rank
    // and hidden 7168, 4096 tokens 134 -> 131 us, 1 token 5.8 -> 4.7; eight logical ranks of 512 tokens 171 -> 166 us.
    struct Item {
        int r, a, b;
        bool live;
    };
    auto fetch = [&](int i) {
        Item w{0, -1, -1, false};
        if (i < n_my) {
            const int item = gw + i * GW;
            if (!slot_order) {
                w.live = walk.locate(item, w.r);
            } else {
                const int slot = p.slot_src[item];
                w.live = slot >= 0;
                w.r = slot >= 0 ? slot / K : 0;
            }
            if (w.live) {
                const int* m = p.meta + int64_t(w.r) * MW;
                if (lane < MW) w.a = m[lane];
                if (lane + 32 < MW) w.b = m[lane + 32];
            }
        }
        return w;
    };
    // lane k: choice k of the item's row
    auto choice = [&](const Item& w) {
        int v = __shfl_sync(kFull, w.a, (lane + 2) & 31);
        if (MW > 32) {
            const int high = __shfl_sync(kFull, w.b, (lane + 2) & 31);
            if (lane >= 30) v = high;
        }
        return lane < K ? v : -1;
    };
    // false: nothing to transfer for this item (in slot order a row goes with the lowest of its slots)
    auto has_row = [&](int i, const Item& w) {
        if (!slot_order || !w.live) return w.live;
        const int v = choice(w);
        int lowest = v >= 0 ? v : 0x7fffffff;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) lowest = min(lowest, __shfl_xor_sync(kFull, lowest, d));
        return lowest == gw + i * GW;
    };

    auto issue = [&](int i, const Item& w) {
        if (!has_row(i, w)) return;
        int src = __shfl_sync(kFull, w.a, 0), tok = __shfl_sync(kFull, w.a, 1);
        if (lane == 0) {
            if (src < 0 || src >= R || tok < 0 || tok >= L.max_tokens) {
                report(status, kBadMetadata, uint32_t(w.r), kTagPull);
                src = p.c.rank;
                tok = 0;
            }
            if (src == p.c.rank && p.x_local != nullptr) {
                mbar_expect_tx(ring.bar(i), uint32_t(H) * 2u);
                bulk_load(ring.slot(i), p.x_local + int64_t(tok) * H, uint32_t(H) * 2u, ring.bar(i));
            } else {
                const char* from = window(p.c, src) + L.stage_rows_offset + int64_t(p.parity) * L.stage_rows_stride + int64_t(tok) * rb;
                mbar_expect_tx(ring.bar(i), uint32_t(rb));
                bulk_load(ring.slot(i), from, uint32_t(rb), ring.bar(i));
            }
        }
    };
    constexpr int kAhead = 3;  // most stages of a ring
    Item queue[kAhead + 1];    // items i .. i + 3
#pragma unroll
    for (int i = 0; i < kAhead; ++i) queue[i] = fetch(i);
#pragma unroll
    for (int i = 0; i < kAhead - 1; ++i)
        if (i < min(S - 1, n_my)) issue(i, queue[i]);

    // Gaps between an expert's last real row and the next expert's first slot: zero rows are bulk
    // stores from a zero buffer behind the rings (few instructions, no LSU store traffic).
    char* zero_buf = s_ring + (align_up(rb, 128) + 8) * int64_t(wpb) * S;
    zero_buf = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(zero_buf) + 127) & ~uintptr_t(127));
    if (p.expand && p.zero_padding) {
        for (int i = threadIdx.x; i < p.zero_bytes / 16; i += blockDim.x) reinterpret_cast<int4*>(zero_buf)[i] = make_int4(0, 0, 0, 0);
        fence_proxy_async_smem();
        __syncthreads();
    }
    if (p.expand && (p.zero_padding || p.slot_map != nullptr)) {
        // Gap rows are dealt out over the warps without a walk over the experts: a lane reads the geometry of
        // kGapWaves experts at once, a warp scan of the gap lengths numbers the gap rows of 32 experts, and a ballot
        // finds the expert that owns a number.  (A scalar walk over 256 experts took 45 us of every warp's time, which
        // was all of a one-token dispatch and ran ahead of the rows in a large one.)
        constexpr int kGapWaves = 8;
        int base = 0;  // gap rows of the experts before this wave, modulo the number of warps
        for (int l0 = 0; l0 < Le; l0 += 32 * kGapWaves) {
            int start[kGapWaves], len[kGapWaves];
#pragma unroll
            for (int u = 0; u < kGapWaves; ++u) {
                const int l = l0 + 32 * u + lane;
                start[u] = l < Le ? int(p.expert_offsets[l] + p.expert_counts[l]) : 0;
                len[u] = l < Le ? int(p.expert_offsets[l + 1]) - start[u] : 0;
            }
#pragma unroll
            for (int u = 0; u < kGapWaves; ++u) {
                if (!__any_sync(kFull, len[u] > 0)) continue;
                const int incl = warp_inclusive_sum(len[u]);
                const int total = __shfl_sync(kFull, incl, 31);
                for (int j = gw >= base ? gw - base : gw - base + GW; j < total; j += GW) {
                    const int owner = __ffs(__ballot_sync(kFull, incl > j)) - 1;
                    const int64_t row = __shfl_sync(kFull, start[u] + len[u] - incl, owner) + j;
                    if (p.zero_padding) {
                        if (lane == 0) {
                            char* dst = reinterpret_cast<char*>(p.x_out + row * H);
                            for (int at = 0; at < H * 2; at += p.zero_bytes) bulk_store(dst + at, zero_buf, uint32_t(min(p.zero_bytes, H * 2 - at)));
                            bulk_commit();
                            if (p.w_out != nullptr) p.w_out[row] = 0.f;
                        }
                        if (p.tile_ready != nullptr) bulk_wait<0>();
                    }
                    if (lane == 0 && p.slot_map != nullptr) p.slot_map[row] = -1;
                    if (p.tile_ready != nullptr) {
                        fence_proxy_async();
                        __threadfence();
                        __syncwarp();
                        if (lane == 0) red_release_gpu_add(p.tile_ready + int(row / 128), 1);
                    }
                }
                base = (base + total) % GW;
            }
        }
    }

    // With tile counters, a row is announced one iteration late: after the bulk group that stored it
    // has fully completed (not only been read from shared memory).
    const bool announce = p.tile_ready != nullptr && p.expand;
    int announced_slot = -1;
    auto retire_previous = [&]() {
        if (announce) {
            bulk_wait<1>();
            if (announced_slot >= 0) {
                fence_proxy_async();
                red_release_gpu_add(p.tile_ready + announced_slot / 128, 1);
            }
        } else {
            bulk_wait_read<1>();
        }
    };
    for (int i = 0; i < n_my; ++i) {
        queue[kAhead] = fetch(i + kAhead);
        const Item now = queue[0];
        int stored = -1;
        if (has_row(i, now)) {
            if (!ring.wait(i, p.c.timeout_ns)) {
                if (lane == 0) report(status, kCopyTimeout, uint32_t(gw), kTagPull);
                break;
            }
            const int r = now.r, v = choice(now);
            const char* st = ring.slot(i);
            const float* st_w = reinterpret_cast<const float*>(st + wire_weights_offset(H));
            const int src = __shfl_sync(kFull, now.a, 0), tok = __shfl_sync(kFull, now.a, 1);
            if (src == p.c.rank && p.x_local != nullptr && p.w_local != nullptr) st_w = p.w_local + int64_t(tok) * K;
            if (p.expand) {
                if (v >= 0) {
                    bulk_store(p.x_out + int64_t(v) * H, st, uint32_t(H) * 2u);
                    if (p.w_out != nullptr) p.w_out[v] = st_w[lane];
                    if (p.slot_map != nullptr) p.slot_map[v] = r * K + lane;
                }
                stored = v;
            } else {
                if (lane == 0) bulk_store(p.x_out + int64_t(r) * H, st, uint32_t(H) * 2u);
                if (lane < K) {
                    p.topk_out[int64_t(r) * K + lane] = v;
                    if (p.w_out != nullptr) p.w_out[int64_t(r) * K + lane] = st_w[lane];
                }
            }
            if (p.write_meta) {
                if (lane < MW) p.meta_out[int64_t(r) * MW + lane] = now.a;
                if (lane + 32 < MW) p.meta_out[int64_t(r) * MW + lane + 32] = now.b;
            }
        }
        bulk_commit();
        retire_previous();
        announced_slot = stored;
        __syncwarp();
        if (i + S - 1 < n_my) issue(i + S - 1, S == kAhead ? queue[kAhead - 1] : queue[1]);
#pragma unroll
        for (int j = 0; j < kAhead; ++j) queue[j] = queue[j + 1];
    }
    bulk_wait<0>();
    if (announce && announced_slot >= 0) {
        fence_proxy_async();
        red_release_gpu_add(p.tile_ready + announced_slot / 128, 1);
    }
}

// ------------------------------------------------------------------------------------------
// combine: one launch.  Transfer warps return expert outputs to the source ranks' partitions and flag every
// row on arrival; reduce warps sum a source token once all of its rows are flagged.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ char* ret_row(const CommonParams& c, int src, int part, int tok) {
    const WindowLayout& L = c.layout;
    return window(c, src) + L.ret_offset + (int64_t(part) * L.max_tokens + tok) * L.hidden * 2;
}
__device__ __forceinline__ float* ret_w_row(const CommonParams& c, int src, int tok) {
    const WindowLayout& L = c.layout;
    return reinterpret_cast<float*>(window(c, src) + L.ret_w_offset) + int64_t(tok) * L.topk;
}
__device__ __forceinline__ uint32_t* ret_flag(const CommonParams& c, int src, int part, int tok) {
    const WindowLayout& L = c.layout;
    return reinterpret_cast<uint32_t*>(window(c, src) + L.ret_flag_offset) + int64_t(part) * L.max_tokens + tok;
}
// Value a combine writes into the arrival flags: never 0 (a fresh window), different for consecutive combines.
__device__ __forceinline__ uint32_t combine_tag(uint64_t epoch) { return uint32_t(epoch % 0xffffffffull) + 1u; }

__device__ __forceinline__ void accumulate8(float* acc, const int4& v) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        acc[2 * j] += f.x;
        acc[2 * j + 1] += f.y;
    }
}
__device__ __forceinline__ int4 pack8(const float* acc) {
    int4 v;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
    return v;
}

// Arrival flags are published by a dedicated warp, not by the transfer warps: a flag needs a system-scope
// release after its row has landed, and that fence waits for remote stores in flight.  A transfer warp only
// appends the flag's address to its ring on this board and reports how many of its bulk stores have COMPLETED
// (cp.async.bulk.wait_group, not .read; up to a FlagQueue's depth may be pending).  The publisher warp sweeps the
// boards, fences once per sweep and writes the flags of everything that completed since its last sweep.
constexpr int kMaxPushWarps = 8;
__device__ __forceinline__ void bulk_wait_depth(int depth) {
    switch (depth) {
        case 4: bulk_wait<4>(); break;
        case 6: bulk_wait<6>(); break;
        case 8: bulk_wait<8>(); break;
        case kMaxStoreDepth: bulk_wait<kMaxStoreDepth>(); break;
        default: bulk_wait<2>(); break;
    }
}
struct FlagBoard {
    uint32_t* ring[kMaxPushWarps][kFlagRing];
    int completed[kMaxPushWarps];  // transfers whose rows have landed (written by the transfer warp, release)
    int published[kMaxPushWarps];  // transfers whose flags are out (written by the publisher)
    int finished[kMaxPushWarps];   // the transfer warp has no more work
};

// A transfer warp's end of the board, under a FlagQueue (all lanes hold the same values, except `kept`).
struct FlagWriter {
    FlagBoard* board;
    int warp;
    uint64_t timeout_ns;
    StatusRef status;
    int kept = 0;  // lane i: mark i
    __device__ __forceinline__ void append(uint32_t* flag, int at) {
        if ((threadIdx.x & 31) == 0) {
            volatile int* published = board->published + warp;
            if (at - *published >= kFlagRing) {  // ring full: the publisher is behind (bounded wait)
                const uint64_t start = global_timer_ns();
                while (at - *published >= kFlagRing && global_timer_ns() - start < timeout_ns) __nanosleep(64);
            }
            if (at - *published < kFlagRing)
                board->ring[warp][at % kFlagRing] = flag;
            else  // the entry still holds a flag that has to go out
                report(status, kCopyTimeout, uint32_t(warp), kTagPush);
        }
    }
    __device__ __forceinline__ void set_mark(int i, int count) {
        if ((threadIdx.x & 31) == i) kept = count;
    }
    __device__ __forceinline__ int mark(int i) const { return __shfl_sync(kFull, kept, i); }
    __device__ __forceinline__ void wait_landed(int depth) {
        if (depth == 0) {
            bulk_wait<0>();
        } else {
            bulk_wait_read<1>();  // the ring stage of the previous row may be refilled
            bulk_wait_depth(depth);
        }
        __syncwarp();  // by any lane; and other lanes' stores are ordered before a hand-over
    }
    __device__ __forceinline__ void publish_up_to(int count) {
        if ((threadIdx.x & 31) == 0) st_release_cta_smem(board->completed + warp, count);
    }
    __device__ __forceinline__ void no_more() {
        if ((threadIdx.x & 31) == 0) st_release_cta_smem(board->finished + warp, 1);
    }
};

// The publisher warp of a combine CTA.
__device__ void combine_publish_role(const CombineParams& p, FlagBoard* board) {
    const int lane = threadIdx.x & 31, PW = p.push_warps;
    const uint32_t tag = combine_tag(p.epoch);
    int pub = 0;  // lane w < PW: flags of transfer warp w published so far
    const uint64_t start = global_timer_ns();
    for (;;) {
        const int fin = lane < PW ? ld_acquire_cta_smem(board->finished + lane) : 1;
        const int done = lane < PW ? ld_acquire_cta_smem(board->completed + lane) : 0;
        const unsigned fresh = __ballot_sync(kFull, lane < PW && done > pub);
        if (fresh != 0) {
            fence_acq_rel_sys();  // one release for everything that landed since the last sweep
            for (unsigned left = fresh; left != 0; left &= left - 1) {
                const int w = __ffs(left) - 1;
                const int from = __shfl_sync(kFull, pub, w), to = __shfl_sync(kFull, done, w);
                for (int i = from + lane; i < to; i += 32) st_relaxed_sys_u32(board->ring[w][i % kFlagRing], tag);
            }
            __syncwarp();  // every ring entry has been read before its slot is handed back
            if (lane < PW && done > pub) {
                pub = done;
                *(volatile int*)(board->published + lane) = pub;
            }
        }
        if (__all_sync(kFull, fin != 0 && pub == done)) break;
        if (fresh == 0) {
            __nanosleep(200);
            if (global_timer_ns() - start > 4 * p.c.timeout_ns) {  // transfer warps give up long before this
                if (lane == 0) report(status_of(p.c), kCopyTimeout, 0xfffeu, kTagPush);
                break;
            }
        }
    }
}

// Whether the rows of a rank's own tokens stay in the expert output for the reduction to read: in the modes that return rows as they
// are, and with the reduction that takes rows from anywhere (the loader of combine_reduce_smem_role bulk-loads them into its ring).
// Eight ranks of 512 tokens on one GPU: combine 238 -> 228 us (one row in eight is a rank's own: its copy was 2 x 59 MB through L2 and
// 59 MB to memory); four ranks of 1000 skewed tokens 94 -> 92.
__device__ __forceinline__ bool own_rows_in_place(const CombineParams& p) { return p.reduce_stages >= 2 && p.mode != kPushExpandedReduce; }

// Transfer warps.  Receive rows are visited round-robin over the source ranks (SourceWalk), so at every moment
// the warps of a GPU address all destinations evenly; a row of the expert-major layout yields one transfer per
// local slot.
__device__ void combine_push_role(const CombineParams& p, char* smem, FlagBoard* board) {
    const WindowLayout& L = p.c.layout;
    const int R = L.ranks, K = L.topk, H = L.hidden;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, PW = p.push_warps;
    const int gw = blockIdx.x * PW + warp;
    const StatusRef status = status_of(p.c);
    const int MW = K + 2;
    const uint32_t xb = uint32_t(H) * 2u;
    Ring ring = make_ring(smem, PW, p.stages, xb);
    const int S = p.stages;
    const SourceWalk walk = make_walk(p.recv_rank_prefix, p.c.rank, R);
    // The walk is shared by all transfer warps of the rank: a warp takes the next position from one counter when it
    // needs work (the request for the position after that is already in flight).  Rows differ in how many transfers
    // they need (0 to K local slots), so equal shares of rows leave the warps with the most slots working alone at
    // the end; with a shared position all warps end within one row of each other and rows leave in walk order
    // (measured at 2 GPUs and 4096 tokens per rank: the transfer warps end 8 us earlier).
    int* work = ctrl_words(p.c) + WindowLayout::kWorkCursor;
    int claimed = 0;  // lane 0: the position requested last
    auto request = [&]() {
        if (lane == 0) claimed = atomicAdd(work, 1);
    };
    auto take = [&]() {  // the requested position, on every lane; requests the one after it
        const int v = __shfl_sync(kFull, claimed, 0);
        if (v < walk.items) request();
        return v;
    };
    request();
    const int depth = (p.store_depth == 4 || p.store_depth == 6 || p.store_depth == 8 || p.store_depth == kMaxStoreDepth) ? p.store_depth : 2;
    FlagQueue<FlagWriter, uint32_t*> flags{FlagWriter{board, warp, p.c.timeout_ns, status}, depth};

    if (p.mode == kPushExpandedReduce) {
        // FP32 sum of the row's local slots, one bf16 round, one store per (token, this rank).
        const int vecs = H / 8;
        int q = 0;  // rows sent so far: consecutive rows use consecutive ring stages
        for (;;) {
            const int item = take();
            if (item >= walk.items) break;
            int r;
            const bool live_row = walk.locate(item, r);
            const int* m = p.meta + int64_t(live_row ? r : 0) * MW;
            const int v = (live_row && lane < K) ? m[2 + lane] : -1;
            const unsigned vm = __ballot_sync(kFull, v >= 0 && v < p.capacity);
            const int src = m[0], tok = m[1];
            bool fine = live_row && vm != 0;
            if (fine && (src < 0 || src >= R || tok < 0 || tok >= L.max_tokens || __any_sync(kFull, v >= p.capacity))) {
                if (lane == 0) report(status, kBadMetadata, uint32_t(r), kTagPush);
                fine = false;
            }
            if (!fine) continue;
            char* st = ring.slot(q++);
            // four 16-byte column chunks x two slots per step: eight independent loads per lane in flight
            for (int c0 = lane; c0 < vecs; c0 += 128) {
                float acc[4][8];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[u][j] = 0.f;
                unsigned left = vm;
                while (left) {
                    const int k0 = __ffs(left) - 1;
                    left &= left - 1;
                    const int k1 = left ? __ffs(left) - 1 : -1;
                    if (left) left &= left - 1;
                    const int slot0 = __shfl_sync(kFull, v, k0);
                    const int slot1 = __shfl_sync(kFull, v, k1 < 0 ? 0 : k1);
                    const int4* r0 = reinterpret_cast<const int4*>(p.y + int64_t(slot0) * H);
                    const int4* r1 = reinterpret_cast<const int4*>(p.y + int64_t(slot1) * H);
                    int4 d0[4], d1[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (c0 + 32 * u < vecs) {
                            d0[u] = ld_nc_v4(r0 + c0 + 32 * u);
                            if (k1 >= 0) d1[u] = ld_nc_v4(r1 + c0 + 32 * u);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (c0 + 32 * u < vecs) {
                            accumulate8(acc[u], d0[u]);
                            if (k1 >= 0) accumulate8(acc[u], d1[u]);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (c0 + 32 * u < vecs) reinterpret_cast<int4*>(st)[c0 + 32 * u] = pack8(acc[u]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            const int part = L.rank_indexed ? p.c.rank : __ffs(vm) - 1;
            if (lane == 0) bulk_store(ret_row(p.c, src, part, tok), st, xb);
            if (p.w != nullptr && ((vm >> lane) & 1u)) st_relaxed_sys_f32(ret_w_row(p.c, src, tok) + lane, p.w[v]);
            bulk_commit();
            flags.push(ret_flag(p.c, src, part, tok));
        }
        flags.finish();
        flags.io.no_more();
        return;
    }

    // One bulk load + one bulk store per transfer.  A cursor enumerates the transfers of this warp's rows:
    // compact layout = one per receive row; expert-major layout = one per local slot of the row.
    // Rows of this rank's own tokens are not transferred where the reduction can read them in place (own_rows_in_place).
    const bool by_slot = p.mode == kPushExpanded, direct = own_rows_in_place(p);
    struct Cursor {
        unsigned left;  // choices of the current row that still need a transfer
        unsigned vm;    // all valid choices of the current row
        int r, v, src, tok, k;
    };
    // The loads run ahead of the stores over the same sequence of rows: the leading cursor takes positions from the
    // shared counter and queues the live ones (lane n % 32 keeps the n-th), the trailing cursor reads them back.
    int queued = 0, q_head = 0, q_tail = 0;
    auto next = [&](Cursor& c, bool leading) {
        while (c.left == 0) {
            int r;
            if (leading) {
                const int item = take();
                if (item >= walk.items) return false;
                if (!walk.locate(item, r)) continue;
            } else {
                if (q_tail == q_head) return false;
                r = __shfl_sync(kFull, queued, q_tail & 31);
                ++q_tail;
            }
            const int* m = p.meta + int64_t(r) * MW;
            c.r = r;
            c.src = m[0];
            c.tok = m[1];
            c.v = lane < K ? m[2 + lane] : -1;
            c.vm = __ballot_sync(kFull, c.v >= 0);
            const bool bad_slot = __any_sync(kFull, by_slot && c.v >= p.capacity);
            if (c.src < 0 || c.src >= R || c.tok < 0 || c.tok >= L.max_tokens || bad_slot) {
                if (lane == 0) report(status, kBadMetadata, uint32_t(r), kTagPush);
                c.vm = 0;
            }
            c.left = by_slot ? c.vm : (c.vm & (0u - c.vm));  // compact: the first valid choice names the partition
            if (!leading) continue;
            if (direct && c.src == p.c.rank) {
                // The row stays where it is: its place in the return area takes its index, and the reduction reads the row itself.
                const int part = L.rank_indexed ? p.c.rank : lane;
                if ((c.left >> lane) & 1u) *reinterpret_cast<int*>(ret_row(p.c, c.src, part, c.tok)) = by_slot ? c.v : c.r;
                if (p.w != nullptr && ((c.vm >> lane) & 1u))
                    st_relaxed_sys_f32(ret_w_row(p.c, c.src, c.tok) + lane, by_slot ? p.w[c.v] : p.w[int64_t(c.r) * K + lane]);
                for (; c.left != 0; c.left &= c.left - 1) flags.note(ret_flag(p.c, c.src, __shfl_sync(kFull, part, __ffs(c.left) - 1), c.tok));
                continue;
            }
            if (lane == (q_head & 31)) queued = r;
            ++q_head;
        }
        c.k = __ffs(c.left) - 1;
        c.left &= c.left - 1;
        return true;
    };
    const uint64_t once = l2_evict_first_policy();  // expert rows are read exactly once: keep L2 for the return rows
    auto issue = [&](const Cursor& c, int q) {
        const int y_row = by_slot ? __shfl_sync(kFull, c.v, c.k) : c.r;
        if (lane == 0) {
            mbar_expect_tx(ring.bar(q), xb);
            bulk_load_hint(ring.slot(q), p.y + int64_t(y_row) * H, xb, ring.bar(q), once);
        }
    };
    Cursor ahead{0u, 0u, 0, -1, 0, 0, 0}, now{0u, 0u, 0, -1, 0, 0, 0};
    int issued = 0;
    bool more = true;
    while (issued < S - 1 && (more = next(ahead, true))) issue(ahead, issued++);
    for (int q = 0; next(now, false); ++q) {
        if (!ring.wait(q, p.c.timeout_ns)) {
            if (lane == 0) report(status, kCopyTimeout, uint32_t(gw), kTagPush);
            break;
        }
        const int part = by_slot ? now.k : (L.rank_indexed ? p.c.rank : now.k);
        if (lane == 0) bulk_store(ret_row(p.c, now.src, part, now.tok), ring.slot(q), xb);
        if (p.w != nullptr) {
            if (by_slot) {
                const int slot = __shfl_sync(kFull, now.v, now.k);
                if (lane == 0) st_relaxed_sys_f32(ret_w_row(p.c, now.src, now.tok) + now.k, p.w[slot]);
            } else if ((now.vm >> lane) & 1u) {
                st_relaxed_sys_f32(ret_w_row(p.c, now.src, now.tok) + lane, p.w[int64_t(now.r) * K + lane]);
            }
        }
        bulk_commit();
        flags.push(ret_flag(p.c, now.src, part, now.tok));
        if (more && (more = next(ahead, true))) issue(ahead, issued++);
    }
    flags.finish();
    flags.io.no_more();
}

// Which return partitions hold a row for source token `t`, as a mask over the lanes (choices) that name them;
// `valid` is the lane's own choice.  One partition per valid choice, or one per destination rank (named by
// the rank's first choice).
__device__ __forceinline__ unsigned expected_parts(const int64_t* topk, int t, int K, int E, int Le, bool sum_all_choices, bool& valid,
                                                   int& dest) {
    const int lane = threadIdx.x & 31;
    const int64_t e = lane < K ? topk[int64_t(t) * K + lane] : -1;
    valid = e >= 0 && e < E;
    dest = valid ? int(e) / Le : -1;
    const unsigned vmask = __ballot_sync(kFull, valid);
    if (sum_all_choices) return vmask;
    bool leader = false;
    if (valid) {
        const unsigned same = __match_any_sync(vmask, dest);
        leader = lane == __ffs(same) - 1;
    }
    return __ballot_sync(kFull, leader);
}

// FP32 sum of the partitions in `parts` for the 16-byte column chunks `first`, `first + step`, ... of token t.
// All partitions of a chunk are loaded before any is added, two chunks at a time.
__device__ __forceinline__ void reduce_columns(const CommonParams& c, int t, unsigned parts, int my_part, const __nv_bfloat16* bias,
                                               __nv_bfloat16* out, int first_base, int step, uint64_t once) {
    const WindowLayout& L = c.layout;
    const int H = L.hidden, lane = threadIdx.x & 31;
    const int vecs = H / 8;
    const int64_t part_stride = L.max_tokens * int64_t(H) * 2;
    const char* row0 = window(c, c.rank) + L.ret_offset + int64_t(t) * H * 2;
    // `base` is the same for every lane of the warp (the loop holds warp shuffles); lanes past the row's end idle
    for (int base = first_base; base < vecs; base += 2 * step) {
        const int col = base + lane;
        const bool one = col < vecs, two = col + step < vecs;
        float a0[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float a1[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        unsigned left = parts;
        while (left) {
            int part[8];
            int4 d0[8], d1[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int k = left ? __ffs(left) - 1 : -1;
                if (left) left &= left - 1;
                part[j] = __shfl_sync(kFull, my_part, k < 0 ? 0 : k);
                if (k < 0) part[j] = -1;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (part[j] >= 0) {
                    const int4* src = reinterpret_cast<const int4*>(row0 + part[j] * part_stride);
                    if (one) d0[j] = ld_cg_v4_hint(src + col, once);
                    if (two) d1[j] = ld_cg_v4_hint(src + col + step, once);
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (part[j] >= 0) {
                    if (one) accumulate8(a0, d0[j]);
                    if (two) accumulate8(a1, d1[j]);
                }
            }
        }
        if (bias != nullptr) {
            const int4* b = reinterpret_cast<const int4*>(bias + int64_t(t) * H);
            if (one) accumulate8(a0, ld_nc_v4(b + col));
            if (two) accumulate8(a1, ld_nc_v4(b + col + step));
        }
        int4* o = reinterpret_cast<int4*>(out + int64_t(t) * H);
        if (one) st_v4_hint(o + col, pack8(a0), once);
        if (two) st_v4_hint(o + col + step, pack8(a1), once);
    }
}

constexpr int kReduceFlowWords = 2 + 2 * (kCombineThreads / 32 + 1);

// Reduce warps of the combine kernel.  They form groups of `reduce_group` warps; a group sums ONE source token at a
// time, each lane its own column chunks.  The group's first warp waits (bounded) until every partition the token
// expects carries this combine's tag and releases the others through the group's named barrier.
//
// How long one token takes decides how long the kernel runs after the last row has landed: under the load of the
// transfers a group of two warps needs ~30 us per token (seven dependent batches of loads at ~4 us each), five warps
// ~13 us, all ten ~9 us - but larger groups hold fewer tokens at a time and fall behind the arrivals, and handing only
// the last tokens of a CTA to all of its warps measured slower as well (they are summed one after the other).
//
// `flow` is a small shared array: [0] the CTA's abort word (sticky), then two go/stop words per group.  The warp that waited writes "go" or "stop" into the word of the barrier's
// parity BEFORE the barrier and everybody reads it AFTER the barrier, so all warps of a barrier take the same branch
// (reading the sticky abort word instead would let two warps of one barrier see different values and strand one of
// them at the next barrier, which has no time limit).
__device__ void combine_reduce_role(const CombineParams& p, int* flow) {
    int* abort_word = flow;
    const WindowLayout& L = p.c.layout;
    const int K = L.topk, Le = L.local_experts, E = int(L.num_experts);
    const int lane = threadIdx.x & 31;
    const int RW = (blockDim.x >> 5) - p.push_warps - 1;  // one warp publishes flags
    const int rwarp = (threadIdx.x >> 5) - p.push_warps - 1;
    const int G = p.reduce_group < 1 ? 1 : (p.reduce_group > RW ? RW : p.reduce_group);
    const int groups = RW / G, g = rwarp / G, wi = rwarp % G;
    const StatusRef status = status_of(p.c);
    const uint32_t tag = combine_tag(p.epoch);
    const uint32_t* flag_base = reinterpret_cast<const uint32_t*>(window(p.c, p.c.rank) + L.ret_flag_offset);
    const float* ret_w = reinterpret_cast<const float*>(window(p.c, p.c.rank) + L.ret_w_offset);
    // returned rows are read once and the result is written once: both leave L2 first
    const uint64_t once = l2_evict_first_policy();
    unsigned waited = 0, worked = 0, longest = 0, summed = 0;  // nanoseconds (a kernel runs far below four seconds)
    unsigned long long longest_at = 0, last_seen = 0;

    // One warp waits for the token's rows (bounded); on a timeout it reports and raises the CTA's abort word.
    auto await_rows = [&](int t, unsigned parts, int my_part) -> bool {
        const bool mine = (parts >> lane) & 1u;
        const uint32_t* flag = flag_base + int64_t(mine ? my_part : 0) * L.max_tokens + t;
        const uint64_t start = global_timer_ns();
        uint32_t spins = 0;
        bool arrived = false;
        for (;;) {
            const bool here = !mine || ld_relaxed_sys_u32(flag) == tag;
            arrived = __all_sync(kFull, here);
            if (arrived) break;
            __nanosleep(200);
            if ((++spins & 15u) == 0u && __any_sync(kFull, global_timer_ns() - start > p.c.timeout_ns)) break;
        }
        // the polls were relaxed; one acquiring load of each flag orders the rows behind them
        if (arrived && mine) (void)ld_acquire_sys_u32(flag);
        __syncwarp();
        if (!arrived && lane == 0) {
            report(status, kBarrierTimeout, uint32_t(t), kTagReduce);
            *(volatile int*)abort_word = 1;  // a peer never delivered: stop reducing, the host reports the status
        }
        return arrived;
    };
    auto sum_token = [&](int t, unsigned parts, int my_part, bool valid, bool first_warp, int first_base, int step, uint64_t t_wait) {
        const uint64_t t_work = p.trace != nullptr ? global_timer_ns() : 0;
        reduce_columns(p.c, t, parts, my_part, p.bias, p.out, first_base, step, once);
        if (first_warp && p.w_out != nullptr && lane < K) p.w_out[int64_t(t) * K + lane] = valid ? __ldcg(ret_w + int64_t(t) * K + lane) : 0.f;
        if (p.trace != nullptr) {
            const uint64_t t_done = global_timer_ns();
            waited += unsigned(t_work - t_wait);
            worked += unsigned(t_done - t_work);
            if (unsigned(t_done - t_work) > longest) {
                longest = unsigned(t_done - t_work);
                longest_at = t_work;
            }
            last_seen = t_work;
            ++summed;
        }
    };

    // warps that do not fill a group sit out
    if (g < groups) {
        int* go = flow + 2 + 2 * g;
        unsigned syncs = 0;
        for (int t = blockIdx.x * groups + g; t < p.tokens; t += gridDim.x * groups) {
            bool valid;
            int dest;
            const unsigned parts = expected_parts(p.topk, t, K, E, Le, p.sum_all_choices != 0, valid, dest);
            const int my_part = L.rank_indexed ? dest : lane;
            const uint64_t t_wait = p.trace != nullptr ? global_timer_ns() : 0;
            if (parts != 0) {
                bool ok = true;
                if (wi == 0) {
                    ok = !*(volatile int*)abort_word && await_rows(t, parts, my_part);
                    if (G > 1 && lane == 0) *(volatile int*)(go + (syncs & 1u)) = ok;
                }
                if (G > 1) {
                    // named barrier 1 + g: this group's reduce warps only
                    asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(G * 32) : "memory");
                    ok = *(volatile int*)(go + (syncs & 1u)) != 0;
                    ++syncs;
                }
                if (!ok) break;
            }
            sum_token(t, parts, my_part, valid, wi == 0, wi * 32, G * 32, t_wait);
        }
    }
    if (p.trace != nullptr && (rwarp % G) == 0 && lane == 0) {
        atomicAdd(p.trace + 4, (unsigned long long)waited);
        atomicAdd(p.trace + 5, (unsigned long long)worked);
        atomicAdd(p.trace + 6, (unsigned long long)summed);
        const unsigned long long t0 = *(volatile unsigned long long*)p.trace;
        atomicMax(p.trace + 7, ((unsigned long long)longest << 32) | (unsigned long long)unsigned(longest_at - t0));
        atomicMax(p.trace + 8, last_seen);
    }
}

// Bounded mbarrier wait of the reduce pipeline: also gives up as soon as the CTA's abort word is raised.
__device__ __forceinline__ bool mbar_wait_or_abort(uint64_t* bar, uint32_t parity, uint64_t timeout_ns, const int* abort_word) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t start = global_timer_ns();
    uint32_t spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++spins & 63u) == 0u && (*(volatile const int*)abort_word != 0 || global_timer_ns() - start > timeout_ns)) return false;
    }
    return true;
}

// Where the reduce pipeline's stages start in dynamic shared memory (behind the transfer rings and the flag board).
__device__ __forceinline__ char* reduce_area(const CombineParams& p, char* smem) {
    const int64_t ring_end = (align_up(int64_t(p.c.layout.hidden) * 2, 128) + 8) * int64_t(p.push_warps) * p.stages;
    const uintptr_t board = (reinterpret_cast<uintptr_t>(smem + ring_end) + 15) & ~uintptr_t(15);
    return reinterpret_cast<char*>((board + sizeof(FlagBoard) + 127) & ~uintptr_t(127));
}

// The source-side sum fed through shared memory.  The CTA sums ONE of its tokens at a time: the first reduce warp
// (the loader) waits for the token's arrival flags and bulk-loads `reduce_chunk_bytes` of every expected partition
// row into the next free stage of a small ring; the other reduce warps wait on the stage's mbarrier, add the rows
// in FP32 in ascending partition order straight from shared memory, add the bias, round once and store.  A bulk load
// keeps no registers busy, so all partitions of a chunk are in flight at once and several chunks ahead: what is left
// of the kernel after the last row has landed is one load latency and a sum from shared memory, where the register
// path needs seven dependent batches of loads per token.
__device__ void combine_reduce_smem_role(const CombineParams& p, int* abort_word, char* area) {
    const WindowLayout& L = p.c.layout;
    const int K = L.topk, Le = L.local_experts, E = int(L.num_experts), H = L.hidden, P = p.reduce_parts;
    const int lane = threadIdx.x & 31;
    const int RW = (blockDim.x >> 5) - p.push_warps - 1;
    const int rwarp = (threadIdx.x >> 5) - p.push_warps - 1;
    const int CW = RW - 1;  // consumer warps
    const int NS = p.reduce_stages, cw = p.reduce_chunk_bytes, xb = H * 2;
    const int nc = (xb + cw - 1) / cw;
    const ReduceArea place = ReduceArea::make(NS, P, cw);
    uint64_t* full = reinterpret_cast<uint64_t*>(area + place.barriers);
    uint64_t* empty = full + NS;
    int* rows_in_stage = reinterpret_cast<int*>(area + place.rows);
    const StatusRef status = status_of(p.c);
    const uint32_t tag = combine_tag(p.epoch);
    const int n_tok = p.tokens > int(blockIdx.x) ? (p.tokens - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x) : 0;
    const int units = n_tok * nc;
    const uint64_t once = l2_evict_first_policy();

    if (rwarp == 0) {
        // ---- loader.  It looks at the flags of several tokens at once: a token has G lanes, one per choice, so a poll, an
        // acquiring load and a read of the routing serve 32 / G tokens.  (One token at a time, the chain routing -> flag ->
        // acquire -> gate weights -> load took 3.6 us per token, which a combine of 1000 compact tokens over four ranks
        // waited for: 138 -> 105 us.  With one system fence for all tokens instead of the acquiring loads it took 141 us.)
        const uint32_t* flag_base = reinterpret_cast<const uint32_t*>(window(p.c, p.c.rank) + L.ret_flag_offset);
        const float* ret_w = reinterpret_cast<const float*>(window(p.c, p.c.rank) + L.ret_w_offset);
        const int G = K <= 4 ? 4 : K <= 8 ? 8 : K <= 16 ? 16 : 32, W = 32 / G;
        const unsigned token_lanes = G == 32 ? kFull : (1u << G) - 1u;
        const int sub = lane / G, k = lane % G;
        const bool direct = own_rows_in_place(p);
        auto token_of = [&](int i) { return int(blockIdx.x) + i * int(gridDim.x); };
        auto choice_of = [&](int i) -> int64_t { return i < n_tok && k < K ? p.topk[int64_t(token_of(i)) * K + k] : -1; };
        int64_t next = choice_of(sub);
        int u = 0;
        bool alive = true;
        for (int base = 0; base < n_tok && alive; base += W) {
            const int t = token_of(base + sub);
            const int64_t e = next;
            next = choice_of(base + W + sub);
            const bool valid = e >= 0 && e < E;
            const int dest = valid ? int(e) / Le : -1;
            // one partition per valid choice, or one per destination rank, named by the rank's first choice
            const unsigned same = __match_any_sync(kFull, valid ? sub * kMaxRanks + dest : 32 * kMaxRanks + lane);
            const bool mine = valid && (p.sum_all_choices != 0 || lane == __ffs(same) - 1);
            const unsigned parts = __ballot_sync(kFull, mine);
            const int my_part = L.rank_indexed ? dest : k;
            const uint32_t* flag = flag_base + int64_t(mine ? my_part : 0) * L.max_tokens + (mine ? t : 0);
            const unsigned my_lanes = token_lanes << (sub * G);
            const bool in_place = mine && dest == p.c.rank && direct;
            const char* from = ret_row(p.c, p.c.rank, mine ? my_part : 0, mine ? t : 0);  // the lane's row
            bool here = !mine;
            unsigned ordered = 0;  // lanes of the tokens that are complete and may be loaded
            for (int j = 0; j < W && base + j < n_tok; ++j) {
                const unsigned lanes = token_lanes << (j * G);
                const int tok = token_of(base + j);
                if ((ordered & lanes) != lanes) {
                    const uint64_t start = global_timer_ns();
                    uint32_t spins = 0;
                    unsigned seen;  // lanes whose row has arrived
                    for (;;) {
                        if (!here) here = ld_relaxed_sys_u32(flag) == tag;
                        seen = __ballot_sync(kFull, here);
                        if ((seen & lanes) == lanes) break;
                        __nanosleep(100);
                        if ((++spins & 15u) == 0u &&
                            __any_sync(kFull, *(volatile int*)abort_word != 0 || global_timer_ns() - start > p.c.timeout_ns)) {
                            alive = false;
                            break;
                        }
                    }
                    if (!alive) {
                        if (lane == 0) {
                            report(status, kBarrierTimeout, uint32_t(tok), kTagReduce);
                            *(volatile int*)abort_word = 1;  // a peer never delivered: the consumers stop at their next wait
                        }
                        break;
                    }
                    // the polls were relaxed; one acquiring load of each flag orders the rows behind them, and the
                    // proxy fence orders the bulk loads below behind that
                    const bool complete = (seen & my_lanes) == my_lanes, fresh = complete && !((ordered >> lane) & 1u);
                    if (fresh && mine) (void)ld_acquire_sys_u32(flag);
                    if (fresh && in_place) from = reinterpret_cast<const char*>(p.y + int64_t(*reinterpret_cast<const volatile int*>(from)) * H);
                    __syncwarp();
                    if (fresh && p.w_out != nullptr && k < K && base + sub < n_tok)
                        p.w_out[int64_t(t) * K + k] = valid ? __ldcg(ret_w + int64_t(t) * K + k) : 0.f;
                    fence_proxy_async();
                    __syncwarp();
                    ordered = __ballot_sync(kFull, complete);
                }
                const bool own = sub == j;
                const unsigned token_parts = parts & lanes;
                const int np = __popc(token_parts);
                for (int c = 0; c < nc; ++c, ++u) {
                    const int s = u % NS, n = u / NS;
                    if (n >= 1) {
                        // the stage is free once every consumer warp has read its previous contents
                        bool ok = mbar_wait_or_abort(empty + s, uint32_t(n - 1) & 1u, p.c.timeout_ns, abort_word);
                        ok = __all_sync(kFull, ok);
                        if (!ok) {
                            if (lane == 0 && *(volatile int*)abort_word == 0) {
                                report(status, kCopyTimeout, uint32_t(tok), kTagReduce);
                                *(volatile int*)abort_word = 1;
                            }
                            alive = false;
                            break;
                        }
                    }
                    const int bytes = min(cw, xb - c * cw);
                    if (lane == 0) {
                        rows_in_stage[s] = np;  // the arrival below hands it to the consumers
                        mbar_expect_tx(full + s, uint32_t(np * bytes));
                    }
                    __syncwarp();
                    if (own && mine) {
                        const int at = __popc(token_parts & lanemask_lt());
                        bulk_load_hint(area + (int64_t(s) * P + at) * cw, from + int64_t(c) * cw, uint32_t(bytes),
                                       full + s, once);
                    }
                }
                if (!alive) break;
            }
        }
        return;
    }

    // ---- consumers
    const int cwarp = rwarp - 1;
    unsigned waited = 0, worked = 0, longest = 0, summed = 0;  // nanoseconds
    unsigned long long longest_at = 0, last_seen = 0;
    for (int u = 0; u < units; ++u) {
        const int c = u % nc, t = int(blockIdx.x) + (u / nc) * int(gridDim.x);
        const int s = u % NS, n = u / NS;
        const uint64_t t_wait = p.trace != nullptr ? global_timer_ns() : 0;
        {
            bool ok = mbar_wait_or_abort(full + s, uint32_t(n) & 1u, p.c.timeout_ns, abort_word);
            ok = __all_sync(kFull, ok);
            if (!ok) {
                if (lane == 0 && *(volatile int*)abort_word == 0) {
                    report(status, kCopyTimeout, uint32_t(t), kTagReduce);
                    *(volatile int*)abort_word = 1;
                }
                break;
            }
        }
        const uint64_t t_work = p.trace != nullptr ? global_timer_ns() : 0;
        const int np = *(volatile const int*)(rows_in_stage + s);
        const int bytes = min(cw, xb - c * cw);
        const char* rows = area + int64_t(s) * P * cw;
        for (int v = cwarp * 32 + lane; v * 16 < bytes; v += CW * 32) {
            float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int j = 0; j < np; ++j) accumulate8(a, *reinterpret_cast<const int4*>(rows + int64_t(j) * cw + v * 16));
            const int64_t at = (int64_t(t) * xb + int64_t(c) * cw) / 16 + v;  // 16-byte units from the start of the output
            if (p.bias != nullptr) accumulate8(a, ld_nc_v4(reinterpret_cast<const int4*>(p.bias) + at));
            st_v4_hint(reinterpret_cast<int4*>(p.out) + at, pack8(a), once);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + s);
        if (p.trace != nullptr) {
            const uint64_t t_done = global_timer_ns();
            waited += unsigned(t_work - t_wait);
            worked += unsigned(t_done - t_work);
            if (unsigned(t_done - t_work) > longest) {
                longest = unsigned(t_done - t_work);
                longest_at = t_work;
            }
            last_seen = t_work;
            summed += c == 0 ? 1u : 0u;
        }
    }
    if (p.trace != nullptr && cwarp == 0 && lane == 0) {
        atomicAdd(p.trace + 4, (unsigned long long)waited);
        atomicAdd(p.trace + 5, (unsigned long long)worked);
        atomicAdd(p.trace + 6, (unsigned long long)summed);
        const unsigned long long t0 = *(volatile unsigned long long*)p.trace;
        atomicMax(p.trace + 7, ((unsigned long long)longest << 32) | (unsigned long long)unsigned(longest_at - t0));
        atomicMax(p.trace + 8, last_seen);
    }
}

__device__ void combine_body(const CombineParams& p) {
    extern __shared__ __align__(128) char s_ring[];
    __shared__ int s_enter;
    __shared__ int s_flow[kReduceFlowWords];  // see combine_reduce_role
    const WindowLayout& L = p.c.layout;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const StatusRef status = status_of(p.c);
    int* ctrl = ctrl_words(p.c);
    // the flag board sits behind the transfer rings (plan_ring leaves room for it)
    FlagBoard* board = reinterpret_cast<FlagBoard*>(
        (reinterpret_cast<uintptr_t>(s_ring + (align_up(int64_t(L.hidden) * 2, 128) + 8) * int64_t(p.push_warps) * p.stages) + 15) & ~uintptr_t(15));
    if (threadIdx.x == 0) {
        s_enter = 1;
        if (p.reduce_stages >= 2) {
            // full: the loader's arrival plus the bytes of its bulk loads; empty: one arrival per consumer warp
            char* area = reduce_area(p, s_ring);
            uint64_t* full = reinterpret_cast<uint64_t*>(area + ReduceArea::make(p.reduce_stages, p.reduce_parts, p.reduce_chunk_bytes).barriers);
            const int consumers = int(blockDim.x >> 5) - p.push_warps - 2;
            for (int s = 0; s < p.reduce_stages; ++s) {
                mbar_init(full + s, 1);
                mbar_init(full + p.reduce_stages + s, uint32_t(consumers));
            }
            mbar_init_fence();
            fence_proxy_async_smem();
        }
    }
    if (threadIdx.x < kReduceFlowWords) s_flow[threadIdx.x] = 0;
    if (threadIdx.x < kMaxPushWarps) board->completed[threadIdx.x] = board->published[threadIdx.x] = board->finished[threadIdx.x] = 0;
    __syncthreads();
    if (p.wait_epoch != 0) {
        // Every peer has finished reading what the previous combine left in its return area.
        if (warp == 0) {
            const bool ok = peer_wait_warp(p.c.peers, p.c.rank, L.ranks, L.signal_offset, p.wait_epoch, p.c.timeout_ns, status, kTagPush);
            if (lane == 0) s_enter = ok;
        }
        __syncthreads();
    }
    if (p.trace != nullptr && threadIdx.x == 0) atomicMin(p.trace, global_timer_ns());
    if (s_enter) {
        const int role = warp < p.push_warps ? 1 : warp == p.push_warps ? 2 : 3;
        if (role == 1)
            combine_push_role(p, s_ring, board);
        else if (role == 2)
            combine_publish_role(p, board);
        else if (p.reduce_stages >= 2)
            combine_reduce_smem_role(p, s_flow, reduce_area(p, s_ring));
        else
            combine_reduce_role(p, s_flow);
        if (p.trace != nullptr && lane == 0) atomicMax(p.trace + role, global_timer_ns());
    }
    // The last block out tells every peer that this rank is done with the combine (nobody waits here).  Rows and
    // flags are out already (completed bulk groups, the publishers' fences); the ticket orders this block's reads of
    // the return area before the signal that lets peers overwrite it.
    if (!take_last_ticket(ctrl + WindowLayout::kTicketCombine)) return;
    if (threadIdx.x == 0) {
        ctrl[WindowLayout::kTicketCombine] = 0;
        ctrl[WindowLayout::kWorkCursor] = 0;  // every transfer warp of the rank is done: the next combine starts its walk at 0
    }
    if (warp == 0) peer_signal_warp(p.c.peers, p.c.rank, L.ranks, L.signal_offset, p.epoch);
}

// ------------------------------------------------------------------------------------------
// Sums of whole rows that are already in local memory: the reduction of a combine whose rows another kernel pushed
// (`reduce`), and the combine of a single-rank group (`local_combine`).  Bound by reading up to K rows per token once.
// One work item is kItemVecs 16-byte columns of one token, so that a lane has all of its loads (eight rows x two
// columns) in flight at once and a few tokens still occupy many warps; with a warp per token, one token took 14
// dependent rounds of loads and 3001 tokens left a third of the warps without work.
// Hidden 7168, top-8, local_combine with a cold L2, before and now: 1 token 32 -> 3.6 us, 128 tokens 38 -> 6.9 us; warm: 3001
// tokens 84 -> 59 us, 4096 tokens (529 MB) 91 -> 80 us = 6.6 TB/s; reduce at 64 tokens 35 -> 4.7 us.  Two blocks of 256
// threads per SM keep all loads of a lane in registers (126); three blocks (80 registers) took 217 us, a grid without the
// loop 120 us.  Compact, 8192 x 4096: 40 -> 17 us.
// ------------------------------------------------------------------------------------------
constexpr int kItemVecs = 64, kCopyItemVecs = 128;

// FP32 sum of the rows named by the lanes in `mask`, in ascending lane order: lane k holds the row's index in `base`.
// `a0`/`a1` take the columns col and col + 32 (16-byte units) where `one`/`two` say that they exist.
__device__ __forceinline__ void sum_rows(const char* base, int64_t row_bytes, unsigned mask, int my_row, int col, bool one, bool two, float* a0,
                                         float* a1, uint64_t once) {
    while (mask) {
        int row[8];
        int4 d0[8], d1[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = mask ? __ffs(mask) - 1 : -1;
            if (mask) mask &= mask - 1;
            row[j] = __shfl_sync(kFull, my_row, k < 0 ? 0 : k);
            if (k < 0) row[j] = -1;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (row[j] >= 0) {
                const int4* src = reinterpret_cast<const int4*>(base + row[j] * row_bytes);
                if (one) d0[j] = ld_cg_v4_hint(src + col, once);
                if (two) d1[j] = ld_cg_v4_hint(src + col + 32, once);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (row[j] >= 0) {
                if (one) accumulate8(a0, d0[j]);
                if (two) accumulate8(a1, d1[j]);
            }
        }
    }
}

// Bias once, one bf16 round, store.
__device__ __forceinline__ void finish_columns(float* a0, float* a1, int col, bool one, bool two, const __nv_bfloat16* bias_row,
                                               __nv_bfloat16* out_row, uint64_t once) {
    if (bias_row != nullptr) {
        const int4* b = reinterpret_cast<const int4*>(bias_row);
        if (one) accumulate8(a0, ld_nc_v4(b + col));
        if (two) accumulate8(a1, ld_nc_v4(b + col + 32));
    }
    int4* o = reinterpret_cast<int4*>(out_row);
    if (one) st_v4_hint(o + col, pack8(a0), once);
    if (two) st_v4_hint(o + col + 32, pack8(a1), once);
}

__device__ void reduce_body(const ReduceParams& p) {
    const WindowLayout& L = p.c.layout;
    const int K = L.topk, Le = L.local_experts, E = int(L.num_experts), H = L.hidden;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const int gw = blockIdx.x * wpb + warp, GW = gridDim.x * wpb;
    const int vecs = H / 8, per_token = (vecs + kItemVecs - 1) / kItemVecs;
    const char* ret = window(p.c, p.c.rank) + L.ret_offset;
    const float* ret_w = reinterpret_cast<const float*>(window(p.c, p.c.rank) + L.ret_w_offset);
    const uint64_t once = l2_evict_first_policy();
    const int64_t items = int64_t(p.tokens) * per_token;
    for (int64_t item = gw; item < items; item += GW) {
        const int t = int(item / per_token), c = int(item - int64_t(t) * per_token);
        bool valid;
        int dest;
        const unsigned parts = expected_parts(p.topk, t, K, E, Le, p.sum_all_choices != 0, valid, dest);
        const int part = L.rank_indexed ? dest : lane;
        const int col = c * kItemVecs + lane;
        const bool one = col < vecs, two = col + 32 < vecs;
        float a0[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float a1[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        sum_rows(ret, int64_t(H) * 2, parts, part * int(L.max_tokens) + t, col, one, two, a0, a1, once);
        finish_columns(a0, a1, col, one, two, p.bias != nullptr ? p.bias + int64_t(t) * H : nullptr, p.out + int64_t(t) * H, once);
        if (c == 0 && p.w_out != nullptr && lane < K) p.w_out[int64_t(t) * K + lane] = valid ? __ldcg(ret_w + int64_t(t) * K + lane) : 0.f;
    }
}

// Tokens without any valid choice have no receive row: result = bias (or zero), weights = 0.
__device__ void finish_rowless_tokens(const LocalCombineParams& p, int rows, int first, int step) {
    if (rows == p.tokens) return;
    const WindowLayout& L = p.c.layout;
    const int lane = threadIdx.x & 31, K = L.topk, H = L.hidden;
    for (int t = first; t < p.tokens; t += step) {
        const int64_t e = lane < K ? p.topk[int64_t(t) * K + lane] : -1;
        if (__ballot_sync(kFull, e >= 0 && e < L.num_experts) != 0) continue;
        int4* out = reinterpret_cast<int4*>(p.out + int64_t(t) * H);
        const int4* bias = p.bias != nullptr ? reinterpret_cast<const int4*>(p.bias + int64_t(t) * H) : nullptr;
        for (int c = lane; c < H / 8; c += 32) out[c] = bias != nullptr ? ld_nc_v4(bias + c) : make_int4(0, 0, 0, 0);
        if (p.w_out != nullptr && lane < K) p.w_out[int64_t(t) * K + lane] = 0.f;
    }
}

__device__ __forceinline__ int local_rows(const LocalCombineParams& p) {
    return p.rows_device != nullptr ? int(min(int64_t(p.rows), *p.rows_device)) : p.rows;
}

// Token and choices of receive row r on all lanes: lane k holds choice k.  False: nothing to add up (or bad metadata).
__device__ __forceinline__ bool local_row(const LocalCombineParams& p, int r, int& tok, int& v, unsigned& vm) {
    const int lane = threadIdx.x & 31, K = p.c.layout.topk;
    const int* m = p.meta + int64_t(r) * (K + 2);
    const int src = m[0];
    tok = m[1];
    v = lane < K ? m[2 + lane] : -1;
    if (src != p.c.rank || tok < 0 || tok >= p.tokens) {
        if (lane == 0) report(status_of(p.c), kBadMetadata, uint32_t(r), kTagReduce);
        return false;
    }
    vm = __ballot_sync(kFull, v >= 0 && (!p.expand || v < p.capacity));
    return vm != 0;
}

__device__ void local_combine_body(const LocalCombineParams& p) {
    const WindowLayout& L = p.c.layout;
    const int K = L.topk, H = L.hidden;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const int gw = blockIdx.x * wpb + warp, GW = gridDim.x * wpb;
    const int vecs = H / 8, per_row = (vecs + kItemVecs - 1) / kItemVecs;
    const uint64_t once = l2_evict_first_policy();
    const int rows = local_rows(p);
    const int64_t items = int64_t(rows) * per_row;
    for (int64_t item = gw; item < items; item += GW) {
        const int r = int(item / per_row), c = int(item - int64_t(r) * per_row);
        int tok, v;
        unsigned vm;
        if (!local_row(p, r, tok, v, vm)) continue;
        const int col = c * kItemVecs + lane;
        const bool one = col < vecs, two = col + 32 < vecs;
        float a0[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float a1[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        sum_rows(reinterpret_cast<const char*>(p.y), int64_t(H) * 2, vm, v, col, one, two, a0, a1, once);
        if (p.round_partial) {
            const int4 r0 = pack8(a0), r1 = pack8(a1);
#pragma unroll
            for (int j = 0; j < 8; ++j) a0[j] = a1[j] = 0.f;
            accumulate8(a0, r0);
            accumulate8(a1, r1);
        }
        finish_columns(a0, a1, col, one, two, p.bias != nullptr ? p.bias + int64_t(tok) * H : nullptr, p.out + int64_t(tok) * H, once);
        if (c == 0 && p.w_out != nullptr && lane < K) p.w_out[int64_t(tok) * K + lane] = ((vm >> lane) & 1u) ? p.w[v] : 0.f;
    }
    finish_rowless_tokens(p, rows, gw, GW);
}

// The compact layout: a row is its token's sum already.  A streaming copy (plus bias); few registers, so that many warps
// are resident, each with kCopyItemVecs / 32 loads per lane in flight.
__device__ void local_combine_compact_body(const LocalCombineParams& p) {
    const WindowLayout& L = p.c.layout;
    const int K = L.topk, H = L.hidden;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const int gw = blockIdx.x * wpb + warp, GW = gridDim.x * wpb;
    constexpr int kCols = kCopyItemVecs / 32;
    const int vecs = H / 8, per_row = (vecs + kCopyItemVecs - 1) / kCopyItemVecs;
    const uint64_t once = l2_evict_first_policy();
    const int rows = local_rows(p);
    const int64_t items = int64_t(rows) * per_row;
    for (int64_t item = gw; item < items; item += GW) {
        const int r = int(item / per_row), c = int(item - int64_t(r) * per_row);
        const int col = c * kCopyItemVecs + lane;
        const int4* from = reinterpret_cast<const int4*>(p.y + int64_t(r) * H);
        int4 d[kCols];
#pragma unroll
        for (int j = 0; j < kCols; ++j)
            if (col + 32 * j < vecs) d[j] = ld_cg_v4_hint(from + col + 32 * j, once);
        int tok, v;
        unsigned vm;
        if (!local_row(p, r, tok, v, vm)) continue;
        int4* to = reinterpret_cast<int4*>(p.out + int64_t(tok) * H);
        const int4* bias = p.bias != nullptr ? reinterpret_cast<const int4*>(p.bias + int64_t(tok) * H) : nullptr;
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
            if (col + 32 * j < vecs) {
                float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                accumulate8(a, d[j]);
                if (bias != nullptr) accumulate8(a, ld_nc_v4(bias + col + 32 * j));
                st_v4_hint(to + col + 32 * j, pack8(a), once);
            }
        }
        if (c == 0 && p.w_out != nullptr && lane < K) p.w_out[int64_t(tok) * K + lane] = ((vm >> lane) & 1u) ? p.w[int64_t(r) * K + lane] : 0.f;
    }
    finish_rowless_tokens(p, rows, gw, GW);
}

__device__ void barrier_body(const BarrierParams& p) {
    if (p.signal_only) {
        peer_signal_warp(p.c.peers, p.c.rank, p.c.layout.ranks, p.c.layout.signal_offset, p.epoch);
        return;
    }
    peer_barrier_warp(p.c.peers, p.c.rank, p.c.layout.ranks, p.c.layout.signal_offset, p.epoch, p.c.timeout_ns, status_of(p.c),
                      kTagBarrier);
}

// Test utility: holds a stream until a word in pinned host memory becomes non-zero (bounded; gate[1] = 1 when the wait
// ran out).  The poll is a system-scope load: it must not be served from a cache on the GPU.
// Lets a test keep one rank's kernel pending at a chosen point while the other ranks run on.
__global__ void gate_kernel(volatile int* gate, uint64_t timeout_ns) {
    const uint64_t start = global_timer_ns();
    while (ld_relaxed_sys(const_cast<const int*>(gate)) == 0) {
        __nanosleep(500);
        if (global_timer_ns() - start > timeout_ns) {
            gate[1] = 1;
            break;
        }
    }
}

// ---------------------------------------------------------------- wrappers
template <typename P>
__device__ __forceinline__ const P& block_of(const Many<P>& all) {
    return all.device != nullptr ? all.device[blockIdx.y] : all.host[blockIdx.y];
}
#define NEP_KERNEL_PAIR(name, Params, ...)                                                                          \
    __global__ void __launch_bounds__(__VA_ARGS__) name##_kernel(const __grid_constant__ Params p) { name##_body(p); } \
    __global__ void __launch_bounds__(__VA_ARGS__) name##_multi_kernel(const __grid_constant__ Many<Params> all) { name##_body(block_of(all)); }

// Two blocks per SM, which the grid counts on: the kernel for several ranks took 76 registers and half of its grid waited for a second
// wave (39.9 -> 35.2 us at eight ranks of 512 tokens, 34.3 -> 25.5 at four of 1000); its 64 registers cost it a few spilled words.
__global__ void __launch_bounds__(kStageThreads, 2) stage_kernel(const __grid_constant__ StageParams p) { stage_body(p); }
__global__ void __launch_bounds__(kStageThreads, 2) stage_multi_kernel(const __grid_constant__ Many<StageParams> all) { stage_body(block_of(all)); }
__global__ void __launch_bounds__(kLocalPlanThreads) local_plan_kernel(const __grid_constant__ LocalPlanParams p) { local_plan_body(p); }
NEP_KERNEL_PAIR(plan, PlanParams, kPlanThreads)
NEP_KERNEL_PAIR(pull, PullParams, 256)
__global__ void __launch_bounds__(kCombineThreads, 1) combine_kernel(const __grid_constant__ CombineParams p) { combine_body(p); }
__global__ void __launch_bounds__(kCombineThreads, 1) combine_multi_kernel(const __grid_constant__ Many<CombineParams> all) { combine_body(block_of(all)); }
NEP_KERNEL_PAIR(reduce, ReduceParams, kRowSumThreads, kRowSumBlocks)
NEP_KERNEL_PAIR(barrier, BarrierParams, 32)
NEP_KERNEL_PAIR(local_combine, LocalCombineParams, kRowSumThreads, kRowSumBlocks)
NEP_KERNEL_PAIR(local_combine_compact, LocalCombineParams, kRowSumThreads, kRowCopyBlocks)

// Fresh dispatch of a small call in ONE cooperative launch: stage (count exchange, peer barrier, prefixes, mailbox),
// plan, pull.  Outputs are sized by the caller at an upper bound and trimmed on the host once N and C are known, so
// the host's wait for the mailbox runs beside the kernel instead of between two launches.
__device__ void fused_fresh_dispatch_body(const StageParams& sp, const PlanParams& lp, const PullParams& pp) {
    if (!stage_body(sp)) return;
    plan_body(lp);
    // every block of this rank has planned its chunks before any row is pulled
    int* ctrl = ctrl_words(sp.c);
    if (take_last_ticket(ctrl + WindowLayout::kTicketPlan)) {
        if (threadIdx.x == 0) {
            ctrl[WindowLayout::kTicketPlan] = 0;
            publish_go(ctrl, sp.epoch, true, WindowLayout::kGoWordPlan);
        }
    } else if (!wait_go(ctrl, sp.epoch, sp.c.timeout_ns, status_of(sp.c), kTagPlan, WindowLayout::kGoWordPlan)) {
        return;
    }
    __syncthreads();
    fence_proxy_async();
    pull_body(pp);
}
__global__ void __launch_bounds__(256) fused_fresh_dispatch_kernel(const __grid_constant__ StageParams sp, const __grid_constant__ PlanParams lp,
                                                                   const __grid_constant__ PullParams pp) {
    fused_fresh_dispatch_body(sp, lp, pp);
}
__global__ void __launch_bounds__(256) fused_fresh_dispatch_multi_kernel(const __grid_constant__ Many<StageParams> sp,
                                                                         const __grid_constant__ Many<PlanParams> lp,
                                                                         const __grid_constant__ Many<PullParams> pp) {
    fused_fresh_dispatch_body(block_of(sp), block_of(lp), block_of(pp));
}

// stage + peer barrier + pull in one cooperative launch (cached dispatch, small calls)
__global__ void __launch_bounds__(256) fused_cached_dispatch_kernel(const __grid_constant__ StageParams sp, const __grid_constant__ PullParams pp) {
    if (!stage_body(sp)) return;
    fence_proxy_async();
    pull_body(pp);
}
__global__ void __launch_bounds__(256) fused_cached_dispatch_multi_kernel(const __grid_constant__ Many<StageParams> sp,
                                                                          const __grid_constant__ Many<PullParams> pp) {
    if (!stage_body(block_of(sp))) return;
    fence_proxy_async();
    pull_body(block_of(pp));
}

// Raises a kernel's dynamic shared-memory limit when a launch needs more than it was granted so far.  The limit belongs
// to the kernel on its device, not to a thread: the record is shared, and a smaller request never lowers it.
cudaError_t allow_shared_memory(const void* fn, size_t smem) {
    static std::mutex mutex;
    static std::map<std::pair<const void*, int>, size_t> granted;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const std::lock_guard<std::mutex> lock(mutex);
    size_t& have = granted[{fn, device}];
    if (smem <= have) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e == cudaSuccess) have = smem;
    return e;
}

// Launch with programmatic stream serialization: the kernel may be set up while its predecessor still runs and waits
// for it with wait_for_previous().
template <typename Params>
cudaError_t launch_dependent(void (*fn)(const Params), const Params& params, int grid, int cluster, int threads, size_t smem, cudaStream_t stream) {
    if (smem > 48 * 1024) {
        const cudaError_t e = allow_shared_memory((const void*)fn, smem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(unsigned(grid));
    config.blockDim = dim3(unsigned(threads));
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = unsigned(cluster);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    config.attrs = attr;
    config.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&config, fn, params);
}

template <typename P>
Many<P> make_many(const P* params, int ranks) {
    Many<P> many{};
    if (ranks > kInlineRanks)
        many.device = params;
    else
        for (int r = 0; r < ranks; ++r) many.host[r] = params[r];
    return many;
}

template <typename Params>
cudaError_t launch_pair(void (*single)(const Params), void (*multi)(const Many<Params>), const Params* params, LaunchShape shape, int threads,
                        size_t smem, cudaStream_t stream) {
    if (smem > 48 * 1024) {
        const cudaError_t e = allow_shared_memory(shape.ranks_y > 1 ? (const void*)multi : (const void*)single, smem);
        if (e != cudaSuccess) return e;
    }
    const dim3 grid(shape.grid_x, shape.ranks_y > 1 ? shape.ranks_y : 1);
    if (shape.ranks_y > 1)
        multi<<<grid, threads, smem, stream>>>(make_many(params, shape.ranks_y));
    else
        single<<<grid, threads, smem, stream>>>(*params);
    return cudaGetLastError();
}

}  // namespace

int row_sum_grid(int64_t tokens, int hidden, bool sums, int sms) {
    // one work item per warp until every SM is full; from there on the blocks loop (a larger grid measured slower)
    const int64_t item_vecs = sums ? kItemVecs : kCopyItemVecs;
    const int64_t items = tokens * ((hidden / 8 + item_vecs - 1) / item_vecs);
    const int64_t blocks = (items + kRowSumThreads / 32 - 1) / (kRowSumThreads / 32);
    return int(std::max<int64_t>(1, std::min<int64_t>(blocks, int64_t(sums ? kRowSumBlocks : kRowCopyBlocks) * sms)));
}
int stage_smem_bytes(const WindowLayout& l) { return int((l.ranks + l.num_experts) * 4); }
int plan_smem_bytes(const WindowLayout& l) { return (kPlanThreads / 32) * 32 * l.topk * 4; }

RingPlan plan_ring(int64_t row_bytes, int max_smem_bytes, bool shared) {
    // smem = warps * stages * (row pitch + one mbarrier) + zero buffer + alignment slack + static smem.
    // The software pipeline needs at least two stages; a row that does not fit twice is rejected by
    // the caller (warps == 0).
    const int64_t pitch = align_up(row_bytes, 128);
    const int64_t fixed = kZeroBytes + 256 + 256;
    RingPlan r{};
    r.stages = 3;
    int warps = int((int64_t(max_smem_bytes) - fixed) / ((pitch + 8) * r.stages));
    // Under a small budget two warps with two stages beat one warp with three: the same number of
    // loads in flight, twice the instruction issue.
    const int warps2 = int((int64_t(max_smem_bytes) - fixed) / ((pitch + 8) * 2));
    if (warps < 2 && warps2 > warps) {
        r.stages = 2;
        warps = warps2;
    }
    if (warps < 1) warps = 0;
    r.warps = warps > 8 ? 8 : warps;
    // What the rings leave goes to the zero source of the padding rows, up to a whole row: stores of 2 KB reach
    // 4.8 TB/s, of 3.5 KB and more 5.9 TB/s (rows in random order).  Not beside a gated GEMM: its blocks wait for this
    // kernel's rows, so both have to fit an SM, and at hidden 4096 a ring of 80 KB leaves the three-stage GEMM (148 KB of the
    // SM's 228) its place with 2 KB of zeros (75.4 KB) but not with 6 KB (79.7 KB).
    const int64_t used = int64_t(r.warps) * r.stages * (pitch + 8);
    const int64_t left = shared ? 0 : std::min(pitch, (int64_t(max_smem_bytes) - 512 - used) / 128 * 128);
    r.zero_bytes = int(std::max<int64_t>(kZeroBytes, left));
    r.smem_bytes = size_t(used) + r.zero_bytes + 256;
    return r;
}

CombinePlan plan_combine(int64_t row_bytes, int parts, int max_smem_bytes, int reduce_stages, int reduce_chunk_bytes) {
    // smem = transfer rings (warps x stages x (row pitch + mbarrier)) + flag board + reduce pipeline
    // (ReduceArea) + alignment slack + static smem.
    CombinePlan c{};
    const int64_t pitch = align_up(row_bytes, 128);
    const int64_t fixed = int64_t(sizeof(FlagBoard)) + 16 + 128 + 512;
    int64_t chunk = 0;
    if (reduce_stages >= 2) {
        // about half of shared memory for the pipeline unless the caller names a chunk; whole rows when they fit
        chunk = reduce_chunk_bytes > 0 ? align_up(reduce_chunk_bytes, 128) : (int64_t(max_smem_bytes) / 2 / reduce_stages / parts) / 128 * 128;
        chunk = std::min<int64_t>(chunk, pitch);
    }
    // transfer warps the rings would get without a pipeline: an automatic chunk shrinks rather than take the second one
    const int64_t alone = std::min<int64_t>((int64_t(max_smem_bytes) - fixed) / (pitch + 8) / 2, 8);
    for (;;) {
        const bool piped = reduce_stages >= 2 && chunk >= 128;
        const int64_t pipe = piped ? ReduceArea::make(reduce_stages, parts, chunk).bytes : 0;
        const int64_t slots = (int64_t(max_smem_bytes) - fixed - pipe) / (pitch + 8);
        // three stages per transfer warp when there is room for at least four such warps, else two
        const int stages = slots >= 12 ? 3 : 2;
        const int64_t warps = std::min<int64_t>(slots / stages, 8);
        if (piped && reduce_chunk_bytes <= 0 && warps >= 1 && warps < std::min<int64_t>(2, alone) && chunk >= 2048) {
            chunk = chunk / 2 / 128 * 128;
            continue;
        }
        if (warps < 1 && piped) {
            // a long row leaves no room for the transfer rings: halve the chunk, and without any room left fall back
            // to the register path
            chunk = chunk > 128 ? std::max<int64_t>(128, chunk / 2 / 128 * 128) : 0;
            continue;
        }
        c.ring.stages = stages;
        c.ring.warps = warps < 1 ? 0 : int(warps);
        c.reduce_stages = piped ? reduce_stages : 0;
        c.reduce_chunk_bytes = piped ? int(chunk) : 0;
        c.ring.smem_bytes = size_t(c.ring.warps) * stages * (pitch + 8) + size_t(fixed - 256) + size_t(pipe);
        return c;
    }
}

cudaError_t launch_stage(const StageParams* params, LaunchShape shape, size_t smem, cudaStream_t stream) {
    return launch_pair<StageParams>(stage_kernel, stage_multi_kernel, params, shape, kStageThreads, smem, stream);
}
cudaError_t launch_plan(const PlanParams* params, LaunchShape shape, size_t smem, cudaStream_t stream) {
    return launch_pair<PlanParams>(plan_kernel, plan_multi_kernel, params, shape, kPlanThreads, smem, stream);
}
bool local_plan_fits(const WindowLayout& l, int64_t tokens) { return l.ranks == 1 && tokens <= kLocalPlanMaxTokens && l.num_experts <= kLocalPlanMaxExperts; }
cudaError_t launch_local_plan(const LocalPlanParams& params, cudaStream_t stream) {
    const WindowLayout& l = params.c.layout;
    // one chunk of 32 tokens per warp until the cluster is full
    int ctas = 1;
    while (ctas < kLocalPlanCtas && ctas * kLocalPlanThreads < params.tokens) ctas *= 2;
    const size_t smem = (4 * size_t(l.num_experts) + kLocalPlanChunks + size_t(kLocalPlanThreads) * l.topk) * 4;
    return launch_dependent<LocalPlanParams>(local_plan_kernel, params, ctas, ctas, kLocalPlanThreads, smem, stream);
}
cudaError_t launch_pull(const PullParams* params, LaunchShape shape, int warps, size_t smem, cudaStream_t stream) {
    if (shape.ranks_y <= 1) return launch_dependent<PullParams>(pull_kernel, *params, shape.grid_x, 1, warps * 32, smem, stream);
    return launch_pair<PullParams>(pull_kernel, pull_multi_kernel, params, shape, warps * 32, smem, stream);
}
cudaError_t launch_reduce(const ReduceParams* params, LaunchShape shape, cudaStream_t stream) {
    return launch_pair<ReduceParams>(reduce_kernel, reduce_multi_kernel, params, shape, kRowSumThreads, 0, stream);
}
cudaError_t launch_barrier(const BarrierParams* params, LaunchShape shape, cudaStream_t stream) {
    return launch_pair<BarrierParams>(barrier_kernel, barrier_multi_kernel, params, shape, 32, 0, stream);
}

namespace {
// Cooperative launch: fails instead of deadlocking if the grid cannot be resident at once.
cudaError_t launch_cooperative(const void* fn, void** args, LaunchShape shape, int threads, size_t smem, cudaStream_t stream) {
    if (smem > 48 * 1024) {
        const cudaError_t e = allow_shared_memory(fn, smem);
        if (e != cudaSuccess) return e;
    }
    return cudaLaunchCooperativeKernel(fn, dim3(shape.grid_x, shape.ranks_y > 1 ? shape.ranks_y : 1), dim3(threads), args, smem, stream);
}
static_assert(sizeof(Many<StageParams>) + sizeof(Many<PlanParams>) + sizeof(Many<PullParams>) <= 32764, "kernel parameters");
}  // namespace

cudaError_t launch_fused_cached_dispatch(const StageParams* stage, const PullParams* pull, LaunchShape shape, int warps, size_t smem,
                                         cudaStream_t stream) {
    if (shape.ranks_y <= 1) {
        void* args[2] = {(void*)stage, (void*)pull};
        return launch_cooperative((const void*)fused_cached_dispatch_kernel, args, shape, warps * 32, smem, stream);
    }
    auto sp = make_many(stage, shape.ranks_y);
    auto pp = make_many(pull, shape.ranks_y);
    void* args[2] = {&sp, &pp};
    return launch_cooperative((const void*)fused_cached_dispatch_multi_kernel, args, shape, warps * 32, smem, stream);
}

cudaError_t launch_fused_fresh_dispatch(const StageParams* stage, const PlanParams* plan, const PullParams* pull, LaunchShape shape, int warps,
                                        size_t smem, cudaStream_t stream) {
    if (shape.ranks_y <= 1) {
        void* args[3] = {(void*)stage, (void*)plan, (void*)pull};
        return launch_cooperative((const void*)fused_fresh_dispatch_kernel, args, shape, warps * 32, smem, stream);
    }
    auto sp = make_many(stage, shape.ranks_y);
    auto lp = make_many(plan, shape.ranks_y);
    auto pp = make_many(pull, shape.ranks_y);
    void* args[3] = {&sp, &lp, &pp};
    return launch_cooperative((const void*)fused_fresh_dispatch_multi_kernel, args, shape, warps * 32, smem, stream);
}

cudaError_t launch_combine(const CombineParams* params, LaunchShape shape, size_t smem, cudaStream_t stream, bool cooperative) {
    if (!cooperative) return launch_pair<CombineParams>(combine_kernel, combine_multi_kernel, params, shape, kCombineThreads, smem, stream);
    if (shape.ranks_y <= 1) {
        void* args[1] = {(void*)params};
        return launch_cooperative((const void*)combine_kernel, args, shape, kCombineThreads, smem, stream);
    }
    auto all = make_many(params, shape.ranks_y);
    void* args[1] = {&all};
    return launch_cooperative((const void*)combine_multi_kernel, args, shape, kCombineThreads, smem, stream);
}

cudaError_t launch_gate(int* gate, uint64_t timeout_ns, cudaStream_t stream) {
    gate_kernel<<<1, 1, 0, stream>>>(gate, timeout_ns);
    return cudaGetLastError();
}

cudaError_t launch_local_combine(const LocalCombineParams* params, LaunchShape shape, bool compact, cudaStream_t stream) {
    if (compact)
        return launch_pair<LocalCombineParams>(local_combine_compact_kernel, local_combine_compact_multi_kernel, params, shape, kRowSumThreads, 0, stream);
    return launch_pair<LocalCombineParams>(local_combine_kernel, local_combine_multi_kernel, params, shape, kRowSumThreads, 0, stream);
}

int kernel_table(KernelInfo* out, int capacity) {
    struct Entry {
        const char* name;
        const void* fn;
    };
    const Entry entries[] = {
        {"stage", (const void*)stage_kernel},   {"plan", (const void*)plan_kernel},     {"pull", (const void*)pull_kernel},
        {"combine", (const void*)combine_kernel}, {"reduce", (const void*)reduce_kernel}, {"barrier", (const void*)barrier_kernel},
        {"local_combine", (const void*)local_combine_kernel}, {"fused_cached_dispatch", (const void*)fused_cached_dispatch_kernel},
        {"fused_fresh_dispatch", (const void*)fused_fresh_dispatch_kernel},
        {"local_plan", (const void*)local_plan_kernel}, {"local_combine_compact", (const void*)local_combine_compact_kernel},
    };
    int n = 0;
    for (const Entry& e : entries) {
        if (n >= capacity) break;
        cudaFuncAttributes a{};
        if (cudaFuncGetAttributes(&a, e.fn) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        out[n++] = KernelInfo{e.name, a.numRegs, int(a.sharedSizeBytes), a.maxThreadsPerBlock, int(a.constSizeBytes)};
    }
    return n;
}

}  // namespace nep
