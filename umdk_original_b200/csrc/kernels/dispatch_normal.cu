// Normal-mode (prefill) dispatch for sm_100a: ONE kernel that builds the routing layout,
// all-gathers the per-expert counts through peer memory, quantises every token once and pushes
// each (token, k) row with plain P2P stores into its final, expert-grouped position in the
// destination rank's receive buffer, then raises a completion flag in every peer's memory.
//
// It replaces, in the reference, the chain dispatch_layout + notify_dispatch + two host loops +
// moe_dispatch_normal (pybind/moe_dispatch_prefill.cpp:96-160 and
// ascend_kernels/moe_dispatch_normal/op_kernel/moe_dispatch_normal.h:331-535): there a row is
// staged in the sender's window, flagged, pulled by the receiver and copied again; the slot of a
// row inside its expert and the receive offsets are computed on the host after two device->host
// copies.  Here the slot arithmetic runs on the device and a row crosses NVLink exactly once.
//
// Receive-buffer row order (same contract as the reference): local expert major, then source
// rank ascending, then the sender's (token, k) scan order.
#include <cooperative_groups.h>
#include "../common/cam_types.h"
#include "../common/ptx.cuh"
#include "../common/quant.cuh"
#include "../common/slots.cuh"
#include "launch.h"

namespace cg = cooperative_groups;

namespace cam {

constexpr int kDispThreads = 512;
constexpr int kDispWarps = kDispThreads / 32;
constexpr int kDispGroups = 16;  // most runs of rows that the column sums of the count phase are cut into
// Count-phase tables in dynamic shared memory: warp x expert counts, later the partial column sums (2 x groups x E
// words with groups * E <= 4 * kDispThreads).
constexpr int kDispTableBytes = kDispWarps * CAM_MAX_EXPERTS * 4;
static_assert(kDispTableBytes >= 2 * 4 * kDispThreads * 4, "the partial column sums must fit");

__device__ __forceinline__ void record_status(CamStatus* st, int code, int who, int detail) {
    if (atomicCAS(&st->code, 0, code) == 0) {
        st->who = who;
        st->detail = detail;
        st->block = static_cast<int>(blockIdx.x);
    }
}

// Inclusive prefix sum of v[0..n) in shared memory, n <= CAM_MAX_EXPERTS, by the whole CTA (s_part: one word per warp).
// Two values per thread, warp shuffles and one pass over the warps' totals; the serial loops over the experts that this
// replaces cost every CTA microseconds before its first row (a chain of up to 255 shared-memory reads).
__device__ __forceinline__ void block_inclusive_scan(int* v, int n, int* s_part) {
    const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5;
    const int lane = tid & 31;
    static_assert(CAM_MAX_EXPERTS <= 2 * kDispThreads, "two values per thread must cover all experts");
    const int i0 = 2 * tid, i1 = i0 + 1;
    const int a = (i0 < n) ? v[i0] : 0, b = (i1 < n) ? v[i1] : 0;
    int incl = a + b;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const int o = __shfl_up_sync(0xFFFFFFFFu, incl, s);
        if (lane >= s) incl += o;
    }
    if (lane == 31) s_part[warp] = incl;
    __syncthreads();
    int before = 0;
#pragma unroll
    for (int w = 0; w < kDispWarps; ++w) before += (w < warp) ? s_part[w] : 0;
    if (i0 < n) v[i0] = before + incl - b;
    if (i1 < n) v[i1] = before + incl;
    __syncthreads();
}

// A group of one rank exchanges nothing, and a small batch needs not even the grid-wide barrier of the count phase: every
// CTA counts all ids itself (at most kSmallPairs, 16 KB of shared memory), which gives it the first row of every expert, finds
// the slots of its own tokens' pairs by scanning the ids, and stores the rows at their places.  At most kSmallTokensPerCta
// tokens per CTA, one after the other with all threads on a row (int8: four at a time, four warps each); larger batches keep
// 16 rows in flight per CTA in the general kernel below.  What bounds it is latency: the general kernel spends 24 us on a
// batch of 16 tokens, 3 of them moving rows (grid barrier and column sums 5, count flag 3, row bases 2, data flag and its
// system-wide fences 4, the rest one warp quantising a row).  The int8 layer of 16 tokens went from 205 to 166 us with it.
// The line at four tokens per CTA (592 tokens): bf16 / e4m3 rows of 2048, top-4, take 11.0 / 12.1 us there against 13.3 / 13.4 in
// the general kernel, with 768 tokens 15.2 / 16.6 against 13.8 / 13.6; rows of 4096, top-1, 9.4 / 10.8 against 12.4 / 14.8, then
// 11.5 / 13.7 against 12.3 / 14.8; int8, four rows at a time, is ahead on both sides (7.8 against 14.0, 10.8 against 14.3).  The
// pairs are bounded by the shared memory that every mode has: 4096 of 7168 take 23.5 / 14.4 / 18.5 us (bf16 / int8 / e4m3)
// against 31.4 / 24.8 / 22.8.
constexpr int kSmallPairs = 4096, kSmallTokensPerCta = 4;
static_assert(kSmallPairs * 4 <= kDispTableBytes, "the ids must fit the dynamic shared memory of every quant mode");

__device__ void dispatch_one_rank_small(const DispatchNormalParams& p, uint8_t* dyn_smem, int* s_run, int* s_cum, float* s_red) {
    const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5;
    const uint32_t lane = lane_id();
    const int nb = static_cast<int>(gridDim.x), b = static_cast<int>(blockIdx.x);
    const int E = p.E, K = p.K, npairs = p.T * p.K;
    const int nscale = CAM_QUANT_IS_FP8(p.quant_mode) ? (p.h >> 7) : (p.quant_mode == CAM_QUANT_INT8_TOKEN) ? 1 : 0;
    const int row_bytes = (p.quant_mode == CAM_QUANT_NONE) ? p.h * 2 : p.h;
    const int stage_bytes = (p.quant_mode == CAM_QUANT_NONE) ? 0 : ((p.h + nscale * 4 + 15) & ~15);
    int* s_ids = reinterpret_cast<int*>(dyn_smem);
    uint8_t* stage0 = dyn_smem + ((static_cast<size_t>(npairs) * 4 + 15) & ~static_cast<size_t>(15));
    uint8_t* const base = p.peer_base[p.rank];
    uint8_t* const rx = base + p.off_recv_x;
    float* const rs = reinterpret_cast<float*>(base + p.off_recv_scales);
    int* const tri = reinterpret_cast<int*>(base + p.off_recv_src);

    for (int e = tid; e < E; e += kDispThreads) s_run[e] = 0;
    __syncthreads();
    for (int i = tid; i < npairs; i += kDispThreads) {
        int id = load_expert_id(p.topk_idx, p.idx_is_i64, i);
        if (id < 0 || id >= E) id = -1;
        s_ids[i] = id;
        if (id >= 0) atomicAdd(&s_run[id], 1);
    }
    __syncthreads();
    if (warp == 0) warp_scan_counts(s_run, s_cum, E, lane);
    __syncthreads();
    const int total = s_cum[E - 1];
    const bool fits = total <= p.capacity;
    if (b == 0) {  // the same bookkeeping as in the general kernel; zero rows are published when they do not fit
        for (int e = tid; e < E; e += kDispThreads) {
            const int start = fits ? s_cum[e] - s_run[e] : 0;
            p.expert_offsets[e] = start;
            p.recv_count[e] = fits ? s_cum[e] : 0;
            p.num_recv_per_expert[e] = fits ? static_cast<long long>(s_run[e]) : 0ll;
            if (p.num_tokens_per_expert_out != nullptr) p.num_tokens_per_expert_out[e] = s_run[e];
        }
        if (tid == 0) {
            p.expert_offsets[E] = fits ? total : 0;
            p.total_recv[0] = fits ? total : 0;
            if (!fits) record_status(p.status, CAM_ERR_RECV_OVERFLOW, 0, total);
            if (p.stats != nullptr) {
                atomicAdd(&p.stats->rows_routed[0], static_cast<unsigned long long>(total));
                atomicAdd(&p.stats->calls[0], 1ull);
            }
        }
    }
    if (p.g1_done != nullptr && b == nb - 1)
        for (int i = tid; i < p.g1_done_len; i += kDispThreads) p.g1_done[i] = 0u;
    // Pair k of token t by one warp: its row (or -1), noted for the caller; lanes 0..2 write the origin of a row.
    auto place = [&](int t, int k) -> int {
        const int i = t * K + k, id = s_ids[i];
        int row = -1;
        if (id >= 0 && fits) {
            row = s_cum[id] - s_run[id] + warp_slot_of(s_ids, i, lane);
            if (lane < 3) tri[static_cast<size_t>(row) * 3 + lane] = (lane == 0) ? p.rank : (lane == 1) ? t : k;
        }
        if (lane == 0) p.send_row[i] = row;
        return row;
    };
    __shared__ int s_row[4][CAM_MAX_TOPK];
    if (p.quant_mode == CAM_QUANT_INT8_TOKEN) {
        const int group = warp >> 2, gw = warp & 3, gt = tid & 127;
        uint8_t* q = stage0 + static_cast<size_t>(group) * stage_bytes;
        float* sc = reinterpret_cast<float*>(q + p.h);
        for (int t = group * nb + b; t < p.T; t += 4 * nb) {  // the first tokens go to different CTAs
            for (int k = gw; k < K; k += 4) {
                const int row = place(t, k);
                if (lane == 0) s_row[group][k] = row;
            }
            group_quant_int8_token(p.x + static_cast<size_t>(t) * p.h, p.h, q, sc, nullptr, s_red + group * 4,
                                   1u + static_cast<uint32_t>(group));
            for (int k = 0; k < K; ++k) {
                const int row = s_row[group][k];
                if (row < 0) continue;
                uint8_t* dst = rx + static_cast<size_t>(row) * row_bytes;
                for (int o = gt * 16; o < row_bytes; o += 2048) st_na_v4(dst + o, *reinterpret_cast<const uint4*>(q + o));
                if (gt == 0) rs[row] = sc[0];
            }
            asm volatile("bar.sync %0, 128;" ::"r"(1u + static_cast<uint32_t>(group)) : "memory");  // staging is free again
        }
        return;
    }
    const int parts = max(1, kDispWarps / K);
    const int part_bytes = ((row_bytes + parts - 1) / parts + 511) & ~511;
    for (int t = b; t < p.T; t += nb) {
        const __nv_bfloat16* xrow = p.x + static_cast<size_t>(t) * p.h;
        float* sc = reinterpret_cast<float*>(stage0 + p.h);
        if (p.quant_mode == CAM_QUANT_FP8_1x128) block_quant_fp8_1x128<false>(xrow, p.h, stage0, sc);
        else if (p.quant_mode == CAM_QUANT_FP8_1x128_UE8M0) block_quant_fp8_1x128<true>(xrow, p.h, stage0, sc);
        for (int k = warp; k < K; k += kDispWarps) {
            const int row = place(t, k);
            if (lane == 0) s_row[0][k] = row;
        }
        __syncthreads();
        for (int item = warp; item < K * parts; item += kDispWarps) {
            const int k = item / parts, part = item - k * parts;
            const int row = s_row[0][k];
            if (row < 0) continue;
            uint8_t* dst = rx + static_cast<size_t>(row) * row_bytes;
            const int b0 = part * part_bytes, b1 = min(row_bytes, b0 + part_bytes);
            if (p.quant_mode == CAM_QUANT_NONE) {
                if (b1 > b0) warp_copy_row<false>(dst + b0, reinterpret_cast<const uint8_t*>(xrow) + b0, b1 - b0, lane);
            } else {
                for (int o = b0 + static_cast<int>(lane) * 16; o < b1; o += 512)
                    st_na_v4(dst + o, *reinterpret_cast<const uint4*>(stage0 + o));
                if (part == 0)
                    for (int o = static_cast<int>(lane); o < nscale; o += 32) rs[static_cast<size_t>(row) * nscale + o] = sc[o];
            }
        }
        __syncthreads();  // the staged row and the places are overwritten by the next token
    }
}

__global__ void __launch_bounds__(kDispThreads, 1)
dispatch_normal_kernel(const DispatchNormalParams p) {
    extern __shared__ __align__(16) uint8_t dyn_smem[];
    __shared__ int s_hist[CAM_MAX_EXPERTS];     // running per-expert count of this CTA's chunk
    __shared__ int s_aux[CAM_MAX_EXPERTS];      // prefix over earlier CTAs / totals / bases
    __shared__ int s_tot[CAM_MAX_EXPERTS];      // rows per expert summed over all sources
    __shared__ int s_warp[kDispWarps];
    __shared__ float s_red[16];
    int* const s_cum = s_hist;                  // SEND: s_tot summed over experts (inclusive)
    __shared__ int s_rank_ok[CAM_MAX_RANKS];
    __shared__ uint32_t s_abort;
    __shared__ int s_dup_pre[CAM_MAX_RANKS + 1];

    const int tid = static_cast<int>(threadIdx.x);
    const int nb = static_cast<int>(gridDim.x);
    const int b = static_cast<int>(blockIdx.x);
    const int E = p.E, R = p.R, K = p.K, El = p.E / p.R;
    const int tpc = (p.T + nb - 1) / nb;  // tokens per CTA (contiguous chunk keeps scan order)
    const int t0 = min(p.T, b * tpc);
    const int t1 = min(p.T, t0 + tpc);
    const int npairs = (t1 - t0) * K;
    // epochs of this call, one per phase (equal when a call runs all phases in one launch)
    const uint32_t ep_count = p.epochs[0] + 1u, ep_send = p.epochs[1] + 1u, ep_recv = p.epochs[2] + 1u;
    uint8_t* const my_base = p.peer_base[p.rank];

    if (tid == 0) s_abort = 0u;
    // One rank, the whole call in this launch: nothing is exchanged and no flag is raised or waited for.  4096 tokens x 8 of
    // 7168 (302 MB in and out): 85 us -> 74 us with the parallel column sums and scans, eight loads in flight per lane and
    // without the flags; the rows themselves move at 6 TB/s.
    const bool solo = R == 1 && (p.phase_mask & CAM_PHASE_ALL) == CAM_PHASE_ALL && !p.defer_push && p.dbg_drop_flags == 0;
    if (solo && p.T * K <= kSmallPairs && p.T <= kSmallTokensPerCta * nb) {
        dispatch_one_rank_small(p, dyn_smem, s_hist, s_tot, s_red);
        goto done;
    }

    // ------------------------------------------------------------------ phase COUNT
    if (p.phase_mask & CAM_PHASE_COUNT) {
        const int parity = static_cast<int>(ep_count & 1u);
        for (int e = tid; e < E; e += kDispThreads) s_hist[e] = 0;
        __syncthreads();
        // Slot of every (token, k) pair inside its expert, in scan order, chunk-local first: match.any gives a pair's
        // rank among the equal ids of its warp, a warp x expert table of counts the rank of its warp among the 16.
        int* const tab = reinterpret_cast<int*>(dyn_smem);  // [kDispWarps][E]; the staging rows come later
        for (int sub = 0; sub < npairs; sub += kDispThreads) {
            for (int o = tid; o < kDispWarps * E; o += kDispThreads) tab[o] = 0;
            const int i = sub + tid;
            int id = -1;
            if (i < npairs) {
                id = load_expert_id(p.topk_idx, p.idx_is_i64, static_cast<size_t>(t0) * K + i);
                if (id < 0 || id >= E) id = -1;
            }
            __syncthreads();
            const uint32_t same = __match_any_sync(0xFFFFFFFFu, id);
            const int before = __popc(same & ((1u << (tid & 31)) - 1u));
            if (id >= 0 && before == 0) tab[(tid >> 5) * E + id] = __popc(same);
            __syncthreads();
            for (int e = tid; e < E; e += kDispThreads) {
                int run = s_hist[e];
#pragma unroll
                for (int w = 0; w < kDispWarps; ++w) {
                    const int c = tab[w * E + e];
                    tab[w * E + e] = run;
                    run += c;
                }
                s_hist[e] = run;
            }
            __syncthreads();
            if (i < npairs)
                p.slot_in_expert[static_cast<size_t>(t0) * K + i] =
                    (id >= 0) ? tab[(tid >> 5) * E + id] + before : -1;
            __syncthreads();
        }
        for (int e = tid; e < E; e += kDispThreads) p.cta_hist[static_cast<size_t>(b) * E + e] = s_hist[e];
        if (p.g1_done != nullptr && b == nb - 1) {
            // Counters of the fused kernel start at zero.  Peers add to this call's arrival counters only after they
            // have seen this rank's count flag, which is raised after the grid-wide barrier below.
            if (p.defer_push) {
                uint32_t* arr = reinterpret_cast<uint32_t*>(my_base + p.off_arrival) + static_cast<size_t>(parity) * E;
                for (int e = tid; e < E; e += kDispThreads) arr[e] = 0u;
            }
            for (int i = tid; i < p.g1_done_len; i += kDispThreads) p.g1_done[i] = 0u;
            __threadfence_system();
        }
        __threadfence();
        cg::this_grid().sync();

        // Exclusive prefix over earlier CTAs (s_aux) and grand total (s_tot) per expert.  The [CTAs, E] table is read by
        // groups of threads, each group a run of its rows, four experts (one 16-byte load) per thread where E allows, so
        // that all loads of a thread are in flight together (one thread per expert walking all rows took 10 us and more).
        {
            const int vec = ((E & 3) == 0) ? 4 : 1;
            const int cols = (E + vec - 1) / vec;                      // threads per group
            const int groups = max(1, min(kDispGroups, kDispThreads / cols));
            int* const s_pre = reinterpret_cast<int*>(dyn_smem);       // [groups][E], then the totals
            int* const s_sum = s_pre + groups * E;
            const int per = (nb + groups - 1) / groups;
            for (int c0 = 0; c0 < cols; c0 += kDispThreads) {          // more than one pass only for E > 512, vec = 1
                const int g = (cols <= kDispThreads) ? tid / cols : 0;
                const int c = c0 + ((cols <= kDispThreads) ? tid - g * cols : tid);
                if (g < groups && c < cols) {
                    int pre[4] = {0, 0, 0, 0}, tot[4] = {0, 0, 0, 0};
                    const int r0 = g * per, r1 = min(nb, r0 + per);
                    const int* col = p.cta_hist + static_cast<size_t>(c) * vec;
#pragma unroll 8
                    for (int bb = r0; bb < r1; ++bb) {
                        int4 v = make_int4(0, 0, 0, 0);
                        if (vec == 4) v = __ldcg(reinterpret_cast<const int4*>(col + static_cast<size_t>(bb) * E));
                        else v.x = __ldcg(col + static_cast<size_t>(bb) * E);
                        const int m = (bb < b) ? -1 : 0;
                        pre[0] += v.x & m; pre[1] += v.y & m; pre[2] += v.z & m; pre[3] += v.w & m;
                        tot[0] += v.x; tot[1] += v.y; tot[2] += v.z; tot[3] += v.w;
                    }
                    if (groups == 1) {
                        for (int u = 0; u < vec; ++u) { s_aux[c * vec + u] = pre[u]; s_tot[c * vec + u] = tot[u]; }
                    } else {
                        for (int u = 0; u < vec; ++u) {
                            s_pre[g * E + c * vec + u] = pre[u];
                            s_sum[g * E + c * vec + u] = tot[u];
                        }
                    }
                }
            }
            __syncthreads();
            if (groups > 1) {
                for (int e = tid; e < E; e += kDispThreads) {
                    int a = 0, t = 0;
                    for (int g = 0; g < groups; ++g) { a += s_pre[g * E + e]; t += s_sum[g * E + e]; }
                    s_aux[e] = a;
                    s_tot[e] = t;
                }
                __syncthreads();
            }
        }
        for (int i = tid; !solo && i < npairs; i += kDispThreads) {
            const size_t g = static_cast<size_t>(t0) * K + i;
            const int id = load_expert_id(p.topk_idx, p.idx_is_i64, g);
            if (id >= 0 && id < E) p.slot_in_expert[g] += s_aux[id];
        }
        // Count all-gather: CTA d writes this rank's full count vector into peer d's matrix.
        for (int d = b; !solo && d < R; d += nb) {
            int* dst = reinterpret_cast<int*>(p.peer_base[d] + p.off_count_matrix) +
                       (static_cast<size_t>(parity) * R + p.rank) * E;
            for (int e = tid; e < E; e += kDispThreads) dst[e] = s_tot[e];
            __syncthreads();
            if (tid == 0 && p.dbg_drop_flags == 0) {
                __threadfence_system();
                st_release_sys_u32(reinterpret_cast<uint32_t*>(p.peer_base[d] + p.off_count_flag) + p.rank,
                                   ep_count);
            }
        }
        if (p.num_tokens_per_expert_out != nullptr && b == 0) {
            for (int e = tid; e < E; e += kDispThreads) p.num_tokens_per_expert_out[e] = s_tot[e];
        }
        __syncthreads();
    }

    // ------------------------------------------------------------------ phase SEND
    if (p.phase_mask & CAM_PHASE_SEND) {
        const int parity = static_cast<int>(ep_send & 1u);
        if (!solo && tid < R) {
            const uint32_t* f = reinterpret_cast<const uint32_t*>(my_base + p.off_count_flag) + tid;
            const uint64_t t_wait = (b == 0 && p.stats != nullptr) ? globaltimer_ns() : 0ull;
            if (!wait_flag_eq_sys(f, ep_send, p.timeout_ns)) {
                record_status(p.status, CAM_ERR_TIMEOUT_COUNT_FLAG, tid, static_cast<int>(ld_acquire_sys_u32(f)));
                s_abort = 1u;
            }
            if (b == 0 && p.stats != nullptr) atomicMax(&p.stats->max_wait_ns[0][tid], globaltimer_ns() - t_wait);
        }
        __syncthreads();
        if (s_abort) goto done;  // no grid-wide sync follows, so leaving here cannot strand another CTA

        const int* cm = reinterpret_cast<const int*>(my_base + p.off_count_matrix) +
                        static_cast<size_t>(parity) * R * E;
        // rows for expert e that come from rank s (alone, this rank's totals from the count phase are all there is)
        auto count_of = [&](int s, int e) { return solo ? s_tot[e] : __ldcg(&cm[static_cast<size_t>(s) * E + e]); };
        for (int e = tid; !solo && e < E; e += kDispThreads) {
            int tot = 0;
            for (int s = 0; s < R; ++s) tot += __ldcg(&cm[static_cast<size_t>(s) * E + e]);
            s_tot[e] = tot;
        }
        __syncthreads();
        for (int e = tid; e < E; e += kDispThreads) s_cum[e] = s_tot[e];
        __syncthreads();
        block_inclusive_scan(s_cum, E, s_warp);
        // first row of expert e in its owner's receive buffer
        auto first_row = [&](int e) {
            const int lo = e - e % El;
            return s_cum[e] - s_tot[e] - (lo > 0 ? s_cum[lo - 1] : 0);
        };
        // Base row, at the owner of expert e, of the block of rows that come from this rank.
        for (int e = tid; e < E; e += kDispThreads) {
            int base = first_row(e) + (solo ? s_aux[e] : 0);  // alone, the slots are still counted inside this CTA
            for (int s = 0; s < p.rank; ++s) base += count_of(s, e);
            s_aux[e] = base;
        }
        for (int d = tid; d < R; d += kDispThreads) {
            const int tot = s_cum[d * El + El - 1] - (d > 0 ? s_cum[d * El - 1] : 0);
            s_rank_ok[d] = (tot <= p.capacity) ? 1 : 0;
            if (tot > p.capacity) record_status(p.status, CAM_ERR_RECV_OVERFLOW, d, tot);
        }
        if (b == 0 && p.stats != nullptr) {  // rows this rank routes to every rank: one warp per destination
            for (int d = tid >> 5; d < R; d += kDispWarps) {
                int mine = 0;
                for (int l = tid & 31; l < El; l += 32) mine += count_of(p.rank, d * El + l);
#pragma unroll
                for (int s = 16; s >= 1; s >>= 1) mine += __shfl_xor_sync(0xFFFFFFFFu, mine, s);
                if ((tid & 31) == 0) {
                    atomicAdd(&p.stats->rows_routed[d], static_cast<unsigned long long>(mine));
                    if (d == 0) atomicAdd(&p.stats->calls[0], 1ull);
                }
            }
        }
        __syncthreads();
        // Receiver-side bookkeeping for this rank's own experts (one CTA is enough).  When more rows are routed
        // here than the buffer holds, every sender skips this rank (s_rank_ok) and the counts published below are
        // zero, so that the kernels that follow touch no row at or past the capacity; the status word says why.
        if (b == 0) {
            const bool fits = s_rank_ok[p.rank] != 0;
            for (int le = tid; le < El; le += kDispThreads) {
                const int start = fits ? first_row(p.rank * El + le) : 0;
                p.expert_offsets[le] = start;
                int run = start;
                for (int s = 0; s < R; ++s) {
                    if (fits) run += count_of(s, p.rank * El + le);
                    p.recv_count[le * R + s] = run;  // inclusive cumsum, expert major / source minor
                }
                p.num_recv_per_expert[le] = fits ? static_cast<long long>(s_tot[p.rank * El + le]) : 0ll;
                if (le == El - 1) {
                    p.expert_offsets[El] = run;
                    p.total_recv[0] = run;
                }
            }
        }
        __syncthreads();

        // Push.  One warp per token: quantise once into the warp's staging area, then store the
        // row, its scales and its (src rank, token, k) triple to every destination.
        const int warp = tid >> 5;
        const uint32_t lane = lane_id();
        const int nscale = CAM_QUANT_IS_FP8(p.quant_mode) ? (p.h >> 7)
                           : (p.quant_mode == CAM_QUANT_INT8_TOKEN) ? 1 : 0;
        const int row_bytes = (p.quant_mode == CAM_QUANT_NONE) ? p.h * 2 : p.h;
        const int stage_bytes = (p.quant_mode == CAM_QUANT_NONE) ? 0 : ((p.h + nscale * 4 + 15) & ~15);
        uint8_t* stage_q = dyn_smem + static_cast<size_t>(warp) * stage_bytes;
        float* stage_s = reinterpret_cast<float*>(stage_q + p.h);

        // Quantised rows leave the staging area as bulk copies (one 7 KB transfer per destination
        // instead of 14 rounds of 16-byte stores per lane): lane k issues the copies of pair (t, k).
        //
        // A token crosses to a destination rank ONCE.  Lane k handles pair (t, k); lanes whose experts
        // live on the same rank find each other with match.any: the lowest of them sends the row, the
        // others append (row that arrives, row to copy it to) to the replicate list of that rank, which
        // the receiver works off locally after the data flags (RECV phase below).
        const bool bulk_rows = (p.quant_mode != CAM_QUANT_NONE) && (row_bytes % 16 == 0);
        const bool bulk_scales = bulk_rows && ((nscale * 4) % 16 == 0);
        if (p.defer_push) {
            // Nothing is pushed here.  Position of every pair in the send list: pairs are ordered by (local expert
            // at the destination, destination rank counted from this rank on, scan order), so expert 0 of every rank is
            // served first and, at any one time, the ranks of the group send to different destinations.
            int* s_mine = reinterpret_cast<int*>(dyn_smem);  // the staging area is unused in this mode
            for (int e = tid; e < E; e += kDispThreads)
                s_mine[e] = s_rank_ok[e / El] ? __ldcg(&cm[static_cast<size_t>(p.rank) * E + e]) : 0;
            __syncthreads();
            for (int e = tid; e < E; e += kDispThreads) {
                const int d = e / El, le = e - d * El;
                const int turn = (d - p.rank + R) % R;  // place of destination d in this rank's order
                int pre = 0;
                for (int l2 = 0; l2 < le; ++l2)
                    for (int d2 = 0; d2 < R; ++d2) pre += s_mine[d2 * El + l2];
                for (int t2 = 0; t2 < turn; ++t2) pre += s_mine[((p.rank + t2) % R) * El + le];
                s_hist[e] = pre;
                // the last key: the last local expert of the destination this rank serves last
                if (b == 0 && le == El - 1 && turn == R - 1) p.send_list_len[0] = pre + s_mine[e];
            }
            __syncthreads();
            for (int t = t0 + warp; t < t1; t += kDispWarps) {
                const __nv_bfloat16* xrow = p.x + static_cast<size_t>(t) * p.h;
                uint8_t* q = p.xq + static_cast<size_t>(t) * p.h;
                float* sc = p.xs + static_cast<size_t>(t) * nscale;
                if (p.quant_mode == CAM_QUANT_FP8_1x128_UE8M0) warp_quant_fp8_1x128<true>(xrow, p.h, q, sc);
                else warp_quant_fp8_1x128<false>(xrow, p.h, q, sc);
                if (lane < static_cast<uint32_t>(K)) {
                    const size_t g = static_cast<size_t>(t) * K + lane;
                    const int id = load_expert_id(p.topk_idx, p.idx_is_i64, g);
                    int row = -1;
                    if (id >= 0 && id < E && s_rank_ok[id / El]) {
                        const int d = id / El, slot = p.slot_in_expert[g];
                        row = s_aux[id] + slot;
                        p.send_list[s_hist[id] + slot] = make_int4(t, d, row, (id - d * El) | (static_cast<int>(lane) << 16));
                    }
                    p.send_row[g] = row;
                }
            }
        } else {
        for (int t = t0 + warp; t < t1; t += kDispWarps) {
            const __nv_bfloat16* xrow = p.x + static_cast<size_t>(t) * p.h;
            if (bulk_rows) {
                if (lane < static_cast<uint32_t>(K)) bulk_wait_group_read<0>();  // staging is free again
                __syncwarp();
            }
            if (p.quant_mode == CAM_QUANT_FP8_1x128) {
                warp_quant_fp8_1x128<false>(xrow, p.h, stage_q, stage_s);
            } else if (p.quant_mode == CAM_QUANT_FP8_1x128_UE8M0) {
                warp_quant_fp8_1x128<true>(xrow, p.h, stage_q, stage_s);
            } else if (p.quant_mode == CAM_QUANT_INT8_TOKEN) {
                warp_quant_int8_token(xrow, p.h, stage_q, stage_s);
            }
            __syncwarp();
            // pair of this lane
            int d = -1, row = -1;
            if (lane < static_cast<uint32_t>(K)) {
                const size_t g = static_cast<size_t>(t) * K + lane;
                const int id = load_expert_id(p.topk_idx, p.idx_is_i64, g);
                if (id >= 0 && id < E && s_rank_ok[id / El]) {
                    d = id / El;
                    row = s_aux[id] + p.slot_in_expert[g];
                }
                p.send_row[g] = row;
            }
            // rows for this rank's own experts are written directly (local stores cost less than a copy pass)
            const uint32_t peers =
                __match_any_sync(0xFFFFFFFFu, (d >= 0 && d != p.rank) ? d : -1 - static_cast<int>(lane));
            const int first = __ffs(static_cast<int>(peers)) - 1;
            const int first_row = __shfl_sync(0xFFFFFFFFu, row, first);
            const bool sends = d >= 0 && static_cast<int>(lane) == first;
            if (d >= 0) {
                uint8_t* pb = p.peer_base[d];
                int* tri = reinterpret_cast<int*>(pb + p.off_recv_src) + static_cast<size_t>(row) * 3;
                tri[0] = p.rank;
                tri[1] = t;
                tri[2] = static_cast<int>(lane);
                if (!sends) {
                    const unsigned int idx = atomicAdd(&p.dup_ctr[d], 1u);
                    int* ent = reinterpret_cast<int*>(pb + p.off_dup_list) +
                               ((static_cast<size_t>(parity) * R + p.rank) * p.dup_cap + idx) * 2;
                    st_na_v2(ent, make_uint2(static_cast<uint32_t>(first_row), static_cast<uint32_t>(row)));
                }
            }
            if (bulk_rows) {
                fence_proxy_async_smem();  // the staged row is read by the async proxy
                __syncwarp();
                if (sends) {
                    uint8_t* pb = p.peer_base[d];
                    bulk_store_s2g(pb + p.off_recv_x + static_cast<size_t>(row) * row_bytes, stage_q,
                                   static_cast<uint32_t>(row_bytes));
                    float* sdst = reinterpret_cast<float*>(pb + p.off_recv_scales) + static_cast<size_t>(row) * nscale;
                    if (bulk_scales) {
                        bulk_store_s2g(sdst, stage_s, static_cast<uint32_t>(nscale * 4));
                    } else {
                        for (int o = 0; o < nscale; ++o) sdst[o] = stage_s[o];
                    }
                }
                if (lane < static_cast<uint32_t>(K)) bulk_commit_group();
                __syncwarp();
                continue;
            }
            const uint32_t senders = __ballot_sync(0xFFFFFFFFu, sends);
            for (uint32_t m = senders; m != 0u; m &= m - 1u) {
                const int k = __ffs(static_cast<int>(m)) - 1;
                const int dk = __shfl_sync(0xFFFFFFFFu, d, k);
                const int rk = __shfl_sync(0xFFFFFFFFu, row, k);
                uint8_t* pb = p.peer_base[dk];
                uint8_t* dst = pb + p.off_recv_x + static_cast<size_t>(rk) * row_bytes;
                if (p.quant_mode == CAM_QUANT_NONE) {
                    warp_copy_row<false>(dst, reinterpret_cast<const uint8_t*>(xrow), row_bytes, lane);
                } else {
                    for (int o = static_cast<int>(lane) * 16; o < row_bytes; o += 512)
                        st_na_v4(dst + o, *reinterpret_cast<const uint4*>(stage_q + o));
                    float* sdst = reinterpret_cast<float*>(pb + p.off_recv_scales) + static_cast<size_t>(rk) * nscale;
                    for (int o = static_cast<int>(lane); o < nscale; o += 32) sdst[o] = stage_s[o];
                }
            }
            __syncwarp();
        }

        // Completion: the last CTA to finish raises this rank's data flag in every peer.
        if (bulk_rows && lane < static_cast<uint32_t>(K)) bulk_wait_group<0>();  // this lane's copies are written
        __syncthreads();
        if (!solo && tid == 0) {
            __threadfence_system();
            const unsigned int old = atomicAdd(p.done_ctr, 1u);
            if (old == static_cast<unsigned int>(nb - 1)) {
                p.done_ctr[0] = 0u;
                __threadfence_system();
                for (int d = 0; d < R; ++d) {  // length of the replicate list this rank wrote at d, then reset the cursor
                    const unsigned int n = atomicExch(&p.dup_ctr[d], 0u);
                    reinterpret_cast<uint32_t*>(p.peer_base[d] + p.off_dup_cnt)[parity * CAM_MAX_RANKS + p.rank] = n;
                }
                __threadfence_system();
                if (p.dbg_drop_flags == 0) {
                    for (int d = 0; d < R; ++d)
                        st_release_sys_u32(reinterpret_cast<uint32_t*>(p.peer_base[d] + p.off_data_flag) + p.rank,
                                           ep_send);
                }
            }
        }
        }  // !defer_push
    }

    // ------------------------------------------------------------------ phase RECV
    if ((p.phase_mask & CAM_PHASE_RECV) && !solo) {
        const int parity = static_cast<int>(ep_recv & 1u);
        if (tid < R) {
            const uint32_t* f = reinterpret_cast<const uint32_t*>(my_base + p.off_data_flag) + tid;
            const uint64_t t_wait = (b == 0 && p.stats != nullptr) ? globaltimer_ns() : 0ull;
            if (!wait_flag_eq_sys(f, ep_recv, p.timeout_ns)) {
                record_status(p.status, CAM_ERR_TIMEOUT_DATA_FLAG, tid, static_cast<int>(ld_acquire_sys_u32(f)));
                s_abort = 1u;
            }
            if (b == 0 && p.stats != nullptr) atomicMax(&p.stats->max_wait_ns[1][tid], globaltimer_ns() - t_wait);
        }
        __syncthreads();
        if (s_abort) goto done;
        // Replicate: rows that several local experts need arrived once; copy them to the other rows.
        if (tid == 0) {
            const uint32_t* cnt = reinterpret_cast<const uint32_t*>(my_base + p.off_dup_cnt) + parity * CAM_MAX_RANKS;
            int run = 0;
            for (int s = 0; s < R; ++s) {
                s_dup_pre[s] = run;
                run += static_cast<int>(min(__ldcg(cnt + s), static_cast<uint32_t>(p.dup_cap)));
            }
            s_dup_pre[R] = run;
        }
        __syncthreads();
        const int nscale = CAM_QUANT_IS_FP8(p.quant_mode) ? (p.h >> 7) : (p.quant_mode == CAM_QUANT_INT8_TOKEN) ? 1 : 0;
        const int row_bytes = (p.quant_mode == CAM_QUANT_NONE) ? p.h * 2 : p.h;
        const int warp = tid >> 5;
        const uint32_t lane = lane_id();
        const int total = s_dup_pre[R];
        uint8_t* rx = my_base + p.off_recv_x;
        float* rs = reinterpret_cast<float*>(my_base + p.off_recv_scales);
        for (int i = b * kDispWarps + warp; i < total; i += nb * kDispWarps) {
            int s = 0;
            while (s + 1 < R && s_dup_pre[s + 1] <= i) ++s;
            const int* ent = reinterpret_cast<const int*>(my_base + p.off_dup_list) +
                             ((static_cast<size_t>(parity) * R + s) * p.dup_cap + (i - s_dup_pre[s])) * 2;
            const int from = __ldcg(ent), to = __ldcg(ent + 1);
            if (from < 0 || to < 0 || from >= p.capacity || to >= p.capacity) {  // never copy out of range
                if (lane == 0) record_status(p.status, CAM_ERR_BAD_INDEX, 2, i);
                continue;
            }
            warp_copy_row<true>(rx + static_cast<size_t>(to) * row_bytes, rx + static_cast<size_t>(from) * row_bytes,
                                row_bytes, lane);
            for (int o = static_cast<int>(lane); o < nscale; o += 32)
                rs[static_cast<size_t>(to) * nscale + o] = __ldcg(rs + static_cast<size_t>(from) * nscale + o);
        }
    }

done:
    if ((p.phase_mask & CAM_PHASE_RECV) && p.nums_out != nullptr && b == 0) {  // CTA 0 wrote the counts (this launch or an earlier one)
        __syncthreads();
        for (int le = tid; le < p.nums_len; le += kDispThreads) p.nums_out[le] = __ldcg(reinterpret_cast<const long long*>(p.num_recv_per_expert) + le);
    }
    // the CTA that leaves last advances the epochs of the phases this launch ran
    __syncthreads();
    if (tid == 0 && last_cta_out(p.exit_ctr, static_cast<unsigned int>(nb))) {
        if (p.phase_mask & CAM_PHASE_COUNT) p.epochs[0] = ep_count;
        if (p.phase_mask & CAM_PHASE_SEND) p.epochs[1] = ep_send;
        if (p.phase_mask & CAM_PHASE_RECV) p.epochs[2] = ep_recv;
        // a deferred push has no receive phase of its own: keep the three counters in step for the next plain dispatch
        if (p.defer_push && (p.phase_mask & CAM_PHASE_SEND)) p.epochs[2] = ep_send;
    }
}

// ----------------------------------------------------------------------------------------
// Stand-alone layout kernel (the reference's dispatch_layout op,
// ascend_kernels/dispatch_layout/op_kernel/dispatch_layout.h:83-134).  Negative ids are skipped.
// ----------------------------------------------------------------------------------------
__global__ void layout_kernel(const void* topk_idx, int idx_is_i64, int T, int K, int E, int R,
                              int* num_tokens_per_rank, int* num_tokens_per_expert,
                              uint8_t* is_token_in_rank) {
    static_assert(CAM_MAX_RANKS <= 128, "the ranks a token goes to are tracked in two 64-bit masks");
    __shared__ int s_rank[CAM_MAX_RANKS];
    __shared__ int s_exp[CAM_MAX_EXPERTS];
    for (int i = threadIdx.x; i < R; i += blockDim.x) s_rank[i] = 0;
    for (int i = threadIdx.x; i < E; i += blockDim.x) s_exp[i] = 0;
    __syncthreads();
    const int El = E / R;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
        unsigned long long seen_lo = 0ull, seen_hi = 0ull;  // ranks 0..63 and 64..127
        for (int k = 0; k < K; ++k) {
            const int id = load_expert_id(topk_idx, idx_is_i64, static_cast<size_t>(t) * K + k);
            if (id < 0 || id >= E) continue;
            atomicAdd(&s_exp[id], 1);
            const int r = id / El;
            if (r < 64) seen_lo |= 1ull << r; else seen_hi |= 1ull << (r - 64);
        }
        for (int r = 0; r < R; ++r) {
            const bool in = (r < 64) ? ((seen_lo >> r) & 1ull) : ((seen_hi >> (r - 64)) & 1ull);
            is_token_in_rank[static_cast<size_t>(t) * R + r] = in ? 1 : 0;
            if (in) atomicAdd(&s_rank[r], 1);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < R; i += blockDim.x) if (s_rank[i]) atomicAdd(&num_tokens_per_rank[i], s_rank[i]);
    for (int i = threadIdx.x; i < E; i += blockDim.x) if (s_exp[i]) atomicAdd(&num_tokens_per_expert[i], s_exp[i]);
}

// Zeroes the counters the kernel above adds to (one launch; a memset node in a graph costs as much as two).
__global__ void layout_zero_kernel(int* num_tokens_per_rank, int R, int* num_tokens_per_expert, int E) {
    for (int i = threadIdx.x; i < R; i += blockDim.x) num_tokens_per_rank[i] = 0;
    for (int i = threadIdx.x; i < E; i += blockDim.x) num_tokens_per_expert[i] = 0;
}

// The same in ONE launch without zeroed outputs, for batches of ordinary size: a cluster of kLayoutCtas CTAs counts in
// shared memory, and after a cluster barrier every CTA adds up its share of the counters over the cluster's shared memories.
// The call is bound by launches (2.5 us of host time each beside 6 us of allocations and dispatch), not by the 64 bytes per
// token it reads, as long as every thread has few tokens, ids and ranks: 4096 tokens x 8 ids, 8 ranks take 9.0 us per call
// (5.4 on the device) against 11.5 (4.6) for the two launches above, 8192 tokens 10.2 (7.5) against 11.4 (4.6).  The few CTAs
// lose beyond that: 16384 tokens (8 ids, 8 ranks) took 16.6 us against 11.4, 4096 tokens x 16 ids 12.3 against 11.4, 64 ranks 33
// against 21.  (Three fills and the kernel: 22 to 27 us.)
constexpr int kLayoutCtas = 8, kLayoutThreads = 512, kLayoutClusterTokens = 2 * kLayoutCtas * kLayoutThreads;
constexpr int kLayoutClusterIds = 8, kLayoutClusterRanks = 8;

__global__ void __cluster_dims__(kLayoutCtas, 1, 1) __launch_bounds__(kLayoutThreads)
layout_cluster_kernel(const void* topk_idx, int idx_is_i64, int T, int K, int E, int R, int* num_tokens_per_rank,
                      int* num_tokens_per_expert, uint8_t* is_token_in_rank) {
    __shared__ int s_cnt[CAM_MAX_EXPERTS + kLayoutClusterRanks];  // per expert, then per rank
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = static_cast<int>(threadIdx.x), rank = static_cast<int>(cluster.block_rank());
    const int n = E + R, El = E / R;
    // two 64-bit ids per load where rows allow it: 8 ids per token are 64 bytes, a cache line for every other lane
    const bool pairs = idx_is_i64 && (K & 1) == 0 && (reinterpret_cast<uintptr_t>(topk_idx) & 15u) == 0u;
    int id[2][kLayoutClusterIds];  // both tokens' ids are in flight before the first is counted
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int t = (u * kLayoutCtas + rank) * kLayoutThreads + tid;
        if (pairs) {
#pragma unroll
            for (int k = 0; k < kLayoutClusterIds; k += 2) {
                const longlong2 v = (t < T && k < K) ? __ldg(reinterpret_cast<const longlong2*>(topk_idx) +
                                                             (static_cast<size_t>(t) * K + k) / 2)
                                                     : make_longlong2(-1, -1);
                id[u][k] = (v.x >= 0 && v.x < E) ? static_cast<int>(v.x) : -1;
                id[u][k + 1] = (v.y >= 0 && v.y < E) ? static_cast<int>(v.y) : -1;
            }
            continue;
        }
#pragma unroll
        for (int k = 0; k < kLayoutClusterIds; ++k)
            id[u][k] = (t < T && k < K) ? load_expert_id(topk_idx, idx_is_i64, static_cast<size_t>(t) * K + k) : -1;
    }
    for (int i = tid; i < n; i += kLayoutThreads) s_cnt[i] = 0;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int t = (u * kLayoutCtas + rank) * kLayoutThreads + tid;  // whole warps stay together: some lanes may be past T
        if (t - (tid & 31) >= T) break;
        uint32_t seen = 0u;
#pragma unroll
        for (int k = 0; k < kLayoutClusterIds; ++k) {
            if (id[u][k] < 0 || id[u][k] >= E) continue;
            atomicAdd(&s_cnt[id[u][k]], 1);
            seen |= 1u << (id[u][k] / El);
        }
        for (int r = 0; r < R; ++r) {
            const bool in = (seen >> r) & 1u;
            if (t < T && R != 8) is_token_in_rank[static_cast<size_t>(t) * R + r] = in ? 1 : 0;
            const uint32_t all = __ballot_sync(0xFFFFFFFFu, in);  // one atomic per warp: few ranks, many tokens
            if ((tid & 31) == 0 && all != 0u) atomicAdd(&s_cnt[E + r], __popc(all));
        }
        if (t < T && R == 8) {  // bit r of `seen` into byte r: one store instead of eight
            uint32_t lo = 0u, hi = 0u;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                lo |= ((seen >> r) & 1u) << (8 * r);
                hi |= ((seen >> (r + 4)) & 1u) << (8 * r);
            }
            *reinterpret_cast<uint2*>(is_token_in_rank + static_cast<size_t>(t) * 8) = make_uint2(lo, hi);
        }
    }
    cluster.sync();
    for (int i = rank * kLayoutThreads + tid; i < n; i += kLayoutCtas * kLayoutThreads) {
        int sum = 0;
#pragma unroll
        for (int c = 0; c < kLayoutCtas; ++c) sum += cluster.map_shared_rank(s_cnt, c)[i];
        if (i < E) num_tokens_per_expert[i] = sum; else num_tokens_per_rank[i - E] = sum;
    }
    cluster.sync();  // no CTA leaves while others read its counters
}

}  // namespace cam

// ----------------------------------------------------------------------------------------
// Launchers (C ABI)
// ----------------------------------------------------------------------------------------
// Staging rows of the push; the slot table of the count phase and the key counts of the deferred push use the same bytes.
extern "C" int cam_dispatch_normal_smem_bytes(int h, int quant_mode) {
    const int table = cam::kDispTableBytes;  // also holds the ids and four staged rows of a small one-rank call, see below
    if (quant_mode == CAM_QUANT_NONE) return table;
    const int nscale = CAM_QUANT_IS_FP8(quant_mode) ? h / 128 : 1;
    const int staging = cam::kDispWarps * ((h + nscale * 4 + 15) & ~15);
    return staging > table ? staging : table;
}

extern "C" int cam_launch_dispatch_normal(const cam::DispatchNormalParams* p, int grid, cudaStream_t stream) {
    const int smem = cam_dispatch_normal_smem_bytes(p->h, p->quant_mode);
    static cam::SmemLimitCache limit;
    cudaError_t e = limit.ensure(cam::dispatch_normal_kernel, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    void* args[] = {const_cast<cam::DispatchNormalParams*>(p)};
    e = cudaLaunchCooperativeKernel(reinterpret_cast<void*>(cam::dispatch_normal_kernel), dim3(grid),
                                    dim3(cam::kDispThreads), args, smem, stream);
    return static_cast<int>(e);
}

extern "C" int cam_launch_layout(const void* topk_idx, int idx_is_i64, int T, int K, int E, int R,
                                 int* num_tokens_per_rank, int* num_tokens_per_expert,
                                 uint8_t* is_token_in_rank, cudaStream_t stream) {
    const bool aligned = (reinterpret_cast<uintptr_t>(is_token_in_rank) & 7u) == 0u;  // eight ranks' bytes in one store
    if (T <= cam::kLayoutClusterTokens && K <= cam::kLayoutClusterIds && R <= cam::kLayoutClusterRanks && aligned) {
        cam::layout_cluster_kernel<<<cam::kLayoutCtas, cam::kLayoutThreads, 0, stream>>>(
            topk_idx, idx_is_i64, T, K, E, R, num_tokens_per_rank, num_tokens_per_expert, is_token_in_rank);
        return static_cast<int>(cudaGetLastError());
    }
    cam::layout_zero_kernel<<<1, 512, 0, stream>>>(num_tokens_per_rank, R, num_tokens_per_expert, E);
    const int threads = 256;
    int blocks = (T + threads - 1) / threads;
    const int cap = 4 * cam::sm_count_of_current_device();  // the kernel strides over the tokens
    if (blocks > cap) blocks = cap;
    cam::layout_kernel<<<blocks, threads, 0, stream>>>(topk_idx, idx_is_i64, T, K, E, R, num_tokens_per_rank,
                                                       num_tokens_per_expert, is_token_in_rank);
    return static_cast<int>(cudaGetLastError());
}
