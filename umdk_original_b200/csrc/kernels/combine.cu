// Combine for sm_100a: every expert-output row is pushed with P2P stores into the (token, k)
// slot of its origin rank, a per-source completion flag follows, and the origin fuses the
// top-k weighted sum in fp32 (k order) with a round-to-nearest bf16 store.
//
// Same data flow as the reference's moe_combine_normal
// (ascend_kernels/moe_combine_normal/op_kernel/moe_combine_normal.h:211-374) and, with the row
// table that low-latency dispatch keeps, as moe_combine_shmem (moe_combine_shmem.h:919-930);
// the per-(token,k) float flags summed by a vector reduce become one integer epoch flag per
// source rank, raised once by the last CTA of the sender.  Pairs whose expert id is negative
// are skipped instead of waited for.
//
// comm_quant = 2 sends a row as int8 with one fp32 scale per 128 elements (h + h/32 bytes instead
// of 2 h) and dequantises inside the reduce: the counterpart of the reference's commQuantMode 2
// (moe_combine_shmem.h:567-591 quantises per 8 elements; 128 keeps the scales at 3 % of the row).
#include "../common/cam_types.h"
#include "../common/ptx.cuh"
#include "../common/quant.cuh"
#include "launch.h"

namespace cam {

constexpr int kCombThreads = 512;
constexpr int kCombWarps = kCombThreads / 32;

__device__ __forceinline__ void comb_record_status(CamStatus* st, int code, int who, int detail) {
    if (atomicCAS(&st->code, 0, code) == 0) {
        st->who = who;
        st->detail = detail;
        st->block = static_cast<int>(blockIdx.x);
    }
}

__device__ __forceinline__ void fma_bf16x8(float (&acc)[8], const uint4& v, float w) {
    acc[0] = fmaf(w, bf16_lo(v.x), acc[0]);
    acc[1] = fmaf(w, bf16_hi(v.x), acc[1]);
    acc[2] = fmaf(w, bf16_lo(v.y), acc[2]);
    acc[3] = fmaf(w, bf16_hi(v.y), acc[3]);
    acc[4] = fmaf(w, bf16_lo(v.z), acc[4]);
    acc[5] = fmaf(w, bf16_hi(v.z), acc[5]);
    acc[6] = fmaf(w, bf16_lo(v.w), acc[6]);
    acc[7] = fmaf(w, bf16_hi(v.w), acc[7]);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
}

// INT8_WIRE: comm_quant 2.  IN_PLACE: rows whose origin is this rank do not move; one launch sends and reduces.  Kernels of their
// own, so that no form takes part in the register allocation of another (int8 with both ways of its rows in one kernel: 16 tokens
// x 2 of 1024, pushed, 12.9 us against 12.0).
template <bool INT8_WIRE, bool IN_PLACE>
__global__ void __launch_bounds__(kCombThreads, 1) combine_kernel(const CombineParams p) {
    __shared__ uint32_t s_abort;
    __shared__ float s_w[kCombWarps][CAM_MAX_TOPK];
    __shared__ uint64_t s_row[kCombWarps][CAM_MAX_TOPK];  // where the row of pair (t, k) is read from
    const int tid = static_cast<int>(threadIdx.x);
    const int warp = tid >> 5;
    const uint32_t lane = lane_id();
    const int nb = static_cast<int>(gridDim.x);
    const int gwarp = static_cast<int>(blockIdx.x) * kCombWarps + warp;
    const int nwarps = nb * kCombWarps;
    const int row_bytes = p.h * 2;
    const uint32_t ep_send = p.epochs[0] + 1u, ep_recv = p.epochs[1] + 1u;
    // Rows whose origin is this rank do not move when one launch sends and reduces: the send phase notes {epoch, row}
    // per (token, k) pair, 8 bytes instead of a row written and read again, and the reduce gathers straight from y.
    // The epoch tells this launch's entries from those of earlier ones.
    // Bound by memory traffic: 4096 tokens x 8 rows of 14 KB on one GPU took 263 us with every row copied to its slot first
    // (1.47 GB moved), 102 us with the rows gathered in place (0.53 GB, 5.2 TB/s).
    constexpr bool in_place = IN_PLACE;
    if (tid == 0) s_abort = 0u;
    __syncthreads();

    trace_point(p.trace, 0);  // kernel start
    // ------------------------------------------------------------------ SEND
    if (p.phase_mask & CAM_PHASE_SEND) {
        const int n = min(p.total_rows[0], p.max_rows);
        if (in_place) {  // one thread per row
            for (int i = static_cast<int>(blockIdx.x) * kCombThreads + tid; i < n; i += nb * kCombThreads) {
                const int src = p.row_src[static_cast<size_t>(i) * 3 + 0];
                const int t = p.row_src[static_cast<size_t>(i) * 3 + 1];
                const int k = p.row_src[static_cast<size_t>(i) * 3 + 2];
                if (src < 0 || src >= p.R || t < 0 || t >= p.max_tokens || k < 0 || k >= p.K)
                    comb_record_status(p.status, CAM_ERR_BAD_INDEX, 1, i);
                else if (src == p.rank)
                    p.local_row[static_cast<size_t>(t) * p.K + k] =
                        (static_cast<uint64_t>(ep_send) << 32) | static_cast<uint32_t>(i);
            }
        }
        // Rows are ordered by expert and, inside an expert, by origin rank.  Every rank starts its walk somewhere else
        // (its share of the rows plus one grid-wide step per rank further on), so that at any one time the ranks of the
        // group push to different origins instead of all filling the same GPU's ingress.
        const int shift = (p.R > 1 && n > 0) ? static_cast<int>((static_cast<long long>(p.rank) * (n / p.R + nwarps)) % n) : 0;
        const int n_push = (in_place && p.R == 1) ? 0 : n;
        for (int i0 = gwarp; i0 < n_push; i0 += nwarps) {
            const int i = (i0 + shift < n) ? i0 + shift : i0 + shift - n;
            const int src = p.row_src[static_cast<size_t>(i) * 3 + 0];
            const int t = p.row_src[static_cast<size_t>(i) * 3 + 1];
            const int k = p.row_src[static_cast<size_t>(i) * 3 + 2];
            if (src < 0 || src >= p.R || t < 0 || t >= p.max_tokens || k < 0 || k >= p.K) {
                // never store out of range: the row is dropped and the status word says which one it was
                if (lane == 0) comb_record_status(p.status, CAM_ERR_BAD_INDEX, 1, i);
                continue;
            }
            if (in_place && src == p.rank) continue;
            const uint8_t* s = reinterpret_cast<const uint8_t*>(p.y) + static_cast<size_t>(i) * row_bytes;
            uint8_t* d = p.peer_base[src] + p.off_combine_buf +
                         (static_cast<size_t>(t) * p.K + k) * static_cast<size_t>(row_bytes);
            if constexpr (INT8_WIRE) {
                // int8 on the wire: lane owns 8 elements per step of 256, 16 lanes share a 128-element block
                float* dscale = reinterpret_cast<float*>(d + p.h);
                for (int base = 0; base < p.h; base += 1024) {
                    uint4 v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int c = base + u * 256 + static_cast<int>(lane) * 8;
                        v[u] = (c < p.h) ? ld_nc_v4(s + static_cast<size_t>(c) * 2) : make_uint4(0, 0, 0, 0);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int c = base + u * 256 + static_cast<int>(lane) * 8;
                        float f[8] = {bf16_lo(v[u].x), bf16_hi(v[u].x), bf16_lo(v[u].y), bf16_hi(v[u].y),
                                      bf16_lo(v[u].z), bf16_hi(v[u].z), bf16_lo(v[u].w), bf16_hi(v[u].w)};
                        float amax = 0.f;
#pragma unroll
                        for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(f[j]));
#pragma unroll
                        for (int sft = 8; sft >= 1; sft >>= 1)
                            amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, sft));
                        const float a = fmaxf(amax, 1e-12f);
                        const float inv = 127.f / a;
                        uint32_t w0 = 0u, w1 = 0u;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            w0 |= (static_cast<uint32_t>(__float2int_rn(f[j] * inv)) & 0xFFu) << (8 * j);
                            w1 |= (static_cast<uint32_t>(__float2int_rn(f[4 + j] * inv)) & 0xFFu) << (8 * j);
                        }
                        if (c < p.h) {
                            st_na_v2(d + c, make_uint2(w0, w1));
                            if ((lane & 15u) == 0u) dscale[c >> 7] = a / 127.f;
                        }
                    }
                }
                continue;
            }
            int o = static_cast<int>(lane) * 16;
            for (; o + 3 * 512 < row_bytes; o += 4 * 512) {
                const uint4 a = ld_nc_v4(s + o), b4 = ld_nc_v4(s + o + 512), c = ld_nc_v4(s + o + 1024),
                            e = ld_nc_v4(s + o + 1536);
                st_na_v4(d + o, a);
                st_na_v4(d + o + 512, b4);
                st_na_v4(d + o + 1024, c);
                st_na_v4(d + o + 1536, e);
            }
            for (; o < row_bytes; o += 512) st_na_v4(d + o, ld_nc_v4(s + o));
        }
        __syncthreads();
        trace_point(p.trace, 1);  // this CTA's rows are issued
        if (tid == 0) {
            __threadfence_system();
            if (p.trace != nullptr && blockIdx.x == 0) p.trace[2] = globaltimer_ns();  // system fence done
            const unsigned int old = atomicAdd(p.done_ctr, 1u);
            if (old == static_cast<unsigned int>(nb - 1)) {
                p.done_ctr[0] = 0u;
                __threadfence_system();
                if (p.dbg_drop_flags == 0) {
                    for (int d = 0; d < p.R; ++d)
                        st_release_sys_u32(
                            reinterpret_cast<uint32_t*>(p.peer_base[d] + p.off_combine_flag) + p.rank, ep_send);
                }
            }
        }
    }

    // ------------------------------------------------------------------ RECV
    if (p.phase_mask & CAM_PHASE_RECV) {
        uint8_t* const my_base = p.peer_base[p.rank];
        if (tid < p.R) {
            const uint32_t* f = reinterpret_cast<const uint32_t*>(my_base + p.off_combine_flag) + tid;
            const bool keep = blockIdx.x == 0 && p.stats != nullptr;
            const uint64_t t_wait = keep ? globaltimer_ns() : 0ull;
            if (!wait_flag_eq_sys(f, ep_recv, p.timeout_ns)) {
                comb_record_status(p.status, CAM_ERR_TIMEOUT_COMBINE_FLAG, tid,
                                   static_cast<int>(ld_acquire_sys_u32(f)));
                s_abort = 1u;
            }
            if (keep) {
                atomicMax(&p.stats->max_wait_ns[2][tid], globaltimer_ns() - t_wait);
                if (tid == 0) atomicAdd(&p.stats->calls[1], 1ull);
            }
        }
        __syncthreads();
        trace_point(p.trace, 3);  // all sources' flags have arrived
        if (s_abort) goto done;

        const uint8_t* buf = my_base + p.off_combine_buf;
        // Weight, source address and presence of the pairs of token t, for this warp; bit k of the result: pair has a row.
        // Bit 0 of an address (rows are 16-byte aligned) marks a row of y.
        auto load_pairs = [&](int t) -> uint32_t {
            bool pair_ok = false;
            if (lane < static_cast<uint32_t>(p.K)) {
                const size_t g = static_cast<size_t>(t) * p.K + lane;
                const int id = load_expert_id(p.topk_idx, p.idx_is_i64, g);
                s_w[warp][lane] = p.topk_weights[g];
                uint64_t from = reinterpret_cast<uint64_t>(buf + g * row_bytes);
                if (in_place) {
                    const uint64_t ent = __ldcg(reinterpret_cast<const unsigned long long*>(p.local_row) + g);
                    const bool here = static_cast<uint32_t>(ent >> 32) == ep_send;
                    if (!here && p.R == 1) from = 0ull;  // no row of this call names the pair, and none can come from elsewhere
                    if (here)
                        from = (reinterpret_cast<uint64_t>(p.y) +
                                static_cast<uint64_t>(static_cast<uint32_t>(ent)) * static_cast<uint64_t>(row_bytes)) | 1ull;
                }
                s_row[warp][lane] = from;
                pair_ok = (id >= 0 && id < p.E && from != 0ull);
            }
            const uint32_t valid = __ballot_sync(0xFFFFFFFFu, pair_ok);
            __syncwarp();
            return valid;
        };
        if constexpr (INT8_WIRE) {
            // rows arrived as int8 + one scale per 128 elements; a lane reduces 16 elements per step
            const int chunks_q = (p.h + 511) / 512;
            const int nsplit_q = min(chunks_q, max(1, nwarps / max(p.T, 1)));
            const int per_q = (chunks_q + nsplit_q - 1) / nsplit_q;
            for (int it = gwarp; it < p.T * nsplit_q; it += nwarps) {
                const int t = it / nsplit_q;
                const int e_begin = (it - t * nsplit_q) * per_q * 512;
                const int e_end = min(p.h, e_begin + per_q * 512);
                const uint32_t valid = load_pairs(t);
                uint8_t* orow = reinterpret_cast<uint8_t*>(p.out) + static_cast<size_t>(t) * row_bytes;
                for (int c = e_begin + static_cast<int>(lane) * 16; c < e_end; c += 512) {
                    float acc[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[j] = 0.f;
                    auto add_wire_row = [&](const uint4& q, float sc) {
                        const uint32_t wq[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const int b8 = static_cast<int>(static_cast<int8_t>((wq[j >> 2] >> (8 * (j & 3))) & 0xFFu));
                            acc[j] = fmaf(sc, static_cast<float>(b8), acc[j]);
                        }
                    };
                    // rows from the slots: the loads of four are in flight before the first is added
                    for (int k0 = 0; !in_place && k0 < p.K; k0 += 4) {
                        uint4 q[4];
                        float sc[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int k = k0 + u;
                            if (k >= p.K || !((valid >> k) & 1u)) continue;
                            const uint8_t* krow = reinterpret_cast<const uint8_t*>(s_row[warp][k]);
                            q[u] = ld_cg_v4(krow + c);
                            sc[u] = __ldcg(reinterpret_cast<const float*>(krow + p.h) + (c >> 7));
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int k = k0 + u;
                            if (k >= p.K || !((valid >> k) & 1u)) continue;
                            add_wire_row(q[u], sc[u] * s_w[warp][k]);
                        }
                    }
                    if constexpr (IN_PLACE) {  // the next row's loads are in flight while a row is quantised
                        uint4 n0 = make_uint4(0, 0, 0, 0), n1 = n0;
                        auto fetch = [&](int k) {  // a row of y as it is, a row from the slots with its scale in n1.x
                            if (k >= p.K || !((valid >> k) & 1u)) return;
                            const uint64_t from = s_row[warp][k];
                            if (from & 1ull) {
                                const uint8_t* yrow = reinterpret_cast<const uint8_t*>(from & ~1ull) + static_cast<size_t>(c) * 2;
                                n0 = ld_cg_v4(yrow);
                                n1 = ld_cg_v4(yrow + 16);
                            } else {
                                const uint8_t* krow = reinterpret_cast<const uint8_t*>(from);
                                n0 = ld_cg_v4(krow + c);
                                n1.x = __float_as_uint(__ldcg(reinterpret_cast<const float*>(krow + p.h) + (c >> 7)));
                            }
                        };
                        fetch(0);
                        for (int k = 0; k < p.K; ++k) {
                            const uint4 y0 = n0, y1 = n1;
                            fetch(k + 1);
                            if (!((valid >> k) & 1u)) continue;
                            if (!(s_row[warp][k] & 1ull)) {
                                add_wire_row(y0, __uint_as_float(y1.x) * s_w[warp][k]);
                                continue;
                            }
                            // a row of y: quantised to the wire format here (8 lanes hold a 128-element block), so that
                            // a row counts the same whether it travelled or not
                            const float f[16] = {bf16_lo(y0.x), bf16_hi(y0.x), bf16_lo(y0.y), bf16_hi(y0.y),
                                                 bf16_lo(y0.z), bf16_hi(y0.z), bf16_lo(y0.w), bf16_hi(y0.w),
                                                 bf16_lo(y1.x), bf16_hi(y1.x), bf16_lo(y1.y), bf16_hi(y1.y),
                                                 bf16_lo(y1.z), bf16_hi(y1.z), bf16_lo(y1.w), bf16_hi(y1.w)};
                            float amax = 0.f;
#pragma unroll
                            for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(f[j]));
                            const uint32_t group = 0xFFu << (lane & 24u);  // h is a multiple of 128: all 8 lanes are here
#pragma unroll
                            for (int sft = 4; sft >= 1; sft >>= 1) amax = fmaxf(amax, __shfl_xor_sync(group, amax, sft));
                            const float a = fmaxf(amax, 1e-12f);
                            const float inv = 127.f / a;
                            const float sc = (a / 127.f) * s_w[warp][k];
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                acc[j] = fmaf(sc, static_cast<float>(static_cast<int>(static_cast<int8_t>(
                                                      static_cast<uint32_t>(__float2int_rn(f[j] * inv)) & 0xFFu))), acc[j]);
                        }
                    }
                    uint4 r0, r1;
                    r0.x = pack_bf16x2(acc[0], acc[1]);   r0.y = pack_bf16x2(acc[2], acc[3]);
                    r0.z = pack_bf16x2(acc[4], acc[5]);   r0.w = pack_bf16x2(acc[6], acc[7]);
                    r1.x = pack_bf16x2(acc[8], acc[9]);   r1.y = pack_bf16x2(acc[10], acc[11]);
                    r1.z = pack_bf16x2(acc[12], acc[13]); r1.w = pack_bf16x2(acc[14], acc[15]);
                    st_na_v4(orow + static_cast<size_t>(c) * 2, r0);
                    st_na_v4(orow + static_cast<size_t>(c) * 2 + 16, r1);
                }
                __syncwarp();
            }
            goto done;
        }
        // Work item = (token, slice of the row).  With few tokens (decode) a row is cut into as many
        // 512-byte-aligned slices as there are warps to spare, so the whole grid takes part.
        const int chunks = (row_bytes + 511) / 512;
        const int nsplit = min(chunks, max(1, nwarps / max(p.T, 1)));
        const int per = (chunks + nsplit - 1) / nsplit;
        for (int it = gwarp; it < p.T * nsplit; it += nwarps) {
            const int t = it / nsplit;
            const int o_begin = (it - t * nsplit) * per * 512;
            const int o_end = min(row_bytes, o_begin + per * 512);
            const uint32_t valid = load_pairs(t);
            uint8_t* orow = reinterpret_cast<uint8_t*>(p.out) + static_cast<size_t>(t) * row_bytes;
            if (p.K <= 8) {
                // The loads of the next 512 bytes of all rows are in flight while these are added up: with one batch at a
                // time a warp has nothing outstanding between its last load and the store (4096 tokens x 8 rows of 14 KB:
                // 102.6 -> 94.7 us, 5.6 TB/s).  The main loop is free of conditions: with the ends of the slice tested in it the
                // compiler may bring the two batches back into step (102.4 us).
                auto load8 = [&](uint4 (&v)[8], int o) {
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        v[k] = ((valid >> k) & 1u) ? ld_cg_v4(reinterpret_cast<const uint8_t*>(s_row[warp][k] & ~1ull) + o)
                                                   : make_uint4(0, 0, 0, 0);
                };
                auto add8 = [&](const uint4 (&v)[8], int o) {
                    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if ((valid >> k) & 1u) fma_bf16x8(acc, v[k], s_w[warp][k]);
                    uint4 r;
                    r.x = pack_bf16x2(acc[0], acc[1]);
                    r.y = pack_bf16x2(acc[2], acc[3]);
                    r.z = pack_bf16x2(acc[4], acc[5]);
                    r.w = pack_bf16x2(acc[6], acc[7]);
                    st_na_v4(orow + o, r);
                };
                uint4 va[8], vb[8];
                int o = o_begin + static_cast<int>(lane) * 16;
                if (o < o_end) load8(va, o);
                for (; o + 1024 < o_end; o += 1024) {
                    load8(vb, o + 512);
                    add8(va, o);
                    load8(va, o + 1024);
                    add8(vb, o + 512);
                }
                if (o < o_end) {
                    if (o + 512 < o_end) load8(vb, o + 512);
                    add8(va, o);
                    if (o + 512 < o_end) add8(vb, o + 512);
                }
                __syncwarp();
                continue;
            }
            for (int o = o_begin + static_cast<int>(lane) * 16; o < o_end; o += 512) {
                float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                for (int k0 = 0; k0 < p.K; k0 += 8) {
                    uint4 v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int k = k0 + j;
                        const bool ok = (k < p.K) && ((valid >> k) & 1u);
                        v[j] = ok ? ld_cg_v4(reinterpret_cast<const uint8_t*>(s_row[warp][k] & ~1ull) + o) : make_uint4(0, 0, 0, 0);
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int k = k0 + j;
                        if (k < p.K && ((valid >> k) & 1u)) fma_bf16x8(acc, v[j], s_w[warp][k]);
                    }
                }
                uint4 r;
                r.x = pack_bf16x2(acc[0], acc[1]);
                r.y = pack_bf16x2(acc[2], acc[3]);
                r.z = pack_bf16x2(acc[4], acc[5]);
                r.w = pack_bf16x2(acc[6], acc[7]);
                st_na_v4(orow + o, r);
            }
            __syncwarp();
        }
    }

done:
    __syncthreads();
    trace_point(p.trace, 4);  // CTA 0 reduced its tokens
    if (tid == 0 && last_cta_out(p.exit_ctr, static_cast<unsigned int>(nb))) {
        if (p.trace != nullptr) p.trace[5] = globaltimer_ns();  // the last CTA leaves
        if (p.phase_mask & CAM_PHASE_SEND) p.epochs[0] = ep_send;
        if (p.phase_mask & CAM_PHASE_RECV) p.epochs[1] = ep_recv;
    }
}

}  // namespace cam

extern "C" int cam_combine_max_grid(int device) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return -1;
    return sms;
}

extern "C" int cam_launch_combine(const cam::CombineParams* p, int grid, cudaStream_t stream) {
    void* args[] = {const_cast<cam::CombineParams*>(p)};
    // A launch that runs one phase only (the fused layer's reduce, whose rows the GEMM epilogue has pushed, and the phase-by-phase
    // harness) uses the slots.  With int8 rows the gathering warp quantises its 512-element slices of K rows one after the other,
    // where the push quantises every row in a warp of its own: in place only if that is no more than a row, and a long one
    // (device time, pushed and in place, one rank: 128 tokens x 8 of 7168 27.0 and 18.5 us, 61 x 6 of 5120 19.9 and 16.6, 64 x 8
    // of 4096 19.6 and 18.2, 64 x 4 of 2048 14.3 and 15.3, 64 x 9 of 1024 14.6 and 19.7, 16 x 2 of 1024 12.0 and 13.9).
    const bool int8 = p->comm_quant == 2;
    const bool in_place = p->local_row != nullptr && p->y != nullptr &&
                          (p->phase_mask & (CAM_PHASE_SEND | CAM_PHASE_RECV)) == (CAM_PHASE_SEND | CAM_PHASE_RECV) &&
                          (!int8 || (p->K * 512 <= p->h && p->h > 2048));
    void* const kernel = int8 ? (in_place ? reinterpret_cast<void*>(cam::combine_kernel<true, true>)
                                          : reinterpret_cast<void*>(cam::combine_kernel<true, false>))
                              : (in_place ? reinterpret_cast<void*>(cam::combine_kernel<false, true>)
                                          : reinterpret_cast<void*>(cam::combine_kernel<false, false>));
    return static_cast<int>(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(cam::kCombThreads), args, 0, stream));
}
