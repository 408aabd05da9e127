// Block-scaled grouped GEMM with the operands exchanged, for experts of up to a few hundred rows: the weights are the M
// operand of the tensor core and the rows of the expert its N operand, on CTA pairs (cta_group::2).
//
// What bounds the expert MLP there is the stream of weights (44 MB per DeepSeek-V3 expert for about 128 rows of work), so
// the form is chosen by what moves per weight byte.  tcgen05.mma fixes M but takes N in steps of 16: all rows of an expert
// (up to kTMaxRows = 224) are ONE tile of just as many columns as it has rows, every weight byte comes to the SMs once, and
// the tensor time follows the rows present.  With the rows as M operand (grouped_gemm_mx.cu) an expert of 130 rows is two
// 128-row tiles: its weights cross from L2 twice and half of the tensor work is padding.  A pair of CTAs shares the rows:
// each loads half of them and 256 weight rows of its own.  Larger experts are cut into equal tiles of at most 224 rows.
// Measured with 7168 x 2048 experts on one GPU: 256 experts x 128 rows, first GEMM 1.44 -> 1.27 ms (5.9 TB/s of weights),
// second 0.78 -> 0.70 ms; the layer in a steady loop, where the 1 kW limit holds the clock down and padded tensor work costs
// twice, 3.15 -> 2.62 ms; 4 rows per expert 2.15 -> 1.78 ms (6.9 TB/s).  A bare TMA read stream reaches 6.9 - 7.1 TB/s.
// Short reductions and few tiles are dearer here than on one CTA: cam_grouped_gemm_rows_n_pays in cam_runtime.cpp keeps those away.
//
// One tile: 512 weight rows (each CTA two blocks of 128: the gate and the up block of the same 128 features for the SwiGLU
// GEMM, two neighbouring blocks of output features otherwise) x N rows, K in steps of 128.  Tensor memory of each CTA
// (512 columns): accumulator of its first block in columns [0, 224), of its second in [224, 448), scale factors of pipeline
// stage s in [448 + 16 s, +16): 4 columns for each weight block, 8 for the rows (row n: lane n % 32, column n / 32).
//
// Barriers and roles are those of grouped_gemm_mx2.cu.  The accumulators hold the tile transposed (lane = feature, column =
// row), so the epilogue goes through shared memory: 64 rows of fp32 at a time for SwiGLU + requantisation (a row's 128
// features are one quantisation block and sit in one CTA), 128 rows of bf16 at a time for the outputs.
// Contract, modes and formats: see grouped_gemm_mx.cu.
//
// KIND selects the arithmetic; the pipeline is the same:
//   kRowsMx   block scaling by the tensor core (power-of-two scales), as above
//   kRowsI8   exact W8A8 (rowquant_i8.cu states the contract): int32 accumulators over the whole K, no scale factors in
//             tensor memory, so 256 rows per tile; the epilogue multiplies by the token scale (one per column) and the
//             channel scale (one per lane) first, and mode 1 writes fp32 activations and the row maxima
//             (128 experts of 4096 x 1536, 512 rows each: layer 1.86 -> 1.76 ms against 128-row tiles on one CTA)
#pragma once
#include "gemm_common.cuh"

namespace cam {

constexpr int kRowsMx = 0, kRowsI8 = 1;
constexpr int kMTEpiThreads = 512;
constexpr int kMTSfWarp0 = 4;
// warps 0..3 control, then (block scaling only) 4 scale-factor warps, then 16 epilogue warps
__host__ __device__ constexpr int rows_n_epi_warp0(int kind) { return kind == kRowsMx ? 8 : 4; }
__host__ __device__ constexpr int rows_n_threads(int kind) { return rows_n_epi_warp0(kind) * 32 + kMTEpiThreads; }
constexpr int kMTStages = 4;
// Rows of one tile: 2 x 224 accumulator columns + 4 x 16 scale-factor columns = 512, or 2 x 256 without scale factors.  The
// MMA takes rows in steps of 16 (block-scaled) and 32 (int8).
__host__ __device__ constexpr int rows_n_max(int kind) { return kind == kRowsMx ? 224 : 256; }
__host__ __device__ constexpr int rows_n_step(int kind) { return kind == kRowsMx ? 16 : 32; }
constexpr int kTRowBox = 32;              // rows of one TMA box of the row operand
constexpr int kMTWBytes = 2 * 128 * BK;   // two weight blocks
constexpr int kMTStgPitch = 272;
constexpr int kMTStgBytes = 128 * kMTStgPitch;
constexpr int kMTPitchF = 132;            // SwiGLU epilogue: floats between the staging rows of two rows
static_assert(64 * kMTPitchF * 4 <= kMTStgBytes, "fp32 staging of 64 rows must fit the staging area");
// Shared memory: pipeline stages (two weight blocks and half of the rows, at most 128, in boxes of 32) | staging | barriers.
constexpr int kMTStageBytes = kMTWBytes + 128 * BK;
constexpr int kMTSmem = kMTStages * kMTStageBytes + kMTStgBytes + 1024;
static_assert(kMTSmem <= 232448, "exceeds the shared memory of one CTA");
constexpr uint32_t kMTTmemCols = 512, kMTSfCol0 = 2 * rows_n_max(kRowsMx), kMTSfStride = 16;
static_assert(kMTSfCol0 + kMTStages * kMTSfStride <= kMTTmemCols, "tensor memory");
// setmaxnreg budget, see grouped_gemm_mx.cu: the shares must not add up to more than the CTA was launched with
// (kMTLaunchRegs per thread, stated by the including file and checked against ptxas by the build).
constexpr uint32_t kMTCtrlRegs = 32, kMTSfRegs = 64;
__host__ __device__ constexpr uint32_t rows_n_epi_regs(int kind) { return kind == kRowsMx ? 96 : 112; }
__host__ __device__ constexpr bool rows_n_regs_fit(int kind, uint32_t launch) {
    return 128 * kMTCtrlRegs + (kind == kRowsMx ? 128 * kMTSfRegs : 0) + kMTEpiThreads * rows_n_epi_regs(kind) <=
           launch * static_cast<uint32_t>(rows_n_threads(kind));
}

// Tiles of (expert, rows, weight blocks): the rows of an expert in ceil(rows / MAX) equal parts, multiples of STEP rows.
template <int MAX, int STEP>
struct RowTileWalker {
    const int* off;
    int num_experts, n_tiles;
    int e = 0, base = 0;
    __device__ RowTileWalker(const int* o, int ne, int nt) : off(o), num_experts(ne), n_tiles(nt) {}
    // rot_num / rot_den: as in TileWalkerT::locate
    __device__ bool locate(int tile, int& e_out, int& nt, int& row0, int& rows, int rot_num, int rot_den) {
        while (e < num_experts) {
            const int first = __ldg(off + e);
            const int cnt = __ldg(off + e + 1) - first;
            const int parts0 = (cnt + MAX - 1) / MAX;
            const int chunk = parts0 > 0 ? ((cnt + parts0 - 1) / parts0 + STEP - 1) & ~(STEP - 1) : STEP;
            const int parts = (cnt + chunk - 1) / chunk;  // <= parts0
            const int tiles = parts * n_tiles;
            if (tile < base + tiles) {
                const int local = tile - base;
                int mt = local / n_tiles;
                nt = local - mt * n_tiles;
                if (rot_den > 0) {
                    mt += rot_num * parts / rot_den;
                    if (mt >= parts) mt -= parts;
                }
                row0 = first + mt * chunk;
                rows = min(chunk, cnt - mt * chunk);
                e_out = e;
                return true;
            }
            base += tiles;
            ++e;
        }
        return false;
    }
};

template <int KIND, bool SWIGLU>  // SWIGLU: mode 1, otherwise modes 0 and 2
__global__ void __launch_bounds__(rows_n_threads(KIND), 1)
grouped_gemm_rows_n_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                           const GroupedGemmParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) {  // swizzled TMA tiles need it; the same in both CTAs of a pair
        if (threadIdx.x == 0) gemm_record_status(p.status, CAM_ERR_BAD_INDEX, 4, static_cast<int>(smem_u32(smem) & 1023u));
        return;
    }
    constexpr int NS = kMTStages;
    constexpr bool MX = KIND == kRowsMx, I8 = KIND == kRowsI8;
    static_assert(rows_n_regs_fit(KIND, kMTLaunchRegs), "setmaxnreg budget exceeds the registers the CTA owns: the kernel would hang");
    constexpr int STEP = rows_n_step(KIND);
    constexpr uint32_t ACC1 = static_cast<uint32_t>(rows_n_max(KIND));  // first column of the second accumulator
    constexpr int EPI0 = rows_n_epi_warp0(KIND);
    uint8_t* stg = smem + NS * kMTStageBytes;
    uint8_t* ctrl = stg + kMTStgBytes;
    uint64_t* bar_full = reinterpret_cast<uint64_t*>(ctrl);  // first CTA: TMA bytes of both CTAs' stage have landed
    uint64_t* bar_sf = bar_full + NS;                        // first CTA: scale factors of both CTAs are in TMEM
    uint64_t* bar_empty = bar_sf + NS;                       // each CTA: the MMAs that read a stage have retired
    uint64_t* bar_tfull = bar_empty + NS;                    // each CTA: accumulators of a tile are complete
    uint64_t* bar_tempty = bar_tfull + 1;                    // first CTA: both CTAs have drained their accumulators
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_tempty + 1);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = static_cast<int>(threadIdx.x) >> 5;
    const uint32_t lane = lane_id();
    const uint32_t cta = cluster_cta_rank();  // 0 = first CTA of the pair (issues the MMAs)
    const int pair_id = static_cast<int>(blockIdx.x) >> 1;
    const int num_pairs = static_cast<int>(gridDim.x) >> 1;
    const int kblocks = p.k_dim / BK;
    const int rot_num = (p.mode == 2 && p.num_ranks > 1) ? p.rank : 0, rot_den = (p.mode == 2 && p.num_ranks > 1) ? p.num_ranks : 0;
    const int nblk = p.n_dim / 128;                                     // weight blocks of an expert
    const int n_tiles = SWIGLU ? (nblk / 2 + 1) / 2 : (nblk + 3) / 4;
    // Weight blocks of this CTA in tile column nt.  Past the last block (feature blocks not a multiple of a tile's) the
    // last one is loaded again and its result is not stored.
    auto block_lo = [&](int nt) { return SWIGLU ? min(2 * nt + static_cast<int>(cta), nblk / 2 - 1) : min(4 * nt + 2 * static_cast<int>(cta), nblk - 1); };
    auto block_hi = [&](int nt) { return SWIGLU ? nblk / 2 + block_lo(nt) : min(4 * nt + 2 * static_cast<int>(cta) + 1, nblk - 1); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(&bar_full[s], 1);
            mbar_init(&bar_sf[s], 8);
            mbar_init(&bar_empty[s], 1);
        }
        mbar_init(bar_tfull, 1);
        mbar_init(bar_tempty, 2 * (kMTEpiThreads / 32));
        *abort_flag = 0u;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, kMTTmemCols);
        tmem_relinquish_pair();
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers are initialised before anything signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    RowTileWalker<static_cast<int>(ACC1), STEP> w(p.expert_offsets, p.num_experts, n_tiles);
    int e, nt, row0, rows;
    bool ok = true;

    if (warp < kMTSfWarp0) {
        reg_dealloc<kMTCtrlRegs>();
        if (warp == 0 && lane == 0) {
            // ------------------------------------------------------------ TMA producer (both CTAs)
            prefetch_tensormap(&tmap_a);
            prefetch_tensormap(&tmap_b);
            uint32_t it = 0;
            for (int tile = pair_id; ok && w.locate(tile, e, nt, row0, rows, rot_num, rot_den); tile += num_pairs) {
                const int half = ((rows + STEP - 1) & ~(STEP - 1)) / 2;  // rows of the tile in each CTA
                const int boxes = (half + kTRowBox - 1) / kTRowBox;
                const int my_row = row0 + static_cast<int>(cta) * half;
                const int w_lo = e * p.n_dim + block_lo(nt) * 128, w_hi = e * p.n_dim + block_hi(nt) * 128;
                const uint32_t bytes = static_cast<uint32_t>(kMTWBytes + boxes * kTRowBox * BK);
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const uint32_t s = it % NS, ph = (it / NS) & 1u;
                    if (!mbar_wait_bounded(&bar_empty[s], ph ^ 1u, abort_flag)) { ok = false; break; }
                    uint8_t* sa = smem + s * kMTStageBytes;
                    if (cta == 0) mbar_arrive_expect_tx(&bar_full[s], 2 * bytes);
                    const uint32_t full0 = map_to_cta(&bar_full[s], 0);
                    tma_load_2d_pair(sa, &tmap_b, full0, kb * BK, w_lo);
                    tma_load_2d_pair(sa + 128 * BK, &tmap_b, full0, kb * BK, w_hi);
                    for (int b = 0; b < boxes; ++b)
                        tma_load_2d_pair(sa + kMTWBytes + b * kTRowBox * BK, &tmap_a, full0, kb * BK, my_row + b * kTRowBox);
                }
            }
            if (!ok) gemm_record_status(p.status, CAM_ERR_TIMEOUT_PIPELINE, 0, static_cast<int>(it));
        } else if (warp == 1 && lane == 0 && cta == 0) {
            // ------------------------------------------------------------ MMA issuer (first CTA only)
            uint32_t it = 0, tcount = 0;
            const uint32_t tfull0 = map_to_cta(bar_tfull, 0), tfull1 = map_to_cta(bar_tfull, 1);
            for (int tile = pair_id; ok && w.locate(tile, e, nt, row0, rows, rot_num, rot_den); tile += num_pairs, ++tcount) {
                const uint32_t n = static_cast<uint32_t>((rows + STEP - 1) & ~(STEP - 1));
                const uint32_t idesc = I8 ? umma_idesc(2 * BM, n, /*c = s32*/ 2u, /*signed 8-bit*/ 1u) : umma_idesc_mxf8(2 * BM, n);
                // both epilogues must have drained the previous tile before its columns are overwritten
                if (!mbar_wait_bounded(bar_tempty, (tcount & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                tc_fence_after_sync();
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const uint32_t s = it % NS, ph = (it / NS) & 1u;
                    if (MX && !mbar_wait_bounded(&bar_sf[s], ph, abort_flag)) { ok = false; break; }
                    if (!mbar_wait_bounded(&bar_full[s], ph, abort_flag)) { ok = false; break; }
                    tc_fence_after_sync();
                    const uint32_t sa = smem_u32(smem + s * kMTStageBytes);
                    const uint64_t wlo = umma_desc_k_sw128(sa);
                    const uint64_t whi = umma_desc_k_sw128(sa + 128 * BK);
                    const uint64_t rdesc = umma_desc_k_sw128(sa + kMTWBytes);
                    const uint32_t sf = tmem_base + kMTSfCol0 + s * kMTSfStride;
#pragma unroll
                    for (int k = 0; k < BK / 32; ++k) {  // 32 bytes (= 2 x 16) further along K inside the swizzle atom
                        const uint32_t add = (kb | k) ? 1u : 0u;
                        if constexpr (MX) {
                            tc_mma_mxf8_pair(tmem_base, wlo + 2u * k, rdesc + 2u * k, idesc, add, sf, sf + 8u);
                            tc_mma_mxf8_pair(tmem_base + ACC1, whi + 2u * k, rdesc + 2u * k, idesc, add, sf + 4u, sf + 8u);
                        } else {
                            tc_mma_i8_pair(tmem_base, wlo + 2u * k, rdesc + 2u * k, idesc, add);
                            tc_mma_i8_pair(tmem_base + ACC1, whi + 2u * k, rdesc + 2u * k, idesc, add);
                        }
                    }
                    // the stage (smem and scale columns, in both CTAs) is reusable once these MMAs retire
                    tc_commit_pair(map_to_cta(&bar_empty[s], 0));
                    tc_commit_pair(map_to_cta(&bar_empty[s], 1));
                }
                if (!ok) break;
                tc_commit_pair(tfull0);  // accumulators complete once every MMA of the tile has retired
                tc_commit_pair(tfull1);
            }
            if (!ok) gemm_record_status(p.status, CAM_ERR_TIMEOUT_PIPELINE, 1, static_cast<int>(it));
        }
    } else if (warp < EPI0) {
        // ---------------------------------------------------------------- scale-factor writers (block scaling only)
        if constexpr (MX) {
        reg_dealloc<kMTSfRegs>();
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        uint32_t it = 0;
        // rows of scales can be read 16 bytes at a time when K is a multiple of 512 and the arrays are aligned
        const bool vec_scales = (kblocks & 3) == 0 &&
                                ((reinterpret_cast<uintptr_t>(p.a_scales) | reinterpret_cast<uintptr_t>(p.b_scales)) & 15u) == 0u;
        for (int tile = pair_id; ok && w.locate(tile, e, nt, row0, rows, rot_num, rot_den); tile += num_pairs) {
            const bool wide = rows > 128;  // rows 128.. have words of their own
            // scales of row 32 j + lane of the tile (every CTA writes the words of all rows, its own weight blocks' words)
            auto row_scales = [&](int j) {
                return p.a_scales + static_cast<size_t>(min(row0 + 32 * j + static_cast<int>(lane), p.a_rows - 1)) * kblocks;
            };
            const float* bs_lo = p.b_scales + (static_cast<size_t>(e) * nblk + block_lo(nt)) * kblocks;
            const float* bs_hi = p.b_scales + (static_cast<size_t>(e) * nblk + block_hi(nt)) * kblocks;
            // One K-block: byte `sel` of the packed words into the columns of stage s; then tell the MMA issuer.
            auto put = [&](const uint32_t (&pk)[10], uint32_t sel) -> bool {
                const uint32_t s = it % NS, ph = (it / NS) & 1u;
                const bool got = mbar_wait_bounded(&bar_empty[s], ph ^ 1u, abort_flag);
                if (!__all_sync(0xFFFFFFFFu, got)) return false;
                tc_fence_after_sync();
                const uint32_t col = tmem_base + lane_base + kMTSfCol0 + s * kMTSfStride;
                const uint32_t lo = __byte_perm(pk[8], 0, sel), hi = __byte_perm(pk[9], 0, sel);
                tmem_st_32x32b_x4(col, lo, lo, lo, lo);
                tmem_st_32x32b_x4(col + 4u, hi, hi, hi, hi);
                tmem_st_32x32b_x4(col + 8u, __byte_perm(pk[0], 0, sel), __byte_perm(pk[1], 0, sel), __byte_perm(pk[2], 0, sel),
                                  __byte_perm(pk[3], 0, sel));
                if (wide)
                    tmem_st_32x32b_x4(col + 12u, __byte_perm(pk[4], 0, sel), __byte_perm(pk[5], 0, sel),
                                      __byte_perm(pk[6], 0, sel), __byte_perm(pk[7], 0, sel));
                tc_wait_st();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) {  // the first CTA's barrier counts the warps of both CTAs
                    if (cta == 0) mbar_arrive(&bar_sf[s]);
                    else mbar_arrive_cluster(map_to_cta(&bar_sf[s], 0));
                }
                ++it;
                return true;
            };
            uint32_t pk[10], nx[10];
#pragma unroll
            for (int j = 0; j < 10; ++j) pk[j] = nx[j] = 0u;
            if (vec_scales) {
                // groups of four K-blocks, one 16-byte load per row and group, the next group's loads in two batches
                // between the puts of this one (the arrive of a put has release semantics and would wait for older loads)
                const int ngroups = kblocks >> 2;
                auto pack = [&](uint32_t (&d)[10], int g, int j0) {
                    float4 v[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] = __ldg(reinterpret_cast<const float4*>(row_scales(j0 + j)) + g);
#pragma unroll
                    for (int j = 0; j < 4; ++j) d[j0 + j] = ue8m0_pack4(v[j]);
                };
                auto pack_w = [&](uint32_t (&d)[10], int g) {
                    const float4 a = __ldg(reinterpret_cast<const float4*>(bs_lo) + g);
                    const float4 b = __ldg(reinterpret_cast<const float4*>(bs_hi) + g);
                    d[8] = ue8m0_pack4(a);
                    d[9] = ue8m0_pack4(b);
                };
                pack(pk, 0, 0);
                if (wide) pack(pk, 0, 4);
                pack_w(pk, 0);
                for (int g = 0; ok && g < ngroups; ++g) {
                    const bool more = g + 1 < ngroups;
                    ok = put(pk, 0x0000);
                    if (more) pack(nx, g + 1, 0);
                    if (ok) ok = put(pk, 0x1111);
                    if (more && wide) pack(nx, g + 1, 4);
                    if (ok) ok = put(pk, 0x2222);
                    if (more) pack_w(nx, g + 1);
                    if (ok) ok = put(pk, 0x3333);
#pragma unroll
                    for (int j = 0; j < 10; ++j) pk[j] = nx[j];
                }
                continue;
            }
            // any other K: scalar loads, one K-block ahead
            auto fetch = [&](uint32_t (&d)[10], int kb) {
                float v[10];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = __ldg(row_scales(j) + kb);
#pragma unroll
                for (int j = 4; j < 8; ++j) v[j] = wide ? __ldg(row_scales(j) + kb) : 0.f;
                v[8] = __ldg(bs_lo + kb);
                v[9] = __ldg(bs_hi + kb);
#pragma unroll
                for (int j = 0; j < 10; ++j) d[j] = (__float_as_uint(v[j]) >> 23) & 0xFFu;
            };
            fetch(pk, 0);
            for (int kb = 0; ok && kb < kblocks; ++kb) {
                if (kb + 1 < kblocks) fetch(nx, kb + 1);
                ok = put(pk, 0x0000);
#pragma unroll
                for (int j = 0; j < 10; ++j) pk[j] = nx[j];
            }
        }
        if (!ok && lane == 0) gemm_record_status(p.status, CAM_ERR_TIMEOUT_PIPELINE, 3, static_cast<int>(it));
        }
    } else {
        reg_alloc<rows_n_epi_regs(KIND)>();
        // ---------------------------------------------------------------- epilogue warps
        const int ew = warp - EPI0;
        const int q = warp & 3;   // TMEM lane quarter this warp may read
        const int cq = ew >> 2;   // which 32 rows (columns of the accumulators) of each 128
        const int f = q * 32 + static_cast<int>(lane);            // feature inside a 128-feature block
        const int te = ew * 32 + static_cast<int>(lane);          // 0..511
        uint32_t tcount = 0;
        for (int tile = pair_id; ok && w.locate(tile, e, nt, row0, rows, rot_num, rot_den); tile += num_pairs, ++tcount) {
            if (!mbar_wait_bounded(bar_tfull, tcount & 1u, abort_flag, 2000000000ull, 256u)) { ok = false; break; }
            tc_fence_after_sync();
#pragma unroll 1
            for (int r0 = 0; r0 < rows; r0 += 128) {  // rows [r0, r0 + 128) of the tile; the same trips in all threads
                const bool has_cols = r0 + cq * 32 < rows;  // columns past the tile's rows were not written
                uint32_t v0[32], v1[32];
                if (has_cols) {
                    const uint32_t t0 = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(r0 + cq * 32);
                    tmem_ld_32x32b_x32(t0, v0);
                    tmem_ld_32x32b_x32(t0 + ACC1, v1);
                    tc_wait_ld_regs(v0);
                    tc_wait_ld_regs(v1);
                }
                if (r0 + 128 >= rows) {  // the rest of the tile now lives in registers: hand the accumulators back
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        if (cta == 0) mbar_arrive(bar_tempty);
                        else mbar_arrive_cluster(map_to_cta(bar_tempty, 0));
                    }
                }
                if constexpr (I8) {
                    // dequantise: int32 accumulator x token scale x output-channel scale
                    if (has_cols) {
                        const float sb_lo = __ldg(p.b_scales + static_cast<size_t>(e) * p.n_dim + block_lo(nt) * 128 + f);
                        const float sb_hi = __ldg(p.b_scales + static_cast<size_t>(e) * p.n_dim + block_hi(nt) * 128 + f);
                        const float my_sa = __ldg(p.a_scales + min(row0 + r0 + cq * 32 + static_cast<int>(lane), p.a_rows - 1));
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const float sa = __shfl_sync(0xFFFFFFFFu, my_sa, j);
                            v0[j] = __float_as_uint(static_cast<float>(static_cast<int>(v0[j])) * sa * sb_lo);
                            v1[j] = __float_as_uint(static_cast<float>(static_cast<int>(v1[j])) * sa * sb_hi);
                        }
                    }
                }
                if constexpr (SWIGLU) {
                    // SiLU(gate) * up; 64 rows at a time go through shared memory as fp32 [row][feature], then 8 threads per
                    // row take the maximum of its 128 features, quantise and store 16 bytes each
                    const int fb = 2 * nt + static_cast<int>(cta);  // block of 128 activation features
                    const bool live = fb < nblk / 2;
                    if (has_cols) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {  // the product replaces the gate value
                            const float g = __uint_as_float(v0[j]);
                            v0[j] = __float_as_uint((g / (1.f + expf(-g))) * __uint_as_float(v1[j]));
                        }
                    }
                    float* stgf = reinterpret_cast<float*>(stg);
                    const int tl = te >> 3, pc = te & 7;
                    for (int half = 0; half < 2 && r0 + half * 64 < rows; ++half) {
                        if (has_cols && (cq >> 1) == half) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) stgf[((cq & 1) * 32 + j) * kMTPitchF + f] = __uint_as_float(v0[j]);
                        }
                        named_bar_sync(1, kMTEpiThreads);
                        const int tok = r0 + half * 64 + tl;
                        const float4* src = reinterpret_cast<const float4*>(stgf + tl * kMTPitchF + pc * 16);
                        const float4 x0 = src[0], x1 = src[1], x2 = src[2], x3 = src[3];
                        float amax = fmaxf(fmaxf(fmaxf(fabsf(x0.x), fabsf(x0.y)), fmaxf(fabsf(x0.z), fabsf(x0.w))),
                                           fmaxf(fmaxf(fabsf(x1.x), fabsf(x1.y)), fmaxf(fabsf(x1.z), fabsf(x1.w))));
                        amax = fmaxf(amax, fmaxf(fmaxf(fmaxf(fabsf(x2.x), fabsf(x2.y)), fmaxf(fabsf(x2.z), fabsf(x2.w))),
                                                 fmaxf(fmaxf(fabsf(x3.x), fabsf(x3.y)), fmaxf(fabsf(x3.z), fabsf(x3.w)))));
                        amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
                        amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
                        amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 4));
                        if constexpr (I8) {  // fp32 activations and the row's running maximum (m >= 0)
                            if (live && tok < rows && row0 + tok < p.a_rows) {
                                const size_t grow = static_cast<size_t>(row0 + tok);
                                float4* dst = reinterpret_cast<float4*>(p.act_f32 + (grow * (nblk / 2) + fb) * 128 + pc * 16);
                                dst[0] = x0; dst[1] = x1; dst[2] = x2; dst[3] = x3;
                                if (pc == 0) atomicMax(reinterpret_cast<int*>(p.row_amax + grow), __float_as_int(amax));
                            }
                            named_bar_sync(1, kMTEpiThreads);  // the staging area may be overwritten
                            continue;
                        }
                        float scale, inv;
                        ue8m0_scale(amax, scale, inv);
                        if (live && tok < rows && row0 + tok < p.a_rows) {
                            uint4 o;
                            o.x = pack_e4m3x4(x0.x * inv, x0.y * inv, x0.z * inv, x0.w * inv);
                            o.y = pack_e4m3x4(x1.x * inv, x1.y * inv, x1.z * inv, x1.w * inv);
                            o.z = pack_e4m3x4(x2.x * inv, x2.y * inv, x2.z * inv, x2.w * inv);
                            o.w = pack_e4m3x4(x3.x * inv, x3.y * inv, x3.z * inv, x3.w * inv);
                            const size_t at = static_cast<size_t>(row0 + tok) * (nblk / 2) + fb;  // in blocks of 128
                            *reinterpret_cast<uint4*>(p.act_q + at * 128 + pc * 16) = o;
                            if (pc == 0) p.act_s[at] = scale;
                        }
                        named_bar_sync(1, kMTEpiThreads);  // the staging area may be overwritten
                    }
                } else {
                    // bf16 rows, to the local output or straight to the origin rank's combine slot: one 256-byte bulk copy
                    // per row and weight block, issued by the thread (cq = 0) that owns the row
                    __nv_bfloat16* orow = nullptr;
                    const int tok = r0 + f;
                    if (cq == 0 && tok < rows && row0 + tok < p.a_rows) {
                        const size_t grow = static_cast<size_t>(row0 + tok);
                        if (p.mode == 0) {
                            orow = p.out + grow * p.n_dim;
                        } else {
                            const int src = p.row_src[grow * 3 + 0], st = p.row_src[grow * 3 + 1], kk = p.row_src[grow * 3 + 2];
                            if (src >= 0 && src < p.num_ranks && st >= 0 && st < p.max_tokens && kk >= 0 && kk < p.topk)
                                orow = reinterpret_cast<__nv_bfloat16*>(p.peer_base[src] + p.off_combine_buf) +
                                       (static_cast<size_t>(st) * p.topk + kk) * static_cast<size_t>(p.n_dim);
                        }
                    }
                    auto push = [&](const uint32_t (&v)[32], int blk) {
                        if (cq == 0) bulk_wait_group_read<0>();  // the previous copies have read the staging area
                        named_bar_sync(1, kMTEpiThreads);
                        if (has_cols) {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                *reinterpret_cast<__nv_bfloat16*>(stg + (cq * 32 + j) * kMTStgPitch + f * 2) =
                                    __float2bfloat16_rn(__uint_as_float(v[j]));
                        }
                        fence_proxy_async_smem();
                        named_bar_sync(1, kMTEpiThreads);
                        if (cq == 0) {
                            if (orow != nullptr) bulk_store_s2g(orow + blk * 128, stg + f * kMTStgPitch, 256);
                            bulk_commit_group();
                        }
                    };
                    const int blk = 4 * nt + 2 * static_cast<int>(cta);  // the same answer in every thread of the CTA
                    if (blk < nblk) push(v0, blk);
                    if (blk + 1 < nblk) push(v1, blk + 1);
                }
            }
        }
        if (!SWIGLU && cq == 0) bulk_wait_group<0>();  // every row this thread sent has been written
        if (!ok) gemm_record_status(p.status, CAM_ERR_TIMEOUT_PIPELINE, 2, static_cast<int>(tcount));
    }

    // ------------------------------------------------------------------ teardown
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();  // the other CTA may still read this CTA's shared memory or signal its barriers
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, kMTTmemCols);
    }
    if (p.mode == 2 && threadIdx.x == 0) {
        __threadfence_system();
        const unsigned int old = atomicAdd(p.done_ctr, 1u);
        if (old == gridDim.x - 1) {
            p.done_ctr[0] = 0u;
            __threadfence_system();
            const uint32_t epoch = *p.epoch_send + 1u;  // this launch is the send phase of a combine
            if (p.dbg_drop_flags == 0) {
                for (int d = 0; d < p.num_ranks; ++d)
                    st_release_sys_u32(reinterpret_cast<uint32_t*>(p.peer_base[d] + p.off_combine_flag) + p.rank,
                                       epoch);
            }
            *p.epoch_send = epoch;
        }
    }
}

}  // namespace cam

namespace {

template <int KIND, bool SWIGLU>
int launch_rows_n(const cam::GroupedGemmParams* p, const CUtensorMap* tmap_a, const CUtensorMap* tmap_b, int grid,
                  cudaStream_t stream) {
    static cam::SmemLimitCache limit;
    cudaError_t err = limit.ensure(cam::grouped_gemm_rows_n_kernel<KIND, SWIGLU>, cam::kMTSmem);
    if (err != cudaSuccess) return static_cast<int>(err);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(static_cast<unsigned>(grid & ~1));  // whole pairs only
    cfg.blockDim = dim3(cam::rows_n_threads(KIND));
    cfg.dynamicSmemBytes = cam::kMTSmem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // Not every SM can always be paired inside its GPC: run exactly as many pairs as fit at once (cached per device).
    static int max_pairs[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) {
        if (max_pairs[dev] == 0) {
            int n = 0;
            const cudaError_t q = cudaOccupancyMaxActiveClusters(&n, cam::grouped_gemm_rows_n_kernel<KIND, SWIGLU>, &cfg);
            max_pairs[dev] = (q == cudaSuccess && n > 0) ? n : -1;
        }
        if (max_pairs[dev] > 0 && 2 * max_pairs[dev] < static_cast<int>(cfg.gridDim.x))
            cfg.gridDim = dim3(static_cast<unsigned>(2 * max_pairs[dev]));
    }
    return static_cast<int>(cudaLaunchKernelEx(&cfg, cam::grouped_gemm_rows_n_kernel<KIND, SWIGLU>, *tmap_a, *tmap_b, *p));
}

}  // namespace
