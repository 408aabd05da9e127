// Exact W8A8 arithmetic of the reference's fused operator: int8 activations with one dynamic scale per token, int8 weights
// with one scale per output channel, int32 accumulation (fused_deep_moe/gemm/kernel/grouped_matmul_slice_m_per_token_dequant_
// swiglu_quant_multistage_workspace.h:558-632 on the cube cores, dequantisation in
// epilogue/block/block_epilogue_per_token_dequant_swiglu.h:236-272 and block_epilogue_per_token_dequant.hpp:664-684 on the
// vector cores).  The two GEMMs are grouped_gemm_i8.cu or the int8 form of grouped_gemm_rows_n.cuh (a_scales [rows], one per token;
// b_scales [E, N], one per output channel); their mode 1 leaves fp32 activations and the maximum of |.| of every row, from which the pass below
// derives the per-token scale of the second GEMM's activations (the reference's BlockQuant pass, ...workspace.h:161-277).
#include "gemm_common.cuh"

namespace cam {

// Per-token int8 quantisation of the SwiGLU output (one warp per row): scale = max|row| / 127 from the
// maxima GEMM1 accumulated, q = rint(x / scale).  Clears the row maximum for the next call.
__global__ void rowquant_int8_kernel(const float* __restrict__ act, float* row_amax, const int* __restrict__ expert_offsets,
                                     int num_experts, int inter, int8_t* __restrict__ out_q, float* __restrict__ out_s) {
    const int rows = expert_offsets[num_experts];
    const int warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t lane = lane_id();
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += warps) {
        const float amax = fmaxf(row_amax[r], 1e-12f);
        __syncwarp();
        if (lane == 0) row_amax[r] = 0.f;
        const float inv = 127.f / amax;
        const float* src = act + static_cast<size_t>(r) * inter;
        int8_t* dst = out_q + static_cast<size_t>(r) * inter;
        for (int c = static_cast<int>(lane) * 4; c < inter; c += 128) {
            const float4 v = *reinterpret_cast<const float4*>(src + c);
            const int a0 = max(-127, min(127, __float2int_rn(v.x * inv))), a1 = max(-127, min(127, __float2int_rn(v.y * inv)));
            const int a2 = max(-127, min(127, __float2int_rn(v.z * inv))), a3 = max(-127, min(127, __float2int_rn(v.w * inv)));
            *reinterpret_cast<uint32_t*>(dst + c) = (static_cast<uint32_t>(a0) & 0xFFu) | ((static_cast<uint32_t>(a1) & 0xFFu) << 8) |
                                                    ((static_cast<uint32_t>(a2) & 0xFFu) << 16) | ((static_cast<uint32_t>(a3) & 0xFFu) << 24);
        }
        if (lane == 0) out_s[r] = amax / 127.f;
    }
}

}  // namespace cam

extern "C" int cam_launch_rowquant_int8(const float* act, float* row_amax, const int* expert_offsets, int num_experts,
                                        int inter, void* out_q, float* out_s, cudaStream_t stream) {
    cam::rowquant_int8_kernel<<<4 * cam::sm_count_of_current_device(), 256, 0, stream>>>(
        act, row_amax, expert_offsets, num_experts, inter, static_cast<int8_t*>(out_q), out_s);
    return static_cast<int>(cudaGetLastError());
}
