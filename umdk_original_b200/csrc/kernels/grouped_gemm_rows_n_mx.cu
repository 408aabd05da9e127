// The block-scaled form of grouped_gemm_rows_n.cuh.
#include <cstdint>

namespace cam {
constexpr uint32_t kMTLaunchRegs = 80;  // what ptxas reports for 768 threads per CTA
}
#include "grouped_gemm_rows_n.cuh"

extern "C" int cam_grouped_gemm_rows_n_box(void) { return cam::kTRowBox; }

// tmap_a: boxes of cam_grouped_gemm_rows_n_box() rows; tmap_b: boxes of 128 rows.
extern "C" int cam_launch_grouped_gemm_mxfp8_rows_n(const cam::GroupedGemmParams* p, const CUtensorMap* tmap_a,
                                                    const CUtensorMap* tmap_b, int grid, cudaStream_t stream) {
    return p->mode == 1 ? launch_rows_n<cam::kRowsMx, true>(p, tmap_a, tmap_b, grid, stream)
                        : launch_rows_n<cam::kRowsMx, false>(p, tmap_a, tmap_b, grid, stream);
}
