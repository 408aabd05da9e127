// Slots of (token, k) pairs inside their experts when all ids are in shared memory.
#pragma once
#include "ptx.cuh"

namespace cam {

// Slot of pair i inside its expert (earlier pairs in scan order with the same id), by one whole warp.
__device__ __forceinline__ int warp_slot_of(const int* s_ids, int i, uint32_t lane) {
    const int id = s_ids[i];
    int n = 0;
#pragma unroll 4
    for (int j = static_cast<int>(lane); j < i; j += 32) n += (s_ids[j] == id) ? 1 : 0;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) n += __shfl_xor_sync(0xFFFFFFFFu, n, o);
    return n;
}

// Inclusive prefix sum of the row counts in s_run[0..E) into s_cum, by one warp.
__device__ __forceinline__ void warp_scan_counts(const int* s_run, int* s_cum, int E, uint32_t lane) {
    const int per = (E + 31) / 32;
    const int lo = static_cast<int>(lane) * per, hi = min(E, lo + per);
    int sum = 0;
    for (int o = lo; o < hi; ++o) sum += s_run[o];
    int incl = sum;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const int n = __shfl_up_sync(0xFFFFFFFFu, incl, s);
        if (static_cast<int>(lane) >= s) incl += n;
    }
    int run = incl - sum;
    for (int o = lo; o < hi; ++o) { run += s_run[o]; s_cum[o] = run; }
}

}  // namespace cam
