// One event's FP64 angular values of the stored polarisations, from the
// [row][ld] table: M_NPOL complex rows per plane, or, paired, M_NPOL real rows
// (x and y of each pair, one real for the polarisation paired with itself).
#pragma once

#include "device_helpers.cuh"
#include "model.cuh"

template <bool PAIRED>
__device__ __forceinline__ void ct_load_angular(const void* __restrict__ table, long long ld, long long e, double2* sl)
{
    constexpr int NPS = PAIRED ? (M_NPOL + 1) / 2 : M_NPOL;
    if constexpr (PAIRED) {
        const double* __restrict__ t = (const double*)table + e;
#pragma unroll
        for (int c = 0; c < M_NPLANE; ++c)
#pragma unroll
            for (int p = 0; p < NPS; ++p) {
                sl[c * NPS + p].x = __ldg(t + (long long)(c * M_NPOL + 2 * p) * ld);
                sl[c * NPS + p].y = 2 * p + 1 < M_NPOL ? __ldg(t + (long long)(c * M_NPOL + 2 * p + 1) * ld) : 0.0;
            }
    } else {
        const double2* __restrict__ t = (const double2*)table + e;
#pragma unroll
        for (int c = 0; c < M_NPLANE * NPS; ++c) sl[c] = __ldg(t + (long long)c * ld);
    }
}
