// CSR SpMV building blocks shared by the assembly and Krylov translation units (sm_103a).
//
// A row is handled by TPR consecutive lanes; each lane issues U column-index and U value loads, then
// U x gathers, before any product, so every thread keeps that many independent loads in flight (the
// rows of the FE matrices here hold 7 to 60 entries). Lanes reduce with shuffles; all TPR lanes end with
// the row sum. Bound by the FP64 pipe, on which a warp-wide instruction takes 64 clocks: a row costs its
// products and log2(TPR) additions for every lane, so few lanes per row pay until the loads of a lane no
// longer coalesce. Measured (us, cold L2, with one accumulator and products between the gathers before):
// 531,441 rows of 28 entries 64.2 with 4 x 8, 59.1 with 2 x 8, 62.1 with 4 x 8 staged, 70.3 with 1 x 8;
// 103,041 of 11.5 entries 15.0 (4 x 4) and 13.1 (2 x 8); 226,981 of 47 entries 45.7 (2 x 8), 43.7 (4 x 8).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "ocmp_internal.h"

namespace ocmp {

struct RowCfg {
    int tpr, u;
};
// Threads per row and loads in flight per lane: the autotuned choice when there is one, else a
// rule on the mean row length.
inline RowCfg row_cfg(const ocmp_space_s* s) {
    if (s->tuned_tpr > 0) return {s->tuned_tpr, s->tuned_u};
    const double avg = (double)s->nnz / (double)s->ndof;
    if (avg <= 6) return {2, 4};
    if (avg <= 16) return {4, 4};
    if (avg <= 32) return {4, 8};
    if (avg <= 64) return {8, 8};
    return {16, 8};
}

// the same for an FP64 product of its own launch: half the lanes for rows of more than 16 entries, once they
// fill the chip's threads. Below, the loads in flight count for more: P2 tetrahedra (us, cold L2, 2 x 8
// against 4 x 8) 20.5 and 18.0 at 9,261 rows, 26.3 and 24.1 at 68,921, 33 and 32.4 at 148,877, 45 and 46
// at 274,625; P3 tetrahedra (4 x 8 against 8 x 8) 27.2 and 23.7 at 29,791, 36.8 and 39.6 at 117,649.
constexpr int64_t kChipThreads = 152 * 2048;
inline RowCfg row_cfg64(const ocmp_space_s* s) {
    if (s->tuned_tpr > 0) return {s->tuned_tpr, s->tuned_u};
    const double avg = (double)s->nnz / (double)s->ndof;
    if (avg <= 6) return {2, 4};
    if (avg <= 16) return {2, 8};
    const RowCfg few = {avg <= 32 ? 2 : avg <= 64 ? 4 : 8, 8};
    return s->ndof * few.tpr < kChipThreads ? row_cfg(s) : few;
}

template <class TM, class TV, int TPR, int U>
__device__ __forceinline__ TV row_dot(int32_t a, int32_t b, const int32_t* __restrict__ col,
                                      const TM* __restrict__ val, const TV* __restrict__ x, int lane) {
    TV acc0 = 0, acc1 = 0;
    for (int32_t base = a + lane; base < b; base += U * TPR) {
        int32_t c[U];
        TM v[U];
        TV g[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int32_t k = base + u * TPR;
            c[u] = k < b ? __ldg(col + k) : -1;
            v[u] = k < b ? __ldg(val + k) : (TM)0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) g[u] = c[u] >= 0 ? __ldg(x + c[u]) : (TV)0;
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c[u] >= 0) (u & 1 ? acc1 : acc0) += (TV)v[u] * g[u];
    }
    TV acc = acc0 + acc1;
#pragma unroll
    for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, TPR);
    return acc;
}


}  // namespace ocmp
