// Column statistics of a row-major FP32 matrix on the device, for the surrogates' input
// standardisation: the mean and the reciprocal standard deviation per column, in FP64 and in the row
// order of the plain loop (sum, mean, sum of squared deviations; every operation rounded once), so the
// result does not depend on how the work is split.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace ta3_stats {

constexpr int COLS = 32;      // columns (threads) per block: 154 blocks for 4,929 columns
constexpr int DEEP = 16;      // rows in flight per thread

// One thread per column; a warp reads 128 contiguous bytes of a row. The adds are one chain per column,
// so the loads run DEEP rows ahead. 2 passes over x (the second mostly from L2). The host loop it
// replaces walked the columns with a stride of a row: 43 ms of a 71 ms retrain on 4,000 x 4,929.
static __global__ void __launch_bounds__(COLS) column_stats_kernel(float const* __restrict__ x, int rows, int cols, int64_t ld,
                                                            float* __restrict__ mean, float* __restrict__ inv_std) {
    int const c = int(blockIdx.x) * COLS + int(threadIdx.x);
    if (c >= cols) return;
    float const* const p = x + c;
    double sum = 0.0, mu = 0.0, sq = 0.0;
    for (int pass = 0; pass < 2; ++pass) {
        float v[DEEP];
#pragma unroll
        for (int i = 0; i < DEEP; ++i) v[i] = i < rows ? __ldg(p + int64_t(i) * ld) : 0.f;
        for (int r0 = 0; r0 < rows; r0 += DEEP) {
            float next[DEEP];
#pragma unroll
            for (int i = 0; i < DEEP; ++i) next[i] = r0 + DEEP + i < rows ? __ldg(p + int64_t(r0 + DEEP + i) * ld) : 0.f;
#pragma unroll
            for (int i = 0; i < DEEP; ++i)
                if (r0 + i < rows) {
                    if (pass == 0) {
                        sum = __dadd_rn(sum, double(v[i]));
                    } else {
                        double const d = __dadd_rn(double(v[i]), -mu);
                        sq = __dadd_rn(sq, __dmul_rn(d, d));
                    }
                }
#pragma unroll
            for (int i = 0; i < DEEP; ++i) v[i] = next[i];
        }
        if (pass == 0) mu = __ddiv_rn(sum, double(rows));
    }
    double const sd = __dsqrt_rn(__ddiv_rn(sq, double(rows)));
    mean[c] = float(mu);
    inv_std[c] = sd > 1e-12 ? float(__ddiv_rn(1.0, sd)) : 1.f;
}

static inline cudaError_t column_stats(float const* x, int rows, int cols, int64_t ld, float* mean, float* inv_std,
                                cudaStream_t st) {
    column_stats_kernel<<<unsigned((cols + COLS - 1) / COLS), COLS, 0, st>>>(x, rows, cols, ld, mean, inv_std);
    return cudaGetLastError();
}

} // namespace ta3_stats
