// Column statistics of a row-major FP32 matrix, for the surrogates' input standardisation: the mean and
// the reciprocal standard deviation per column, in FP64 and in the row order of the plain loop (sum, mean,
// sum of squared deviations; every operation rounded once), so the result does not depend on how the
// work is split, nor on which of the two versions below did it.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstddef>
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

// The same on the host, N neighbouring columns at a time (their chains run side by side)
template <int N>
inline void host_group(float const* x, size_t rows, size_t ld, float* mean, float* inv_std) {
    double sum[N] = {}, sq[N] = {}, mu[N];
    for (size_t r = 0; r < rows; ++r)
        for (int j = 0; j < N; ++j) sum[j] += x[r * ld + j];
    for (int j = 0; j < N; ++j) mu[j] = sum[j] / double(rows);
    for (size_t r = 0; r < rows; ++r)
        for (int j = 0; j < N; ++j) {
            double const d = x[r * ld + j] - mu[j];
            sq[j] += d * d;
        }
    for (int j = 0; j < N; ++j) {
        double const sd = std::sqrt(sq[j] / double(rows));
        mean[j] = float(mu[j]);
        inv_std[j] = sd > 1e-12 ? float(1.0 / sd) : 1.f;
    }
}
// Which of the two: the kernel takes its launch and 57 ns a row however few columns there are, the host 0.6
// to 1.2 ns an element. So the host takes narrow matrices and small ones. A whole set_data call, host against
// device: 1 column, 100,000 rows 0.33 against 5.7 ms; 32 columns, 8,000 rows 0.21 against 0.58 ms (100,000
// rows 3.8 against 6.9); 48 columns, 100,000 rows 6.5 against 7.1 ms; 97 columns, 100 rows 48 against 52 us; but
// 64 columns, 100,000 rows 10.0 against 7.4 ms.
inline bool stats_on_host(size_t rows, size_t cols) { return cols <= 48 || rows * cols <= 16384; }
inline void host_column_stats(float const* x, size_t rows, size_t cols, float* mean, float* inv_std) {
    size_t c = 0;
    for (; c + 8 <= cols; c += 8) host_group<8>(x + c, rows, cols, mean + c, inv_std + c);
    if (cols & 4) host_group<4>(x + c, rows, cols, mean + c, inv_std + c), c += 4;
    if (cols & 2) host_group<2>(x + c, rows, cols, mean + c, inv_std + c), c += 2;
    if (cols & 1) host_group<1>(x + c, rows, cols, mean + c, inv_std + c);
}

} // namespace ta3_stats
