// Surrogate fitness model for any parameter-vector size: an MLP in -> H -> H -> 2
// (predicted mean score, log-variance), the v11 surrogate's scheme scaled to the
// widened evaluator (in = 4,929 parameters, H = 256). No counterpart in the
// reference; the C ABI is the ta3w_* part of include/ta3b_surrogate.h.
//
// Layer by layer instead of one fused kernel (the first layer's weights alone are
// H x in = 1.3 M values): every matrix product is a tcgen05.mma (kind::f16, BF16
// operands staged in shared memory, FP32 accumulators in tensor memory) GEMM on
// 128 x 64 output tiles with K in stages of 64 and optional split-K. A training
// step is six launches: F1 = X W1^T (split-K), act1 (sum, bias, ReLU), F2 = H1 W2^T,
// head (output layer, loss, dH2), dW2 and dH1 side by side (the ReLU mask of layer 1
// in the epilogue), dW1 with AdamW in its epilogue beside the bias and output-layer
// gradients and W2's update. Each launch starts while the previous one drains
// (programmatic dependent launch). Every reduction runs in a fixed order, so two
// identical calls give identical bits. A step of 256 rows at 4,929 -> 256 takes
// 45 us (eleven launches and square 128 x 128 tiles loaded by one warpgroup: 440 us),
// of which six launches' latencies are 24 us and AdamW over 1.3 M parameters 9 us.
//
// Operand tiles (128 of M or 64 of N by 64 of K, BF16) are stored in rows of 128 bytes (64 elements) with
// the 128-byte swizzle (the row's eight 16-byte chunks XORed with the row number mod 8), eight rows an
// atom of 1,024 bytes. An operand whose global rows run along K (K-major) has a row per m or n: SBO 1,024
// (next 8 rows), 32 bytes on per 16 of K. One whose global rows run along M/N (MN-major: the
// weight-gradient products, where K is the batch) has a row per k, in blocks of 64 of M/N: SBO 1,024 (next
// 8 of K), LBO 8,192 (next 64 of M/N), 2,048 bytes on per 16 of K. Either way eight threads copy a
// contiguous 128-byte line into eight different bank groups (with unswizzled core matrices the same
// copies took 30 cycles a warp instruction: 4,200 cycles for three stages against 900 now).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <numeric>
#include <random>
#include <string>
#include <vector>

#include "../../include/ta3b_surrogate.h"
#include "column_stats.cuh"

namespace ta3w {

constexpr int TILE = 128;                       // M per output tile, and the padding of rows and inputs
constexpr int TN = 64;                          // N per output tile: twice the CTAs of a square tile, and two fit an SM
constexpr int KS = 64;                          // K per shared-memory stage
constexpr int STAGES = 4;                       // stages in flight: the whole K of a 256-row minibatch
constexpr int THREADS = 512;                    // 32 warps an SM for the AdamW epilogue (two CTAs)
constexpr uint32_t A_BYTES = TILE * KS * 2, B_BYTES = TN * KS * 2, STAGE_BYTES = A_BYTES + B_BYTES;   // 16 + 8 KB
constexpr uint32_t S_BAR = STAGES * STAGE_BYTES;   // the stages, then an mbarrier each
constexpr uint32_t S_TMEM = S_BAR + 8 * STAGES;
constexpr uint32_t S_ROWS = S_TMEM + 16;        // operand row maps: 128 of A's M, or up to 1,024 of B's K
constexpr int MAP_ROWS = 1024;
constexpr uint32_t SMEM_BYTES = S_ROWS + 4 * MAP_ROWS + 1024;   // + alignment slack
constexpr int LDT = TN + 4;                     // row stride of an output tile in shared memory (16-byte rows, 4 banks apart)
static_assert(TILE * LDT * 4 <= int(S_BAR), "the output tile reuses the stages");
constexpr long long WAIT_LIMIT_CYCLES = 4000000000LL;  // ~2 s at 1.9 GHz

// tcgen05 shared-memory matrix descriptor: start, LBO, SBO (all >> 4), version 1, 128-byte swizzle
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return uint64_t((saddr >> 4) & 0x3FFF) | (uint64_t((lbo >> 4) & 0x3FFF) << 16) |
           (uint64_t((sbo >> 4) & 0x3FFF) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61);
}
// instruction descriptor: D F32, A/B BF16, majors (0 = K, 1 = MN), N = 64, M = 128
__host__ __device__ constexpr uint32_t instr_desc(int a_mn, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(a_mn) << 15) | (uint32_t(b_mn) << 16) |
           (uint32_t(TN >> 3) << 17) | (uint32_t(TILE >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void mbar_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// bounded wait for the completion of the barrier phase with the given parity; false on timeout
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    long long const t0 = clock64();
    while (true) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > WAIT_LIMIT_CYCLES) return false;
    }
}

// The previous launch's results are visible after pdl_wait; pdl_go lets the next launch start (it
// waits for this one to complete in its own pdl_wait, so nothing of it overlaps but its set-up).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Which source row a pass's row r is: r < valid ? (idx ? idx[r] : r) : none (-1, a zero row).
struct RowMap {
    int32_t const* idx;
    int valid;
    __device__ __forceinline__ int at(int r) const { return r < valid ? (idx ? __ldg(idx + r) : r) : -1; }
};

// AdamW's constants and the arrays it updates at flat parameter index i
struct Adam {
    float* param;
    float* m;
    float* v;
    float lr, b1, b2, eps, c1, c2, wd;
    __device__ __forceinline__ float step(float g, float& mi, float& vi, float w) const {
        mi = b1 * mi + (1.f - b1) * g;
        vi = b2 * vi + (1.f - b2) * g * g;
        return w - lr * (mi / c1) / (sqrtf(vi / c2) + eps) - lr * wd * w;
    }
    __device__ __forceinline__ float update(int64_t i, float g) const {       // the new parameter
        float mi = m[i], vi = v[i];
        float const w = step(g, mi, vi, param[i]);
        m[i] = mi;
        v[i] = vi;
        param[i] = w;
        return w;
    }
};

// C[split][M][N] (FP32) = sum over this split's K of A(m, k) B(n, k), where
//   A(m, k) = A_MN ? a[k * lda + m] : a[m' * lda + k]   (BF16; ' = through the row map when
//   B(n, k) = B_MN ? b[k' * ldb + n] : b[n * ldb + k]    MAPPED)
// M a multiple of 128, N and K of 64, k_split of 64.
enum Epilogue { EPI_STORE = 0, EPI_MASK = 1, EPI_ADAM = 2 };
struct GemmArgs {
    __nv_bfloat16 const* a;
    int64_t lda;
    __nv_bfloat16 const* b;
    int64_t ldb;
    RowMap map;
    float* c;
    int64_t ldc;
    int64_t c_split;       // floats between consecutive splits' outputs
    int m, n, k, k_split;
    uint32_t* status;      // bit 0: a tensor-core wait timed out
    __nv_bfloat16 const* mask;   // EPI_MASK: out16 = BF16(mask > 0 ? C : 0), both [M][ldc]
    __nv_bfloat16* out16;        // EPI_MASK; EPI_ADAM: the BF16 copy of the updated weights [M][ldc]
    int live_n;                  // EPI_ADAM: columns that are weights; the rest is padding, which stays zero
    int mapped;                  // the row map applies (to A's rows, or to B's with B_MN)
};

__device__ __forceinline__ void cp_async16(uint32_t dst, void const* src, bool valid) {   // zeros when not valid
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// one operand stage (EXT of M/N x 64 of K) from global memory into its swizzled rows, 16 bytes a copy
template <int MN, int EXT>
__device__ __forceinline__ void stage_operand(uint32_t dst, __nv_bfloat16 const* src, int64_t ld, int32_t const* rows,
                                              RowMap const& map, bool mapped, int r0, int k0, int kbase, int tid) {
#pragma unroll
    for (int q = 0; q < EXT * 8 / THREADS; ++q) {
        int const c = tid + THREADS * q, j = c & 7;    // EXT * 8 chunks, eight to a row
        int outer, inner, row;
        uint32_t off;
        if (MN) {                                      // global rows = K, EXT / 64 tile rows each
            int const blk = EXT == 64 ? 0 : (c >> 3) & 1;
            row = EXT == 64 ? c >> 3 : c >> 4;
            outer = k0 + row;
            if (mapped) outer = outer - kbase < MAP_ROWS ? rows[outer - kbase] : map.at(outer);
            inner = r0 + 64 * blk + 8 * j;
            off = uint32_t(blk * 8192);
        } else {                                       // global rows = M/N, one tile row each
            row = c >> 3;
            outer = mapped ? rows[row] : r0 + row;
            inner = k0 + 8 * j;
            off = 0;
        }
        cp_async16(dst + off + uint32_t(row * 128 + ((j ^ (row & 7)) * 16)), src + (outer >= 0 ? outer : 0) * ld + inner,
                   outer >= 0);
    }
}

// one 128 x 64 output tile, for all threads of a CTA. What bounds it at these sizes (K of 256 to 320 per
// tile) is latency: every stage of a minibatch's K is in flight at once, one thread issues the MMAs as the
// stages land. A 128 x 64 x 256 tile takes 5,000 cycles from its first copy to its last store (15,000 with
// unswizzled operands and each thread storing its own row).
template <int A_MN, int B_MN, int EPI>
__device__ __forceinline__ void gemm_tile(GemmArgs const& g, Adam const& ad, int tile_m, int tile_n, int split,
                                          uint8_t* sm, int tid) {
    uint32_t const sbase = uint32_t(__cvta_generic_to_shared(sm));
    int const warp = tid >> 5, lane = tid & 31;
    int const m0 = tile_m * TILE, n0 = tile_n * TN;
    int const kb = split * g.k_split;
    int const ke = min(g.k, kb + g.k_split);
    int const nk = (ke - kb) / KS;
    uint32_t const bar0 = sbase + S_BAR;                // stage b's barrier: bar0 + 8 b
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + S_TMEM);
    volatile uint32_t* abort_s = reinterpret_cast<volatile uint32_t*>(sm + S_TMEM + 4);
    int32_t* const rows = reinterpret_cast<int32_t*>(sm + S_ROWS);
    if (tid == 0) {
        for (int b = 0; b < STAGES; ++b) mbar_init(bar0 + 8 * b);
        *abort_s = 0u;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + S_TMEM),
                     "r"(uint32_t(TN)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    pdl_go();
    if (g.mapped) {                                     // A's 128 rows, or (B_MN) the first MAP_ROWS of this split's K
        int const first = B_MN ? kb : m0, count = B_MN ? min(ke - kb, MAP_ROWS) : TILE;
        for (int r = tid; r < count; r += THREADS) rows[r] = g.map.at(first + r);
    }
    fence_before();
    __syncthreads();
    fence_after();
    uint32_t const tmem = *tmem_slot;
    uint32_t const idesc = instr_desc(A_MN, B_MN);
    auto load = [&](int it) {
        uint32_t const as = sbase + uint32_t(it % STAGES) * STAGE_BYTES;
        int const k0 = kb + it * KS;
        stage_operand<A_MN, TILE>(as, g.a, g.lda, rows, g.map, g.mapped && !B_MN, m0, k0, kb, tid);
        stage_operand<B_MN, TN>(as + A_BYTES, g.b, g.ldb, rows, g.map, g.mapped && B_MN, n0, k0, kb, tid);
    };
    for (int it = 0; it < STAGES - 1; ++it) {
        if (it < nk) load(it);
        cp_async_commit();
    }
    for (int it = 0; it < nk; ++it) {
        // the buffer loaded below is free once the MMAs of the iteration before completed
        if (tid == 0 && it >= 1 && it + STAGES - 1 < nk &&
            !mbar_wait(bar0 + 8 * ((it - 1) % STAGES), uint32_t((it - 1) / STAGES) & 1u)) {
            *abort_s = 1u;
            atomicOr(g.status, 1u);
        }
        cp_async_wait<STAGES - 2>();                    // this thread's share of stage `it` has landed
        fence_async_smem();
        __syncthreads();
        if (*abort_s) break;
        if (tid == 0) {
            fence_after();
            uint32_t const a_s = sbase + uint32_t(it % STAGES) * STAGE_BYTES, b_s = a_s + A_BYTES;
#pragma unroll
            for (int kk = 0; kk < KS / 16; ++kk) {
                uint64_t const da = smem_desc(a_s + kk * (A_MN ? 2048 : 32), A_MN ? 8192 : 16, 1024);
                uint64_t const db = smem_desc(b_s + kk * (B_MN ? 2048 : 32), B_MN ? 8192 : 16, 1024);
                mma_bf16(tmem, da, db, idesc, (it > 0 || kk > 0) ? 1u : 0u);
            }
            mma_commit(bar0 + 8 * (it % STAGES));
        }
        if (it + STAGES - 1 < nk) load(it + STAGES - 1);
        cp_async_commit();
    }
    cp_async_wait<0>();
    // the last commit completes after every MMA of this CTA
    if (tid == 0 && !*abort_s && nk > 0 && !mbar_wait(bar0 + 8 * ((nk - 1) % STAGES), uint32_t((nk - 1) / STAGES) & 1u)) {
        *abort_s = 1u;
        atomicOr(g.status, 1u);
    }
    __syncthreads();
    fence_after();
    if (!*abort_s) {
        // TMEM lane = output row; each group of four warps takes 16 of the tile's columns
        static_assert(TN == 16 * (THREADS / 128), "four warps per 16 columns");
        int const r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 16;
        uint32_t const lane_base = tmem + (uint32_t((warp & 3) * 32) << 16);
        float v[16];
        if (nk > 0) {
            tmem_ld16(lane_base + c0, v);
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = 0.f;
        }
        // through shared memory (the stages are free), so that 16 threads move a row's 256 contiguous bytes
        float* const t = reinterpret_cast<float*>(sm);
#pragma unroll
        for (int j = 0; j < 16; j += 4)
            *reinterpret_cast<float4*>(t + r * LDT + c0 + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        __syncthreads();
        int const cc = (tid & 15) * 4;
        float* const crow = EPI == EPI_STORE ? g.c + int64_t(split) * g.c_split : nullptr;
#pragma unroll 2
        for (int rr = tid >> 4; rr < TILE; rr += THREADS / 16) {
            int64_t const at = int64_t(m0 + rr) * g.ldc + n0 + cc;
            float4 x = *reinterpret_cast<float4 const*>(t + rr * LDT + cc);
            if (EPI == EPI_STORE) {
                *reinterpret_cast<float4*>(crow + at) = x;
            } else {
                if (EPI == EPI_MASK) {
                    uint2 const h = *reinterpret_cast<uint2 const*>(g.mask + at);
                    x.x = __uint_as_float(h.x << 16) > 0.f ? x.x : 0.f;
                    x.y = __uint_as_float(h.x & 0xFFFF0000u) > 0.f ? x.y : 0.f;
                    x.z = __uint_as_float(h.y << 16) > 0.f ? x.z : 0.f;
                    x.w = __uint_as_float(h.y & 0xFFFF0000u) > 0.f ? x.w : 0.f;
                } else {                                          // AdamW with the gradient x
                    float4 mi = *reinterpret_cast<float4 const*>(ad.m + at), vi = *reinterpret_cast<float4 const*>(ad.v + at);
                    float4 const w = *reinterpret_cast<float4 const*>(ad.param + at);
                    x.x = ad.step(x.x, mi.x, vi.x, w.x);
                    x.y = ad.step(x.y, mi.y, vi.y, w.y);
                    x.z = ad.step(x.z, mi.z, vi.z, w.z);
                    x.w = ad.step(x.w, mi.w, vi.w, w.w);
                    // padding: its gradient is a sum of dH1 * 0, which is NaN where dH1 is not finite
                    if (n0 + TN > g.live_n) {                     // (the row's last tiles: uniform over the CTA)
                        int const live = g.live_n - (n0 + cc);
                        if (live < 1) x.x = mi.x = vi.x = 0.f;
                        if (live < 2) x.y = mi.y = vi.y = 0.f;
                        if (live < 3) x.z = mi.z = vi.z = 0.f;
                        if (live < 4) x.w = mi.w = vi.w = 0.f;
                    }
                    *reinterpret_cast<float4*>(ad.m + at) = mi;
                    *reinterpret_cast<float4*>(ad.v + at) = vi;
                    *reinterpret_cast<float4*>(ad.param + at) = x;
                }
                __nv_bfloat162 const lo = __floats2bfloat162_rn(x.x, x.y), hi = __floats2bfloat162_rn(x.z, x.w);
                *reinterpret_cast<uint2*>(g.out16 + at) = make_uint2(*reinterpret_cast<uint32_t const*>(&lo),
                                                                     *reinterpret_cast<uint32_t const*>(&hi));
            }
        }
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(uint32_t(TN)) : "memory");
}

__device__ __forceinline__ uint8_t* aligned_smem() {
    extern __shared__ uint8_t smem_raw[];
    return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
}

// one product: grid (M/128, N/64, splits)
template <int A_MN, int B_MN>
__global__ void __launch_bounds__(THREADS, 2) gemm_kernel(GemmArgs g) {
    gemm_tile<A_MN, B_MN, EPI_STORE>(g, Adam{}, blockIdx.x, blockIdx.y, blockIdx.z, aligned_smem(), threadIdx.x);
}

// two independent products of the backward pass in one launch (neither fills the chip): dW2 = dH2^T H1 on
// the first tiles, dH1 = BF16((H1 > 0) * dH2 W2) on the others
__global__ void __launch_bounds__(THREADS, 2) backward_kernel(GemmArgs dw2, GemmArgs dh1) {
    int const tiles2 = (dw2.m / TILE) * (dw2.n / TN);
    int const b = int(blockIdx.x);
    if (b < tiles2)
        gemm_tile<1, 1, EPI_STORE>(dw2, Adam{}, b % (dw2.m / TILE), b / (dw2.m / TILE), 0, aligned_smem(), threadIdx.x);
    else
        gemm_tile<0, 1, EPI_MASK>(dh1, Adam{}, (b - tiles2) % (dh1.m / TILE), (b - tiles2) / (dh1.m / TILE), 0,
                                  aligned_smem(), threadIdx.x);
}

using GemmFn = void (*)(GemmArgs);
// (layouts other than 0, 0 run in the backward kernels; as plain products only for ta3w_gemm_test)
GemmFn gemm_fn(int a_mn, int b_mn) {
    return a_mn ? (b_mn ? gemm_kernel<1, 1> : gemm_kernel<1, 0>) : (b_mn ? gemm_kernel<0, 1> : gemm_kernel<0, 0>);
}

// ---------------------------------------------------------- model kernels ---
struct Dims {
    int in, inp, h;          // input size, padded to a multiple of 128; hidden width (multiple of 128)
    int64_t w1, w2, w3, b1, b2, b3, n;   // parameter offsets (FP32 vector) and count
};
inline Dims make_dims(int in, int h) {
    Dims d;
    d.in = in;
    d.inp = (in + TILE - 1) / TILE * TILE;     // the N of dW1 = dH1^T X: a whole number of tiles
    d.h = h;
    d.w1 = 0;
    d.w2 = d.w1 + int64_t(h) * d.inp;
    d.w3 = d.w2 + int64_t(h) * h;
    d.b1 = d.w3 + 2 * int64_t(h);
    d.b2 = d.b1 + h;
    d.b3 = d.b2 + h;
    d.n = d.b3 + 2;
    return d;
}

// standardised FP32 rows [rows][in] -> BF16 [rows][inp] (padding columns zero), 4 columns per thread;
// grid (inp / 4 / 128 rounded up, rows)
__global__ void pack_kernel(float const* __restrict__ x, int in, int inp, float const* __restrict__ mean,
                            float const* __restrict__ inv_std, __nv_bfloat16* __restrict__ xb) {
    int const c0 = 4 * int(blockIdx.x * blockDim.x + threadIdx.x);
    if (c0 >= inp) return;
    int64_t const r = blockIdx.y + int64_t(blockIdx.z) * gridDim.y;
    __nv_bfloat16 o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int const c = c0 + j;
        o[j] = __float2bfloat16_rn(c < in ? (x[r * in + c] - mean[c]) * inv_std[c] : 0.f);
    }
    *reinterpret_cast<uint2*>(xb + r * inp + c0) = *reinterpret_cast<uint2 const*>(o);
}

// H1 = BF16(relu(sum of the split partials + b1)), [rows][h], 4 values per thread (h a multiple of 128);
// the partials' loads are independent, their sum runs in split order
// (no __restrict__ on what the launches before wrote: non-coherent loads do not wait for them)
__global__ void act1_kernel(float const* part, int splits, int64_t split_stride, int64_t n, int h, float const* b1,
                            __nv_bfloat16* h1b) {
    int64_t const i = 4 * (int64_t(blockIdx.x) * blockDim.x + threadIdx.x);
    pdl_wait();
    pdl_go();
    if (i >= n) return;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int k = 0; k < splits; ++k) {
        float4 const p = __ldcg(reinterpret_cast<float4 const*>(part + k * split_stride + i));
        s.x += p.x;
        s.y += p.y;
        s.z += p.z;
        s.w += p.w;
    }
    float4 const b = *reinterpret_cast<float4 const*>(b1 + i % h);
    s.x += b.x;
    s.y += b.y;
    s.z += b.z;
    s.w += b.w;
    __nv_bfloat162 const lo = __floats2bfloat162_rn(s.x > 0.f ? s.x : 0.f, s.y > 0.f ? s.y : 0.f),
                         hi = __floats2bfloat162_rn(s.z > 0.f ? s.z : 0.f, s.w > 0.f ? s.w : 0.f);
    *reinterpret_cast<uint2*>(h1b + i) = make_uint2(*reinterpret_cast<uint32_t const*>(&lo),
                                                    *reinterpret_cast<uint32_t const*>(&hi));
}

// Output layer, loss and the first backward step, 32 rows per block:
//   z2 = F2 + b2, h2 = relu(z2), (mu, s) = W3 h2 + b3 (FP32, ascending);
//   training rows (y given, row valid): NLL 0.5 (s' + (y - mu)^2 e^-s'), s' = clamp(s, +-12),
//   dmu, ds of the batch mean, dH2 = BF16((z2 > 0) (dmu W3[0] + ds W3[1])).
// The two sums are one chain of h multiply-adds per row, so a lane owns a row (warp 0 the mean, warp 1 the
// log-variance) and reads it from shared memory; all threads move the rows in and out in whole lines. With
// one thread per row straight from global memory the kernel took 118 us for any number of rows.
constexpr int HEAD_ROWS = 32, HEAD_THREADS = 256;
inline size_t head_smem(int h) { return size_t(HEAD_ROWS * (h + 1) + 2 * h + 4 * HEAD_ROWS) * 4; }
__global__ void __launch_bounds__(HEAD_THREADS)
    head_kernel(float const* f2, int h, float const* p, int64_t off_w3, int64_t off_b2, int64_t off_b3,
                float const* y, RowMap map, float inv_n, float* out, float* h2f, float* gcols, float* row_loss,
                __nv_bfloat16* dh2b) {
    extern __shared__ uint8_t smem_raw[];
    float* const z = reinterpret_cast<float*>(smem_raw);       // [32][h + 1]
    float* const w3 = z + HEAD_ROWS * (h + 1);                 // [2][h]
    float* const o = w3 + 2 * h;                               // [2][32] outputs
    float* const gd = o + 2 * HEAD_ROWS;                       // [2][32] dmu, ds
    int const tid = threadIdx.x, r0 = int(blockIdx.x) * HEAD_ROWS;
    pdl_wait();
    pdl_go();
    for (int i = tid; i < h; i += HEAD_THREADS) {
        w3[i] = p[off_w3 + i];
        w3[h + i] = p[off_w3 + h + i];
    }
    // a warp moves whole rows (rows is a multiple of 128, h of 128): 16 bytes a lane, four rows in flight
    int const warp = tid >> 5, lane = tid & 31;
    for (int c = 4 * lane; c < h; c += 128) {
        float const* const bp = p + off_b2 + c;                 // (a multiple of 128: the widths before it are)
        float const b[4] = {bp[0], bp[1], bp[2], bp[3]};
        float4 q[HEAD_ROWS / 8];
#pragma unroll
        for (int k = 0; k < HEAD_ROWS / 8; ++k)
            q[k] = __ldcg(reinterpret_cast<float4 const*>(f2 + int64_t(r0 + warp + 8 * k) * h + c));
#pragma unroll
        for (int k = 0; k < HEAD_ROWS / 8; ++k) {
            int const r = warp + 8 * k;
            float const v[4] = {q[k].x + b[0], q[k].y + b[1], q[k].z + b[2], q[k].w + b[3]};
            float* const zr = z + r * (h + 1) + c;
#pragma unroll
            for (int j = 0; j < 4; ++j) zr[j] = v[j];
            if (h2f)
                *reinterpret_cast<float4*>(h2f + int64_t(r0 + r) * h + c) =
                    make_float4(v[0] > 0.f ? v[0] : 0.f, v[1] > 0.f ? v[1] : 0.f, v[2] > 0.f ? v[2] : 0.f, v[3] > 0.f ? v[3] : 0.f);
        }
    }
    __syncthreads();
    if (tid < 2 * HEAD_ROWS) {
        int const r = tid & (HEAD_ROWS - 1), which = tid / HEAD_ROWS;
        float const* const w = w3 + which * h;
        float const* const zr = z + r * (h + 1);
        float acc = p[off_b3 + which];
#pragma unroll 8
        for (int c = 0; c < h; ++c) acc = fmaf(zr[c] > 0.f ? zr[c] : 0.f, w[c], acc);
        o[which * HEAD_ROWS + r] = acc;
    }
    __syncthreads();
    if (tid < HEAD_ROWS) {
        int const r = r0 + tid;
        float const o0 = o[tid], o1 = o[HEAD_ROWS + tid];
        if (out) {
            out[2 * r] = o0;
            out[2 * r + 1] = o1;
        }
        if (y) {
            int const src = map.at(r);
            float dmu = 0.f, ds = 0.f, loss = 0.f;
            if (src >= 0) {
                float const s = fminf(fmaxf(o1, -12.f), 12.f);
                float const e = expf(-s);
                float const d = y[src] - o0;
                loss = 0.5f * (s + d * d * e);
                dmu = -d * e * inv_n;
                ds = (o1 > -12.f && o1 < 12.f) ? 0.5f * (1.f - d * d * e) * inv_n : 0.f;
            }
            gcols[2 * r] = dmu;
            gcols[2 * r + 1] = ds;
            row_loss[r] = loss;
            gd[tid] = dmu;
            gd[HEAD_ROWS + tid] = ds;
        }
    }
    if (!y) return;
    __syncthreads();
    for (int c = 2 * lane; c < h; c += 64) {
        float const wa = w3[c], wb = w3[c + 1], va = w3[h + c], vb = w3[h + c + 1];
#pragma unroll
        for (int k = 0; k < HEAD_ROWS / 8; ++k) {
            int const r = warp + 8 * k;
            float const dmu = gd[r], ds = gd[HEAD_ROWS + r];
            float const* const zr = z + r * (h + 1) + c;
            __nv_bfloat162 const v = __floats2bfloat162_rn(zr[0] > 0.f ? fmaf(dmu, wa, ds * va) : 0.f,
                                                           zr[1] > 0.f ? fmaf(dmu, wb, ds * vb) : 0.f);
            *reinterpret_cast<__nv_bfloat162*>(dh2b + int64_t(r0 + r) * h + c) = v;
        }
    }
}

// The column sums of the backward pass, over the batch rows in order: db1, db2 (of the BF16 dH1, dH2),
// dW3 = sum h2 [dmu, ds], db3, and the summed loss.
struct SmallGrads {
    int rows, h;
    __nv_bfloat16 const* dh1b;
    __nv_bfloat16 const* dh2b;
    float const* h2f;
    float const* gcols;
    float const* row_loss;
    float* grad;
    int64_t w3, b1, b2, b3;     // parameter offsets
    float* loss;
};

// Columns [32 cb, 32 cb + 32) of the hidden units (cb = h / 32: db3 and the loss): four warps, one sum of
// every column each; each sum is a chain over the rows, so the loads run ahead of it.
constexpr int SG_DEEP = 16;
template <class Load>
__device__ __forceinline__ float ordered_sum(int rows, Load load, bool fma_form) {
    float s = 0.f, a[SG_DEEP], b[SG_DEEP];
#pragma unroll
    for (int i = 0; i < SG_DEEP; ++i) load(i, a[i], b[i]);
    for (int r0 = 0; r0 < rows; r0 += SG_DEEP) {        // rows: a multiple of 128
        float na[SG_DEEP], nb[SG_DEEP];
        bool const more = r0 + SG_DEEP < rows;
#pragma unroll
        for (int i = 0; i < SG_DEEP; ++i) {
            na[i] = nb[i] = 0.f;
            if (more) load(r0 + SG_DEEP + i, na[i], nb[i]);
        }
#pragma unroll
        for (int i = 0; i < SG_DEEP; ++i) s = fma_form ? fmaf(a[i], b[i], s) : s + a[i];
#pragma unroll
        for (int i = 0; i < SG_DEEP; ++i) {
            a[i] = na[i];
            b[i] = nb[i];
        }
    }
    return s;
}

// the launch's other work beside the dW1 tiles (update: AdamW on what it computes, else into g.grad)
__device__ __forceinline__ void small_grads(SmallGrads const& g, Adam const& ad, bool update, int cb, int tid) {
    int const warp = tid >> 5, lane = tid & 31;
    if (warp >= 4) return;
    int64_t at = -1;
    float s = 0.f;
    if (cb < g.h / 32) {
        int const o = cb * 32 + lane;
        int64_t const h = g.h;
        if (warp < 2) {
            __nv_bfloat16 const* const src = warp == 0 ? g.dh1b : g.dh2b;
            at = (warp == 0 ? g.b1 : g.b2) + o;
            s = ordered_sum(g.rows, [&](int r, float& a, float&) { a = __bfloat162float(src[r * h + o]); }, false);
        } else {
            int const c = warp - 2;
            at = g.w3 + c * h + o;
            s = ordered_sum(g.rows, [&](int r, float& a, float& b) {
                a = g.h2f[r * h + o];
                b = g.gcols[2 * r + c];
            }, true);
        }
    } else if (warp == 0 && lane < 3) {
        if (lane < 2) at = g.b3 + lane;
        s = ordered_sum(g.rows, [&](int r, float& a, float&) { a = lane < 2 ? g.gcols[2 * r + lane] : g.row_loss[r]; }, false);
        if (lane == 2) *g.loss = s;
    }
    if (at < 0) return;
    if (update) ad.update(at, s);
    else g.grad[at] = s;
}

// AdamW on W2 (its gradient complete since the launch before) and W2's BF16 copy
constexpr int W2_PER_BLOCK = 4 * THREADS;
__device__ __forceinline__ void update_w2(Adam const& ad, float const* grad, int64_t off, int64_t n, __nv_bfloat16* w2b,
                                          int block, int tid) {
#pragma unroll
    for (int q = 0; q < W2_PER_BLOCK / THREADS; ++q) {
        int64_t const i = int64_t(block) * W2_PER_BLOCK + q * THREADS + tid;
        if (i < n) w2b[i] = __float2bfloat16_rn(ad.update(off + i, grad[off + i]));
    }
}

// The last launch of a step: the small gradients first (their chains are the longest), then W2's update,
// then dW1 = dH1^T X (M = h, N = inp, K = rows) tile by tile. UPDATE: each tile's AdamW runs in its
// epilogue, so W1's gradient is never written (and the separate pass over 1.3 M parameters is gone);
// otherwise the gradients are stored.
template <bool UPDATE>
__global__ void __launch_bounds__(THREADS, 2) last_kernel(GemmArgs dw1, SmallGrads sg, Adam ad, int64_t off_w2, __nv_bfloat16* w2b) {
    int const b = int(blockIdx.x), nsmall = sg.h / 32 + 1;
    int64_t const n2 = int64_t(sg.h) * sg.h;
    int const nw2 = UPDATE ? int((n2 + W2_PER_BLOCK - 1) / W2_PER_BLOCK) : 0;
    if (b < nsmall + nw2) {
        pdl_wait();
        pdl_go();
        if (b < nsmall) small_grads(sg, ad, UPDATE, b, threadIdx.x);
        else update_w2(ad, sg.grad, off_w2, n2, w2b, b - nsmall, threadIdx.x);
        return;
    }
    int const t = b - nsmall - nw2;
    gemm_tile<1, 1, UPDATE ? EPI_ADAM : EPI_STORE>(dw1, ad, t % (dw1.m / TILE), t / (dw1.m / TILE), 0, aligned_smem(),
                                                   threadIdx.x);
}

__global__ void refresh_kernel(float const* __restrict__ param, int64_t off_w2, int64_t off_w3,
                               __nv_bfloat16* __restrict__ w1b, __nv_bfloat16* __restrict__ w2b) {
    int64_t const i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < off_w2) w1b[i] = __float2bfloat16_rn(param[i]);
    else if (i < off_w3) w2b[i - off_w2] = __float2bfloat16_rn(param[i]);
}

} // namespace ta3w

using namespace ta3w;

struct ta3w_model {
    int device = 0;
    int sms = 0;
    Dims d{};
    std::string err;
    cudaStream_t stream = nullptr;
    float* d_param = nullptr;
    float* d_m = nullptr;
    float* d_v = nullptr;
    float* d_grad = nullptr;
    __nv_bfloat16* d_w1b = nullptr;
    __nv_bfloat16* d_w2b = nullptr;
    uint32_t* d_status = nullptr;
    float* d_loss = nullptr;
    float* d_stats = nullptr;          // mean [inp], inv_std [inp]
    float y_mean = 0.f, y_std = 1.f;
    // data
    uint32_t rows = 0;
    size_t cap_rows = 0;
    float* d_xraw = nullptr;
    __nv_bfloat16* d_x = nullptr;
    float* d_y = nullptr;
    int32_t* d_idx = nullptr;
    size_t cap_idx = 0;
    // activations for up to cap_act rows (a multiple of 128)
    size_t cap_act = 0;
    int max_splits = 1;
    float* d_f1 = nullptr;             // [splits][rows][h]
    __nv_bfloat16* d_h1b = nullptr;
    float* d_f2 = nullptr;
    float* d_h2f = nullptr;
    float* d_gcols = nullptr;
    float* d_rowloss = nullptr;
    __nv_bfloat16* d_dh2b = nullptr;
    __nv_bfloat16* d_dh1b = nullptr;
    float* d_out = nullptr;
    uint64_t adam_t = 0;
};

namespace {
thread_local std::string g_werr;

#define TA3W_CUDA(m, call, what)                                                               \
    do {                                                                                       \
        cudaError_t const e_ = (call);                                                         \
        if (e_ != cudaSuccess) return wfail(m, std::string(what) + ": " + cudaGetErrorString(e_)); \
    } while (0)

int wfail(ta3w_model* m, std::string msg) {
    if (m) m->err = msg;
    g_werr = msg;
    return 1;
}

template <class T>
int wgrow(ta3w_model* m, T*& ptr, size_t& cap, size_t n, char const* what) {
    if (n <= cap && ptr) return 0;
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    TA3W_CUDA(m, cudaMalloc(&ptr, std::max<size_t>(n, 1) * sizeof(T)), what);
    cap = n;
    return 0;
}
template <class T>
int walloc(ta3w_model* m, T*& ptr, size_t n, char const* what) {
    size_t cap = 0;
    return wgrow(m, ptr, cap, n, what);
}

int round128(int n) { return (n + TILE - 1) / TILE * TILE; }
// rows of one forward / backward pass: bounds the activation buffers (split-K partials
// of the first layer alone take splits x rows x H floats)
constexpr uint32_t kMaxPassRows = 65536;

// activation buffers for `rows` (a multiple of 128) rows
int ensure_act(ta3w_model* m, size_t rows) {
    if (rows <= m->cap_act) return 0;
    int const h = m->d.h;
    int const splits = m->max_splits;
    for (void* p : {(void*)m->d_f1, (void*)m->d_h1b, (void*)m->d_f2, (void*)m->d_h2f, (void*)m->d_gcols,
                    (void*)m->d_rowloss, (void*)m->d_dh2b, (void*)m->d_dh1b, (void*)m->d_out})
        if (p) cudaFree(p);
    m->d_f1 = m->d_f2 = m->d_h2f = m->d_gcols = m->d_rowloss = m->d_out = nullptr;
    m->d_h1b = m->d_dh2b = m->d_dh1b = nullptr;
    m->cap_act = 0;
    if (walloc(m, m->d_f1, size_t(splits) * rows * h, "alloc F1") || walloc(m, m->d_h1b, rows * h, "alloc H1") ||
        walloc(m, m->d_f2, rows * h, "alloc F2") || walloc(m, m->d_h2f, rows * h, "alloc H2") ||
        walloc(m, m->d_gcols, rows * 2, "alloc G") || walloc(m, m->d_rowloss, rows, "alloc loss rows") ||
        walloc(m, m->d_dh2b, rows * h, "alloc dH2") || walloc(m, m->d_dh1b, rows * h, "alloc dH1") ||
        walloc(m, m->d_out, rows * 2, "alloc outputs"))
        return 1;
    m->cap_act = rows;
    return 0;
}

// a launch that may start while the one before it on the stream drains (each kernel waits with pdl_wait
// before it touches what another launch wrote)
template <class... Args>
int launch(ta3w_model* m, char const* what, void (*fn)(Args...), dim3 grid, int threads, size_t smem, Args... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(unsigned(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = m->stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    TA3W_CUDA(m, cudaLaunchKernelEx(&cfg, fn, args...), what);
    return 0;
}

int splits_for(ta3w_model* m, int M, int N, int K) {
    int const tiles = (M / TILE) * (N / TILE);
    int const want = std::max(1, (m->sms + tiles - 1) / tiles);
    return std::min({want, K / KS, m->max_splits});
}

// forward (and with train the backward pass) over `valid_rows` rows of x [..][inp] BF16, selected by idx
// (device, -1 = none; null: rows 0 .. valid_rows - 1), padded to a multiple of 128 here. ad: the step's
// AdamW, applied as the gradients come; without it they go to d_grad.
int pass(ta3w_model* m, __nv_bfloat16 const* x, int32_t const* idx, int valid_rows, bool train, Adam const* ad = nullptr) {
    Dims const& d = m->d;
    int const R = round128(valid_rows);
    if (ensure_act(m, size_t(R))) return 1;
    int const h = d.h;
    RowMap const rows{idx, valid_rows};
    // layer 1: F1 = X W1^T (M = rows, N = h, K = inp), split over K
    int const s1 = splits_for(m, R, h, d.inp);
    int const per = (d.inp / KS + s1 - 1) / s1;
    int const s1_used = (d.inp / KS + per - 1) / per;
    int64_t const n_act = int64_t(R) * h;
    GemmArgs f1{};
    f1.a = x, f1.lda = d.inp, f1.map = rows, f1.mapped = 1;
    f1.b = m->d_w1b, f1.ldb = d.inp;
    f1.c = m->d_f1, f1.ldc = h, f1.c_split = n_act;
    f1.m = R, f1.n = h, f1.k = d.inp, f1.k_split = per * KS, f1.status = m->d_status;
    if (launch(m, "layer 1", gemm_kernel<0, 0>, dim3(unsigned(R / TILE), unsigned(h / TN), unsigned(s1_used)), THREADS,
               SMEM_BYTES, f1))
        return 1;
    if (launch(m, "act1", act1_kernel, dim3(unsigned((n_act / 4 + 127) / 128)), 128, 0, (float const*)m->d_f1, s1_used,
               n_act, n_act, h, (float const*)(m->d_param + d.b1), m->d_h1b))
        return 1;
    // layer 2: F2 = H1 W2^T
    GemmArgs f2{};
    f2.a = m->d_h1b, f2.lda = h, f2.b = m->d_w2b, f2.ldb = h;
    f2.c = m->d_f2, f2.ldc = h, f2.m = R, f2.n = h, f2.k = h, f2.k_split = h, f2.status = m->d_status;
    if (launch(m, "layer 2", gemm_kernel<0, 0>, dim3(unsigned(R / TILE), unsigned(h / TN), 1), THREADS, SMEM_BYTES, f2))
        return 1;
    if (launch(m, "head", head_kernel, dim3(unsigned(R / HEAD_ROWS)), HEAD_THREADS, head_smem(h),
               (float const*)m->d_f2, h, (float const*)m->d_param, d.w3, d.b2, d.b3,
               (float const*)(train ? m->d_y : nullptr), rows, 1.0f / float(valid_rows), m->d_out,
               train ? m->d_h2f : (float*)nullptr, m->d_gcols, m->d_rowloss, m->d_dh2b))
        return 1;
    if (!train) return 0;
    // dW2 = dH2^T H1 (M = h out, N = h in, K = rows) and dH1 = mask(dH2 W2) (M = rows, N = h in, K = h out)
    GemmArgs dw2{}, dh1{};
    dw2.a = m->d_dh2b, dw2.lda = h, dw2.b = m->d_h1b, dw2.ldb = h;
    dw2.c = m->d_grad + d.w2, dw2.ldc = h, dw2.m = h, dw2.n = h, dw2.k = R, dw2.k_split = R, dw2.status = m->d_status;
    dh1.a = m->d_dh2b, dh1.lda = h, dh1.b = m->d_w2b, dh1.ldb = h;
    dh1.ldc = h, dh1.m = R, dh1.n = h, dh1.k = h, dh1.k_split = h, dh1.status = m->d_status;
    dh1.mask = m->d_h1b, dh1.out16 = m->d_dh1b;
    if (launch(m, "backward 2", backward_kernel, dim3(unsigned((h / TILE) * (h / TN) + (R / TILE) * (h / TN))), THREADS,
               SMEM_BYTES, dw2, dh1))
        return 1;
    GemmArgs dw1{};
    dw1.a = m->d_dh1b, dw1.lda = h, dw1.b = x, dw1.ldb = d.inp, dw1.map = rows, dw1.mapped = 1;
    dw1.c = m->d_grad + d.w1, dw1.ldc = d.inp, dw1.m = h, dw1.n = d.inp, dw1.k = R, dw1.k_split = R;
    dw1.status = m->d_status, dw1.out16 = m->d_w1b, dw1.live_n = d.in;
    SmallGrads const sg{R, h, m->d_dh1b, m->d_dh2b, m->d_h2f, m->d_gcols, m->d_rowloss, m->d_grad,
                        d.w3, d.b1, d.b2, d.b3, m->d_loss};
    int const tiles = (h / TILE) * (d.inp / TN), small = h / 32 + 1;
    int const w2_blocks = int((int64_t(h) * h + W2_PER_BLOCK - 1) / W2_PER_BLOCK);
    if (ad)
        return launch(m, "backward 1 and update", last_kernel<true>, dim3(unsigned(small + w2_blocks + tiles)), THREADS,
                      SMEM_BYTES, dw1, sg, *ad, d.w2, m->d_w2b);
    return launch(m, "backward 1", last_kernel<false>, dim3(unsigned(small + tiles)), THREADS, SMEM_BYTES, dw1, sg, Adam{},
                  d.w2, m->d_w2b);
}

int check_status(ta3w_model* m) {
    uint32_t st = 0;
    TA3W_CUDA(m, cudaMemcpyAsync(&st, m->d_status, 4, cudaMemcpyDeviceToHost, m->stream), "status");
    TA3W_CUDA(m, cudaStreamSynchronize(m->stream), "surrogate kernels");
    if (st) return wfail(m, "surrogate: a tensor-core wait timed out");
    return 0;
}

// the rows on the device, standardised in BF16 (with `standardize` by their own statistics, which stay for
// later predictions). They take the place of the training rows, also when it fails half-way: no training
// set from here until a set_data call is complete.
int upload_rows(ta3w_model* m, float const* x, uint32_t n, bool standardize) {
    Dims const& d = m->d;
    m->rows = 0;
    if (n > m->cap_rows) {
        size_t c1 = 0, c2 = 0, c3 = 0;
        if (m->d_xraw) cudaFree(m->d_xraw);
        if (m->d_x) cudaFree(m->d_x);
        if (m->d_y) cudaFree(m->d_y);
        m->d_xraw = nullptr;
        m->d_x = nullptr;
        m->d_y = nullptr;
        m->cap_rows = 0;
        if (wgrow(m, m->d_xraw, c1, size_t(n) * d.in, "alloc rows") ||
            wgrow(m, m->d_x, c2, size_t(n) * d.inp, "alloc rows") || wgrow(m, m->d_y, c3, n, "alloc targets"))
            return 1;
        m->cap_rows = n;
    }
    TA3W_CUDA(m, cudaMemcpyAsync(m->d_xraw, x, size_t(n) * d.in * 4, cudaMemcpyHostToDevice, m->stream), "copy rows");
    if (standardize)
        TA3W_CUDA(m, ta3_stats::column_stats(m->d_xraw, int(n), d.in, d.in, m->d_stats, m->d_stats + d.inp, m->stream),
                  "column statistics");
    uint32_t const fold = 32768, cols = unsigned((d.inp / 4 + 127) / 128);      // grid y and z hold at most 65,535
    for (uint32_t r0 = 0; r0 < n;) {
        uint32_t const left = n - r0, ny = std::min(left, fold), nz = std::min(left / ny, 32768u);
        pack_kernel<<<dim3(cols, ny, nz), 128, 0, m->stream>>>(m->d_xraw + size_t(r0) * d.in, d.in, d.inp, m->d_stats,
                                                               m->d_stats + d.inp, m->d_x + size_t(r0) * d.inp);
        TA3W_CUDA(m, cudaGetLastError(), "pack");
        r0 += ny * nz;
    }
    return 0;
}

} // namespace

extern "C" {

uint32_t ta3w_num_params(uint32_t in_dim, uint32_t hidden) {
    if (in_dim == 0 || hidden == 0 || hidden % TILE) return 0;
    return uint32_t(make_dims(int(in_dim), int(hidden)).n);
}

ta3w_model* ta3w_create(int device, uint32_t in_dim, uint32_t hidden, uint32_t seed) {
    if (in_dim == 0 || in_dim > (1u << 20) || hidden == 0 || hidden % TILE || hidden > 1024) {
        g_werr = "ta3w_create: in_dim in 1..2^20, hidden a multiple of 128 up to 1024";
        return nullptr;
    }
    auto* m = new ta3w_model;
    m->device = device;
    m->d = make_dims(int(in_dim), int(hidden));
    auto bad = [&](std::string what) {
        g_werr = "ta3w_create: " + what;
        ta3w_destroy(m);
        return static_cast<ta3w_model*>(nullptr);
    };
    cudaDeviceProp prop{};
    if (cudaSetDevice(device) != cudaSuccess || cudaGetDeviceProperties(&prop, device) != cudaSuccess)
        return bad("no such device");
    if (prop.major != 10) return bad("needs an sm_100 (B200) device");
    m->sms = prop.multiProcessorCount;
    m->max_splits = 16;
    auto smem = [](auto* fn, size_t bytes) {
        return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)) == cudaSuccess;
    };
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b)
            if (!smem(gemm_fn(a, b), SMEM_BYTES)) return bad("smem attribute");
    if (!smem(backward_kernel, SMEM_BYTES) || !smem(last_kernel<true>, SMEM_BYTES) || !smem(last_kernel<false>, SMEM_BYTES) ||
        !smem(head_kernel, head_smem(1024)))
        return bad("smem attribute");
    if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) return bad("stream");
    Dims const& d = m->d;
    size_t const np = size_t(d.n);
    if (walloc(m, m->d_param, np, "params") || walloc(m, m->d_m, np, "adam m") || walloc(m, m->d_v, np, "adam v") ||
        walloc(m, m->d_grad, np, "grad") || walloc(m, m->d_w1b, size_t(d.h) * d.inp, "w1 bf16") ||
        walloc(m, m->d_w2b, size_t(d.h) * d.h, "w2 bf16") || walloc(m, m->d_status, 1, "status") ||
        walloc(m, m->d_loss, 2, "loss") || walloc(m, m->d_stats, 2 * size_t(d.inp), "stats"))
        return bad(m->err);
    // He-uniform init for the ReLU layers, small output layer (mt19937 + uniform_real_distribution)
    std::mt19937 rng(seed);
    auto uni = [&](float a) { return std::uniform_real_distribution<float>(-a, a)(rng); };
    std::vector<float> w(np, 0.f);
    for (int o = 0; o < d.h; ++o)
        for (int i = 0; i < d.in; ++i) w[size_t(d.w1) + size_t(o) * d.inp + i] = uni(std::sqrt(6.f / float(d.in)));
    for (int64_t k = 0; k < int64_t(d.h) * d.h; ++k) w[size_t(d.w2 + k)] = uni(std::sqrt(6.f / float(d.h)));
    for (int k = 0; k < 2 * d.h; ++k) w[size_t(d.w3) + k] = uni(std::sqrt(1.f / float(d.h)));
    if (ta3w_set_params(m, w.data())) return bad(m->err);
    std::vector<float> stats(2 * size_t(d.inp), 0.f);
    std::fill(stats.begin() + d.inp, stats.end(), 1.f);
    // on the model's stream: its kernels run on a non-blocking stream, which does not wait for the
    // legacy default stream (a pageable cudaMemcpy can even return before its DMA has landed)
    if (cudaMemcpyAsync(m->d_stats, stats.data(), stats.size() * 4, cudaMemcpyHostToDevice, m->stream) != cudaSuccess ||
        cudaMemsetAsync(m->d_status, 0, 4, m->stream) != cudaSuccess ||
        cudaStreamSynchronize(m->stream) != cudaSuccess)
        return bad("init copies");
    return m;
}

void ta3w_destroy(ta3w_model* m) {
    if (!m) return;
    cudaSetDevice(m->device);
    for (void* p : {(void*)m->d_param, (void*)m->d_m, (void*)m->d_v, (void*)m->d_grad, (void*)m->d_w1b,
                    (void*)m->d_w2b, (void*)m->d_status, (void*)m->d_loss, (void*)m->d_stats, (void*)m->d_xraw,
                    (void*)m->d_x, (void*)m->d_y, (void*)m->d_idx, (void*)m->d_f1, (void*)m->d_h1b, (void*)m->d_f2,
                    (void*)m->d_h2f, (void*)m->d_gcols, (void*)m->d_rowloss, (void*)m->d_dh2b, (void*)m->d_dh1b,
                    (void*)m->d_out})
        if (p) cudaFree(p);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
}

const char* ta3w_last_error(const ta3w_model* m) { return m ? m->err.c_str() : g_werr.c_str(); }

uint32_t ta3w_model_params(const ta3w_model* m) { return m ? uint32_t(m->d.n) : 0u; }

int ta3w_set_params(ta3w_model* m, const float* params) {
    if (!m || !params) return wfail(m, "ta3w_set_params: null argument");
    Dims const& d = m->d;
    TA3W_CUDA(m, cudaSetDevice(m->device), "set device");
    std::vector<float> p(params, params + d.n);
    for (int o = 0; o < d.h; ++o)       // padding columns of W1 stay zero
        for (int i = d.in; i < d.inp; ++i) p[size_t(d.w1) + size_t(o) * d.inp + i] = 0.f;
    // on the model's (non-blocking) stream, ahead of the refresh kernel that reads them
    TA3W_CUDA(m, cudaMemcpyAsync(m->d_param, p.data(), size_t(d.n) * 4, cudaMemcpyHostToDevice, m->stream), "params");
    TA3W_CUDA(m, cudaMemsetAsync(m->d_m, 0, size_t(d.n) * 4, m->stream), "adam m");
    TA3W_CUDA(m, cudaMemsetAsync(m->d_v, 0, size_t(d.n) * 4, m->stream), "adam v");
    m->adam_t = 0;
    refresh_kernel<<<unsigned((d.w3 + 255) / 256), 256, 0, m->stream>>>(m->d_param, d.w2, d.w3, m->d_w1b, m->d_w2b);
    TA3W_CUDA(m, cudaGetLastError(), "refresh");
    TA3W_CUDA(m, cudaStreamSynchronize(m->stream), "refresh");
    return 0;
}

int ta3w_get_params(ta3w_model* m, float* params_out) {
    if (!m || !params_out) return wfail(m, "ta3w_get_params: null argument");
    TA3W_CUDA(m, cudaSetDevice(m->device), "set device");
    TA3W_CUDA(m, cudaStreamSynchronize(m->stream), "sync");
    TA3W_CUDA(m, cudaMemcpy(params_out, m->d_param, size_t(m->d.n) * 4, cudaMemcpyDeviceToHost), "params");
    return 0;
}

static int set_data_impl(ta3w_model* m, const float* x, const float* y, uint32_t n, bool standardize) {
    Dims const& d = m->d;
    TA3W_CUDA(m, cudaSetDevice(m->device), "set device");
    std::vector<float> stats(2 * size_t(d.inp), 0.f);
    std::fill(stats.begin() + d.inp, stats.end(), 1.f);
    m->rows = 0;      // (until the call is complete)
    m->y_mean = 0.f;
    m->y_std = 1.f;
    bool const host_stats = standardize && ta3_stats::stats_on_host(n, size_t(d.in));
    if (host_stats) ta3_stats::host_column_stats(x, n, size_t(d.in), stats.data(), stats.data() + d.inp);
    if (standardize) {
        double s = 0, s2 = 0;
        for (uint32_t r = 0; r < n; ++r) s += y[r];
        double const mu = s / n;
        for (uint32_t r = 0; r < n; ++r) s2 += (y[r] - mu) * (y[r] - mu);
        m->y_mean = float(mu);
        m->y_std = s2 > 0 ? float(std::sqrt(s2 / n)) : 1.f;
    }
    TA3W_CUDA(m, cudaMemcpyAsync(m->d_stats, stats.data(), stats.size() * 4, cudaMemcpyHostToDevice, m->stream),
              "stats");
    if (upload_rows(m, x, n, standardize && !host_stats)) return 1;
    std::vector<float> ys(n);
    for (uint32_t r = 0; r < n; ++r) ys[r] = (y[r] - m->y_mean) / m->y_std;
    TA3W_CUDA(m, cudaMemcpyAsync(m->d_y, ys.data(), size_t(n) * 4, cudaMemcpyHostToDevice, m->stream), "targets");
    TA3W_CUDA(m, cudaStreamSynchronize(m->stream), "set data");
    m->rows = n;
    return 0;
}

int ta3w_set_data(ta3w_model* m, const float* x, const float* y, uint32_t n) {
    if (!m || !x || !y || n == 0) return wfail(m, "ta3w_set_data: need n > 0 rows");
    return set_data_impl(m, x, y, n, true);
}

int ta3w_set_data_standardized(ta3w_model* m, const float* x, const float* y, uint32_t n) {
    if (!m || !x || !y || n == 0) return wfail(m, "ta3w_set_data_standardized: need n > 0 rows");
    return set_data_impl(m, x, y, n, false);
}

int ta3w_gradients(ta3w_model* m, float* grad_out, float* loss_sum_out) {
    if (!m || !grad_out) return wfail(m, "ta3w_gradients: null argument");
    if (m->rows == 0) return wfail(m, "ta3w_gradients: no data");
    if (m->rows > kMaxPassRows) return wfail(m, "ta3w_gradients: at most 65,536 rows in one pass");
    TA3W_CUDA(m, cudaSetDevice(m->device), "set device");
    TA3W_CUDA(m, cudaMemsetAsync(m->d_status, 0, 4, m->stream), "status");
    TA3W_CUDA(m, cudaMemsetAsync(m->d_grad, 0, size_t(m->d.n) * 4, m->stream), "grad");
    if (pass(m, m->d_x, nullptr, int(m->rows), true)) return 1;
    if (check_status(m)) return 1;
    TA3W_CUDA(m, cudaMemcpy(grad_out, m->d_grad, size_t(m->d.n) * 4, cudaMemcpyDeviceToHost), "grad");
    if (loss_sum_out) TA3W_CUDA(m, cudaMemcpy(loss_sum_out, m->d_loss, 4, cudaMemcpyDeviceToHost), "loss");
    return 0;
}

int ta3w_train(ta3w_model* m, uint32_t epochs, uint32_t batch, float lr, float weight_decay, uint32_t seed,
               float* final_loss) {
    if (!m || batch == 0 || batch > kMaxPassRows) return wfail(m, "ta3w_train: batch must be 1 .. 65,536");
    if (m->rows == 0) return wfail(m, "ta3w_train: no data");
    TA3W_CUDA(m, cudaSetDevice(m->device), "set device");
    uint32_t const n = m->rows;
    uint32_t const steps = (n + batch - 1) / batch;
    size_t const total = size_t(epochs) * steps * batch;
    std::vector<int32_t> idx(std::max<size_t>(total, 1), -1);
    std::mt19937 rng(seed);
    std::vector<int32_t> perm(n);
    for (uint32_t e = 0; e < epochs; ++e) {
        std::iota(perm.begin(), perm.end(), 0);
        std::shuffle(perm.begin(), perm.end(), rng);
        for (uint32_t s = 0; s < steps; ++s)
            for (uint32_t b = 0; b < batch; ++b) {
                uint32_t const k = s * batch + b;
                idx[(size_t(e) * steps + s) * batch + b] = k < n ? perm[k] : -1;
            }
    }
    if (wgrow(m, m->d_idx, m->cap_idx, idx.size(), "alloc indices")) return 1;
    TA3W_CUDA(m, cudaMemcpyAsync(m->d_idx, idx.data(), idx.size() * 4, cudaMemcpyHostToDevice, m->stream), "indices");
    TA3W_CUDA(m, cudaMemsetAsync(m->d_status, 0, 4, m->stream), "status");
    float const b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    float last_loss = 0.f;
    uint32_t last_rows = 0;
    for (uint32_t e = 0; e < epochs; ++e)
        for (uint32_t s = 0; s < steps; ++s) {
            uint32_t const rows_here = std::min(batch, n - s * batch);
            float const t = float(m->adam_t + 1);
            float const c1 = 1.f - std::pow(b1, t), c2 = 1.f - std::pow(b2, t);
            Adam const ad{m->d_param, m->d_m, m->d_v, lr, b1, b2, eps, c1, c2, weight_decay};
            if (pass(m, m->d_x, m->d_idx + (size_t(e) * steps + s) * batch, int(rows_here), true, &ad)) return 1;
            ++m->adam_t;
            last_rows = rows_here;
        }
    if (check_status(m)) return 1;
    if (final_loss) {
        TA3W_CUDA(m, cudaMemcpy(&last_loss, m->d_loss, 4, cudaMemcpyDeviceToHost), "loss");
        *final_loss = last_rows ? last_loss / float(last_rows) : 0.f;
    }
    return 0;
}

int ta3w_predict(ta3w_model* m, const float* x, uint32_t n, float* mean_out, float* logvar_out) {
    if (!m || !x || !mean_out) return wfail(m, "ta3w_predict: null argument");
    if (n == 0) return 0;
    TA3W_CUDA(m, cudaSetDevice(m->device), "set device");
    if (upload_rows(m, x, n, false)) return 1;
    TA3W_CUDA(m, cudaMemsetAsync(m->d_status, 0, 4, m->stream), "status");
    uint32_t const chunk = 4096;
    std::vector<float> out(size_t(n) * 2);
    for (uint32_t r0 = 0; r0 < n; r0 += chunk) {
        uint32_t const k = std::min(chunk, n - r0);
        if (pass(m, m->d_x + size_t(r0) * m->d.inp, nullptr, int(k), false)) return 1;
        TA3W_CUDA(m, cudaMemcpyAsync(out.data() + size_t(r0) * 2, m->d_out, size_t(k) * 8, cudaMemcpyDeviceToHost,
                                     m->stream), "outputs");
    }
    if (check_status(m)) return 1;
    for (uint32_t r = 0; r < n; ++r) {
        mean_out[r] = out[2 * r] * m->y_std + m->y_mean;
        if (logvar_out) logvar_out[r] = out[2 * r + 1] + 2.f * std::log(m->y_std);
    }
    return 0;
}

// Test hook: C = A B^T-style product of the GEMM kernel on host BF16 data (bit
// patterns as uint16), both operands given in their global layouts; c [m][n].
int ta3w_gemm_test(int device, int a_mn, int b_mn, int m, int n, int k, int splits, const uint16_t* a,
                   const uint16_t* b, float* c) {
    if (m <= 0 || n <= 0 || k <= 0 || m % TILE || n % TILE || k % KS || splits < 1) {
        g_werr = "ta3w_gemm_test: m, n multiples of 128, k of 64";
        return 1;
    }
    ta3w_model tmp;
    tmp.device = device;
    ta3w_model* mm = &tmp;
    TA3W_CUDA(mm, cudaSetDevice(device), "set device");
    cudaDeviceProp prop{};
    TA3W_CUDA(mm, cudaGetDeviceProperties(&prop, device), "properties");
    if (prop.major != 10) return wfail(mm, "needs an sm_100 device");
    tmp.sms = prop.multiProcessorCount;
    TA3W_CUDA(mm, cudaFuncSetAttribute(gemm_fn(a_mn, b_mn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(SMEM_BYTES)), "smem attribute");
    __nv_bfloat16 *da = nullptr, *db = nullptr;
    float* dc = nullptr;
    uint32_t* ds = nullptr;
    int const kst = k / KS;
    int const per = (kst + splits - 1) / splits;
    int const used = (kst + per - 1) / per;
    int rc = 0;
    if (cudaMalloc(&da, size_t(m) * k * 2) != cudaSuccess || cudaMalloc(&db, size_t(n) * k * 2) != cudaSuccess ||
        cudaMalloc(&dc, size_t(used) * m * n * 4) != cudaSuccess || cudaMalloc(&ds, 4) != cudaSuccess) {
        rc = wfail(mm, "alloc");
    } else {
        cudaMemcpy(da, a, size_t(m) * k * 2, cudaMemcpyHostToDevice);
        cudaMemcpy(db, b, size_t(n) * k * 2, cudaMemcpyHostToDevice);
        cudaMemset(ds, 0, 4);
        GemmArgs g{};
        g.a = da, g.lda = a_mn ? m : k, g.b = db, g.ldb = b_mn ? n : k;
        g.c = dc, g.ldc = n, g.c_split = int64_t(m) * n, g.m = m, g.n = n, g.k = k, g.k_split = per * KS, g.status = ds;
        gemm_fn(a_mn, b_mn)<<<dim3(m / TILE, n / TN, used), THREADS, SMEM_BYTES>>>(g);
        cudaError_t e = cudaDeviceSynchronize();
        uint32_t st = 0;
        if (e == cudaSuccess) e = cudaMemcpy(&st, ds, 4, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) rc = wfail(mm, std::string("gemm: ") + cudaGetErrorString(e));
        else if (st) rc = wfail(mm, "gemm: a tensor-core wait timed out");
        else {
            std::vector<float> part(size_t(used) * m * n);
            cudaMemcpy(part.data(), dc, part.size() * 4, cudaMemcpyDeviceToHost);
            for (size_t i = 0; i < size_t(m) * n; ++i) {
                float s = 0.f;
                for (int q = 0; q < used; ++q) s += part[size_t(q) * m * n + i];
                c[i] = s;
            }
        }
    }
    for (void* p : {(void*)da, (void*)db, (void*)dc, (void*)ds})
        if (p) cudaFree(p);
    if (rc) g_werr = tmp.err;
    return rc;
}

} // extern "C"
