// Surrogate fitness model for CMA-ES pre-screening: an MLP 97 -> 128 -> 128 -> 2
// (predicted mean score, log-variance) trained by Gaussian negative log-likelihood
// with Adam. No counterpart in the reference; the trainer calls it through
// include/ta3b_surrogate.h.
//
// Tensor-core path (sm_100a): every 128x128 GEMM of the forward and backward
// pass is a tcgen05.mma (kind::f16, BF16 operands from shared memory, FP32
// accumulators in tensor memory) issued by one thread; the 2-wide output layer,
// the loss and the elementwise parts run on the CUDA cores from TMEM values.
// One CTA (16 warps, ~200 KB shared memory, all 512 TMEM columns) per SM; four
// threads own batch row t of a 128-row tile for the elementwise work (32 columns
// each) and TMEM lane t (= output row t of every MMA).
//
// Training runs whole: one launch of a cluster of eight CTAs loops over the steps.
// Up to eight of them compute a tile of the minibatch each and write their gradient
// partials; after a cluster barrier all eight update their share of the parameters,
// whose FP32 values and Adam moments stay in registers from step to step, and write the
// new weights straight into the tile CTAs' shared memory; another barrier starts the
// next step. A step of 256 rows is bound by the latency of its chain of small products
// and barriers: 20 us (of it the update 3, the gradients' way out 3), where a launch of the tile kernel and one of the Adam kernel
// took 41 us. (Minibatches of more than eight tiles still take those two launches.)
//
// Shared-memory operand layout (no swizzle): a 128 x 128 BF16 tile stores
// element (r, c) at byte (r/8)*2048 + (c/8)*128 + (r%8)*16 + (c%8)*2, i.e. 8x8
// "core matrices" of 128 contiguous bytes. The same bytes read as
//   K-major with rows as M/N:  LBO = 128 (next 8 columns), SBO = 2048 (next 8 rows)
//   MN-major with rows as K:   LBO = 2048 (next 8 rows = K), SBO = 128 (next 8 columns = M/N)
// so an activation tile written once by its row owners serves both as the
// A operand of a row-major GEMM (M = batch) and as an operand of the weight
// gradient GEMMs (K = batch) without a transpose.
//
// Descriptor encodings follow the PTX ISA tcgen05 shared-memory and instruction
// descriptors (field layout as in CUTLASS cute/arch/mma_sm100_desc.hpp).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <numeric>
#include <random>
#include <string>
#include <vector>

#include "../../include/ta3b_surrogate.h"
#include "column_stats.cuh"

namespace ta3s {

constexpr int IN = 97;          // v11 parameter count
constexpr int IN_K = 112;       // first-layer K, padded to a multiple of 16
constexpr int HID = 128;
constexpr int ROWS = 128;       // batch rows per tile = MMA M
constexpr int THREADS = 512;    // four per row of the tile
constexpr int CLUSTER = 8;      // CTAs of a training launch

// flat FP32 parameter vector (also the gradient layout)
constexpr int OFF_W1 = 0;                       // [128][112] (o, i); i >= 97 stays zero
constexpr int OFF_W2 = OFF_W1 + HID * IN_K;     // [128][128] (o, i)
constexpr int OFF_W3 = OFF_W2 + HID * HID;      // [2][128]
constexpr int OFF_B1 = OFF_W3 + 2 * HID;
constexpr int OFF_B2 = OFF_B1 + HID;
constexpr int OFF_B3 = OFF_B2 + HID;
constexpr int NPARAM = OFF_B3 + 2;              // 31234
constexpr int PARTIAL = NPARAM + 2;             // + loss sum + valid rows

// shared memory map (bytes from a 1024-aligned base)
constexpr uint32_t TILE_BYTES = 128 * 128 * 2;
constexpr uint32_t S_X = 0, S_W1 = S_X + TILE_BYTES, S_W2 = S_W1 + TILE_BYTES, S_H1 = S_W2 + TILE_BYTES,
                   S_H2 = S_H1 + TILE_BYTES, S_D1 = S_H2 + TILE_BYTES, S_G = S_D1 + TILE_BYTES;   // S_G: [128][16]
constexpr uint32_t S_F32 = S_G + 128 * 16 * 2;  // W3 [2][128], b1, b2 [128], b3 [2]
constexpr uint32_t S_ROW = S_F32 + (4 * HID + 4) * 4;   // per row: source row, mean, log-variance, dmu, ds
constexpr uint32_t S_BAR = S_ROW + 5 * ROWS * 4;
constexpr uint32_t S_TMEM = S_BAR + 8;
constexpr uint32_t SMEM_BYTES = S_TMEM + 8 + 1024;   // + alignment slack
constexpr int COLS = 32;                        // a thread's columns of its row
constexpr uint32_t S_OUT = S_H1;                // the gradient tiles on their way out: [128][132] FP32 over H1, H2, D1
constexpr int LDT = 132;
static_assert(ROWS * LDT * 4 <= 3 * int(TILE_BYTES) && S_BAR % 8 == 0 && SMEM_BYTES <= 232448, "shared memory");

// TMEM columns
constexpr uint32_t T_F1 = 0, T_F2 = 128, T_DW2 = 256, T_DW1 = 384, T_SMALL = 496;

constexpr long long WAIT_LIMIT_CYCLES = 4000000000LL;   // ~2 s at 1.9 GHz

__host__ __device__ constexpr uint32_t tile_off(int r, int c) {
    return uint32_t((r >> 3) * 2048 + (c >> 3) * 128 + (r & 7) * 16 + (c & 7) * 2);
}
__host__ __device__ constexpr uint32_t gtile_off(int r, int c) {   // [128][16] tile
    return uint32_t((r >> 3) * 256 + (c >> 3) * 128 + (r & 7) * 16 + (c & 7) * 2);
}

// tcgen05 shared-memory matrix descriptor: start, LBO, SBO (all >> 4), version 1, no swizzle
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return uint64_t((saddr >> 4) & 0x3FFF) | (uint64_t((lbo >> 4) & 0x3FFF) << 16) |
           (uint64_t((sbo >> 4) & 0x3FFF) << 32) | (uint64_t(1) << 46);
}

// instruction descriptor: D F32, A/B BF16, majors (0 = K, 1 = MN), N, M = 128
__host__ __device__ constexpr uint32_t instr_desc(int n, int a_mn, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(a_mn) << 15) | (uint32_t(b_mn) << 16) |
           (uint32_t(n >> 3) << 17) | (uint32_t(ROWS >> 4) << 24);
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

// consecutive FP32 columns of this thread's TMEM lane; the values are there after tmem_wait
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
// 32 columns at once (one wait for twice the columns)
__device__ __forceinline__ void tmem_ld32(uint32_t addr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, void const* src, bool valid) {   // zeros when not valid
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// this CTA's shared-memory address, as CTA `rank` of the cluster has it
__device__ __forceinline__ uint32_t map_rank(uint32_t saddr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// bounded wait for the barrier phase with the given parity; false on timeout
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

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    __nv_bfloat162 const h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t const*>(&h);
}
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// 8 FP32 values -> one 16-byte BF16 chunk of a tile
__device__ __forceinline__ uint4 st_chunk(uint8_t* smem, uint32_t off, float const* v) {
    uint4 q;
    q.x = pack_bf16(v[0], v[1]);
    q.y = pack_bf16(v[2], v[3]);
    q.z = pack_bf16(v[4], v[5]);
    q.w = pack_bf16(v[6], v[7]);
    *reinterpret_cast<uint4*>(smem + off) = q;
    return q;
}

// What a tile reads and writes.
struct Params {
    __nv_bfloat16 const* x;     // [rows][128] standardised inputs (columns >= 97 zero)
    float const* y;             // [rows] standardised targets (training)
    int32_t const* idx;         // batch row indices, or null for rows 0..batch-1
    int batch;
    __nv_bfloat16 const* w1;    // [128][128] (o, i), i >= 97 zero
    __nv_bfloat16 const* w2;    // [128][128] (o, i)
    float const* p32;           // FP32 parameters (W3 and biases read from here)
    float* out;                 // prediction: [batch][2]
    float* partial;             // training: [gridDim.x][PARTIAL]
    uint32_t* status;           // nonzero: a tensor-core wait timed out
    float inv_batch;
    int train;
};

// One CTA's shared memory, tensor memory and running sums.
struct Block {
    uint8_t* sm;
    uint32_t sbase, tmem, bar, lane_base;
    int tid, warp, row, part;               // this thread's tile row, and which 32 of the 128 columns it takes
    float *w3s, *b1s, *b2s, *b3s;           // W3 [2][128], b1, b2 [128], b3 [2]
    int32_t* src;                           // per row: its source row, -1 = none
    float *o0s, *o1s, *dmus, *dss;          // per row
    volatile uint32_t* abort_s;             // block-uniform stop
    uint32_t phase;
    bool ok;
    uint32_t* status;
    float acc_w3a, acc_w3b, acc_b1, acc_b2;             // threads 0..127: lane = feature
    float acc_b3a, acc_b3b, acc_loss, acc_rows;         // threads 384..511: row owner
    bool first;                                          // no tile accumulated yet

    __device__ void open(uint8_t* smem_raw, uint32_t* status_word) {
        sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
        sbase = uint32_t(__cvta_generic_to_shared(sm));
        tid = int(threadIdx.x);
        warp = tid >> 5;
        row = tid & (ROWS - 1);
        part = tid >> 7;
        w3s = reinterpret_cast<float*>(sm + S_F32);
        b1s = w3s + 2 * HID;
        b2s = b1s + HID;
        b3s = b2s + HID;
        src = reinterpret_cast<int32_t*>(sm + S_ROW);
        o0s = reinterpret_cast<float*>(src + ROWS);
        o1s = o0s + ROWS;
        dmus = o1s + ROWS;
        dss = dmus + ROWS;
        bar = sbase + S_BAR;
        abort_s = reinterpret_cast<volatile uint32_t*>(sm + S_TMEM + 4);
        status = status_word;
        phase = 0;
        ok = true;
        if (tid == 0) {
            mbar_init(bar);
            *abort_s = 0u;
        }
        if (warp == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + S_TMEM),
                         "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        fence_before();
        __syncthreads();
        fence_after();
        tmem = *reinterpret_cast<uint32_t volatile*>(sm + S_TMEM);
        lane_base = tmem + (uint32_t((warp & 3) * 32) << 16);
        start();
    }
    __device__ void start() {                // no tile accumulated
        first = true;
        acc_w3a = acc_w3b = acc_b1 = acc_b2 = acc_b3a = acc_b3b = acc_loss = acc_rows = 0.f;
    }
    __device__ void close() {
        fence_before();
        __syncthreads();
        fence_after();
        if (warp == 0)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }

    // every thread waits for the last commit; a timeout is recorded and makes the whole block stop at the
    // next tile boundary (all threads read the flag after a barrier)
    __device__ void sync_mma() {
        if (ok && !mbar_wait(bar, phase)) {
            ok = false;
            *abort_s = 1u;
            atomicOr(status, 1u);
        }
        phase ^= 1u;
        fence_after();
    }
    __device__ void publish() {              // smem writes + TMEM reads done -> MMA may run
        fence_async_smem();
        fence_before();
        __syncthreads();
        fence_after();
    }

    // a 128-row, 256-byte-wide BF16 matrix into its tile, 16 bytes a copy: two neighbouring threads take a
    // 32-byte sector, sixteen threads 256 bytes of the tile
    template <class RowOf>
    __device__ void load_tile(uint32_t dst, __nv_bfloat16 const* base, RowOf row_of) {   // (row -1: zeros)
#pragma unroll
        for (int q = 0; q < ROWS * 16 / THREADS; ++q) {
            int const c = tid + THREADS * q, j = 2 * ((c >> 4) & 7) + (c & 1), r = 8 * (c >> 7) + ((c >> 1) & 7);
            int const from = row_of(r);
            cp_async16(sbase + dst + tile_off(r, 8 * j), base + size_t(from < 0 ? 0 : from) * 128 + 8 * j, from >= 0);
        }
    }
    __device__ void load_weights(Params const& p) {
        load_tile(S_W1, p.w1, [](int r) { return r; });
        load_tile(S_W2, p.w2, [](int r) { return r; });
        for (int i = tid; i < 4 * HID + 2; i += THREADS)         // W3, b1, b2, b3 in the parameter vector's order
            w3s[i] = __ldcg(p.p32 + OFF_W3 + i);
    }
    __device__ void load_rows(Params const& p, int tile) {       // the X tile and its rows' sources
        __syncthreads();                                         // (the last tile's rows are done with)
        if (tid < ROWS) {
            int const r = tile * ROWS + tid;
            src[tid] = r < p.batch ? (p.idx ? __ldg(p.idx + r) : r) : -1;
        }
        __syncthreads();
        load_tile(S_X, p.x, [&](int r) { return src[r]; });
    }

    // forward and backward of the tile in shared memory (weights and rows loaded or on their way)
    __device__ void run_tile(Params const& p, int tile) {
        uint32_t const x_s = sbase + S_X, w1_s = sbase + S_W1, w2_s = sbase + S_W2, h1_s = sbase + S_H1,
                       h2_s = sbase + S_H2, d1_s = sbase + S_D1, g_s = sbase + S_G;
        uint32_t const id128_kk = instr_desc(128, 0, 0), id128_mm = instr_desc(128, 1, 1),
                       id128_km = instr_desc(128, 0, 1), id112_mm = instr_desc(IN_K, 1, 1),
                       id16_mm = instr_desc(16, 1, 1);
        int const c0 = COLS * part, srow = src[row];
        bool const valid = srow >= 0, last = part == 3;
        float const yv = p.train && last && valid ? __ldg(p.y + srow) : 0.f;
        cp_async_wait();
        publish();
        // ---- layer 1: H1 = X W1^T (M = rows, N = 128, K = 112)
        if (tid == 0) {
            for (int kk = 0; kk < IN_K / 16; ++kk)
                mma_bf16(tmem + T_F1, smem_desc(x_s + kk * 256, 128, 2048), smem_desc(w1_s + kk * 256, 128, 2048),
                         id128_kk, kk > 0);
            mma_commit(bar);
        }
        sync_mma();
        float h[COLS];
        tmem_ld32(lane_base + T_F1 + c0, h);
#pragma unroll
        for (int j = 0; j < COLS; ++j) h[j] = fmaxf(h[j] + b1s[c0 + j], 0.f);
        uint32_t m1 = 0u, m2 = 0u;           // relu masks of layers 1 (of the stored BF16 values) and 2, this thread's columns
#pragma unroll
        for (int j = 0; j < COLS; j += 8) {
            uint4 const q = st_chunk(sm + S_H1, tile_off(row, c0 + j), h + j);
            uint32_t const w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {    // (relu's results: positive unless all bits are zero)
                m1 |= (w[i] & 0x7FFFu) ? 1u << (j + 2 * i) : 0u;
                m1 |= (w[i] & 0x7FFF0000u) ? 2u << (j + 2 * i) : 0u;
            }
        }
        publish();
        // ---- layer 2: H2 = relu(H1) W2^T
        if (tid == 0) {
            for (int kk = 0; kk < HID / 16; ++kk)
                mma_bf16(tmem + T_F2, smem_desc(h1_s + kk * 256, 128, 2048), smem_desc(w2_s + kk * 256, 128, 2048),
                         id128_kk, kk > 0);
            mma_commit(bar);
        }
        sync_mma();
        // ---- output layer on the CUDA cores (FP32): mean, log-variance; one chain over the columns in
        // order, so each of the row's threads goes on where the one before ended
        tmem_ld32(lane_base + T_F2 + c0, h);
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
            float const z = h[j] + b2s[c0 + j];
            h[j] = fmaxf(z, 0.f);
            m2 |= z > 0.f ? 1u << j : 0u;
        }
        if (p.train) {
#pragma unroll
            for (int j = 0; j < COLS; j += 8) st_chunk(sm + S_H2, tile_off(row, c0 + j), h + j);
        }
        float o0 = b3s[0], o1 = b3s[1];
        for (int q = 0; q < 4; ++q) {
            if (part == q) {
                if (q) {
                    o0 = o0s[row];
                    o1 = o1s[row];
                }
#pragma unroll
                for (int j = 0; j < COLS; ++j) {
                    o0 = fmaf(h[j], w3s[c0 + j], o0);
                    o1 = fmaf(h[j], w3s[HID + c0 + j], o1);
                }
                o0s[row] = o0;
                o1s[row] = o1;
            }
            if (q < 3) __syncthreads();
        }
        if (last) {
            if (!p.train) {
                if (valid) {
                    size_t const r = size_t(tile) * ROWS + row;
                    p.out[2 * r] = o0;
                    p.out[2 * r + 1] = o1;
                }
            } else {
                // ---- Gaussian NLL 0.5 * (s + (y - mu)^2 e^-s), mean over the batch
                float dmu = 0.f, ds = 0.f;
                if (valid) {
                    float const s = fminf(fmaxf(o1, -12.f), 12.f);
                    float const e = expf(-s);
                    float const d = yv - o0;
                    acc_loss += 0.5f * (s + d * d * e);
                    acc_rows += 1.f;
                    dmu = -d * e * p.inv_batch;
                    ds = (o1 > -12.f && o1 < 12.f) ? 0.5f * (1.f - d * d * e) * p.inv_batch : 0.f;
                }
                acc_b3a += dmu;
                acc_b3b += ds;
                dmus[row] = dmu;
                dss[row] = ds;
                float g[16] = {valid ? 1.f : 0.f, dmu, ds, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
                st_chunk(sm + S_G, gtile_off(row, 0), g);
                st_chunk(sm + S_G, gtile_off(row, 8), g + 8);
            }
        }
        if (!p.train) {
            fence_before();
            __syncthreads();
            fence_after();
            ok = *abort_s == 0u;
            return;
        }
        __syncthreads();
        // ---- dH2 = (dmu W3[0] + ds W3[1]) * relu'(H2), into the D1 tile
        {
            float const dmu = dmus[row], ds = dss[row];
#pragma unroll
            for (int j = 0; j < COLS; ++j)
                h[j] = (m2 >> j) & 1u ? fmaf(dmu, w3s[c0 + j], ds * w3s[HID + c0 + j]) : 0.f;
#pragma unroll
            for (int j = 0; j < COLS; j += 8) st_chunk(sm + S_D1, tile_off(row, c0 + j), h + j);
        }
        publish();
        // ---- dW3^T[i][c] = sum_b H2[b][i] G[b][c] (M = feature, N = 16, K = rows) and dH1 = dH2 W2, which
        // the next step waits for; behind them db2 = column sums of dH2 (its 16 columns over F2, which has
        // been read) and dW2 += dH2^T H1, which the last commit covers
        if (tid == 0) {
            for (int kk = 0; kk < ROWS / 16; ++kk)
                mma_bf16(tmem + T_SMALL, smem_desc(h2_s + kk * 4096, 2048, 128), smem_desc(g_s + kk * 512, 256, 128),
                         id16_mm, kk > 0);
            for (int kk = 0; kk < HID / 16; ++kk)
                mma_bf16(tmem + T_F1, smem_desc(d1_s + kk * 256, 128, 2048), smem_desc(w2_s + kk * 4096, 2048, 128),
                         id128_km, kk > 0);
            mma_commit(bar);
            for (int kk = 0; kk < ROWS / 16; ++kk)
                mma_bf16(tmem + T_F2, smem_desc(d1_s + kk * 4096, 2048, 128), smem_desc(g_s + kk * 512, 256, 128),
                         id16_mm, kk > 0);
            for (int kk = 0; kk < ROWS / 16; ++kk)
                mma_bf16(tmem + T_DW2, smem_desc(d1_s + kk * 4096, 2048, 128), smem_desc(h1_s + kk * 4096, 2048, 128),
                         id128_mm, (!first || kk > 0) ? 1u : 0u);
        }
        sync_mma();
        if (part == 0) {
            float v[16];
            tmem_ld16(lane_base + T_SMALL, v);
            acc_w3a += v[1];
            acc_w3b += v[2];
        }
        // ---- dH1 = (dH2 W2) * relu'(H1), into the H2 tile (its product has completed)
        tmem_ld32(lane_base + T_F1 + c0, h);
#pragma unroll
        for (int j = 0; j < COLS; ++j)
            if (!((m1 >> j) & 1u)) h[j] = 0.f;
#pragma unroll
        for (int j = 0; j < COLS; j += 8) st_chunk(sm + S_H2, tile_off(row, c0 + j), h + j);
        publish();
        // ---- dW1 += dH1^T X (N = 112), db1 = column sums of dH1
        if (tid == 0) {
            for (int kk = 0; kk < ROWS / 16; ++kk)
                mma_bf16(tmem + T_SMALL, smem_desc(h2_s + kk * 4096, 2048, 128), smem_desc(g_s + kk * 512, 256, 128),
                         id16_mm, kk > 0);
            for (int kk = 0; kk < ROWS / 16; ++kk)
                mma_bf16(tmem + T_DW1, smem_desc(h2_s + kk * 4096, 2048, 128), smem_desc(x_s + kk * 4096, 2048, 128),
                         id112_mm, (!first || kk > 0) ? 1u : 0u);
            mma_commit(bar);
        }
        sync_mma();
        if (part == 0) {
            float v[16];
            tmem_ld16(lane_base + T_SMALL, v);
            acc_b1 += v[0];
            tmem_ld16(lane_base + T_F2, v);
            acc_b2 += v[0];
        }
        first = false;
        fence_before();
        __syncthreads();
        fence_after();
        ok = *abort_s == 0u;
    }

    // one weight gradient ([128][cols] from `off` of the parameter vector) from TMEM through shared memory, so
    // that rows go out in whole lines
    template <int COLUMNS>
    __device__ void write_gradient(uint32_t t_col, bool have, float* dst) {
        float* const t = reinterpret_cast<float*>(sm + S_OUT);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            int const c = COLS * part + 16 * u;
            if (c < COLUMNS) {                                   // (uniform over a warp)
                float v[16];
                if (have) {
                    tmem_ld16(lane_base + t_col + c, v);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = 0.f;
                }
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (COLUMNS == IN_K && c + j >= IN) v[j] = 0.f;
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    *reinterpret_cast<float4*>(t + row * LDT + c + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            }
        }
        __syncthreads();
        constexpr int QUADS = COLUMNS / 4;
#pragma unroll
        for (int q = 0; q < HID * QUADS / THREADS; ++q) {
            int const i = tid + THREADS * q, r = i / QUADS, c = 4 * (i % QUADS);
            *reinterpret_cast<float4*>(dst + r * COLUMNS + c) = *reinterpret_cast<float4 const*>(t + r * LDT + c);
        }
        __syncthreads();
    }
    // this CTA's gradient partials
    __device__ void write_partial(float* out) {
        float* const red = reinterpret_cast<float*>(sm + S_G);
        bool const have = ok && !first;
        if (part == 3) {                                         // row-owned sums, added in row order below
            red[row] = acc_b3a;
            red[ROWS + row] = acc_b3b;
            red[2 * ROWS + row] = acc_loss;
            red[3 * ROWS + row] = acc_rows;
        }
        if (part == 0) {
            out[OFF_W3 + tid] = acc_w3a;
            out[OFF_W3 + HID + tid] = acc_w3b;
            out[OFF_B1 + tid] = acc_b1;
            out[OFF_B2 + tid] = acc_b2;
        }
        write_gradient<HID>(T_DW2, have, out + OFF_W2);
        if (tid >= THREADS - 4) {
            int const k = tid - (THREADS - 4);
            float s = 0.f;
#pragma unroll 16
            for (int r = 0; r < ROWS; ++r) s += red[k * ROWS + r];
            out[k < 2 ? OFF_B3 + k : NPARAM + k - 2] = s;
        }
        write_gradient<IN_K>(T_DW1, have, out + OFF_W1);
    }
};

// predictions, or one pass's gradient partials: tiles dealt to the CTAs in turn
__global__ void __launch_bounds__(THREADS, 1) mlp_kernel(Params p) {
    extern __shared__ uint8_t smem_raw[];
    Block b;
    b.open(smem_raw, p.status);
    b.load_weights(p);
    int const ntiles = (p.batch + ROWS - 1) / ROWS;
    for (int tile = int(blockIdx.x); tile < ntiles && b.ok; tile += int(gridDim.x)) {
        b.load_rows(p, tile);
        b.run_tile(p, tile);
    }
    if (p.train) b.write_partial(p.partial + size_t(blockIdx.x) * PARTIAL);
    b.close();
}

// AdamW's constants; one parameter's step from its gradient
struct AdamConst {
    float lr, b1, b2, eps, wd;
    __device__ __forceinline__ float step(float g, float c1, float c2, float& m, float& v, float w) const {
        m = b1 * m + (1.f - b1) * g;
        v = b2 * v + (1.f - b2) * g * g;
        return w - lr * (m / c1) / (sqrtf(v / c2) + eps) - lr * wd * w;
    }
};
__device__ __forceinline__ bool is_padding(int i) { return i < OFF_W2 && (i % IN_K) >= IN; }
// the BF16 copy of parameter i (W1, W2)
__device__ __forceinline__ void store_bf16(int i, float w, __nv_bfloat16* w1b, __nv_bfloat16* w2b) {
    if (i < OFF_W2) w1b[(i / IN_K) * 128 + i % IN_K] = __float2bfloat16_rn(w);
    else if (i < OFF_W3) w2b[i - OFF_W2] = __float2bfloat16_rn(w);
}

// `steps` training steps in one launch of one cluster (minibatches of at most CLUSTER tiles).
struct TrainArgs {
    Params p;                    // idx: the first step's rows; batch: rows of a full minibatch
    int steps, first_step;       // steps of this launch; how many of the call came before
    int steps_per_epoch, rows;   // the last minibatch of an epoch has what is left of the rows
    float const* c1;             // [steps] bias corrections 1 - b1^t, 1 - b2^t
    float const* c2;
    float* param;
    float* m;
    float* v;
    __nv_bfloat16* w1b;
    __nv_bfloat16* w2b;
    AdamConst adam;
    float* loss_out;             // the last step's summed loss and rows
};
constexpr int OWN = 8;           // parameters per thread: eight in a row are one 16-byte chunk of a BF16 tile
static_assert(CLUSTER * THREADS * OWN >= NPARAM && IN_K % OWN == 0 && OFF_W2 % OWN == 0 && OFF_W3 % OWN == 0 &&
              PARTIAL % 4 == 0, "the cluster owns every parameter, in whole chunks of the weight matrices");

__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(THREADS, 1) train_kernel(TrainArgs a) {
    extern __shared__ uint8_t smem_raw[];
    int const rank = int(blockIdx.x), tid = int(threadIdx.x);
    Block b;
    b.open(smem_raw, a.p.status);
    // this thread's parameters; values and moments stay in registers
    int const i0 = (rank * THREADS + tid) * OWN;
    auto owned = [&](int k) { return i0 + k < NPARAM; };
    float w[OWN], m[OWN], v[OWN];
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
        w[k] = owned(k) ? a.param[i0 + k] : 0.f;
        m[k] = owned(k) ? a.m[i0 + k] : 0.f;
        v[k] = owned(k) ? a.v[i0 + k] : 0.f;
    }
    // where they live in a tile CTA's shared memory: a BF16 chunk of W1 or W2, or FP32 words of W3 and the
    // biases (in the parameter vector's order; the last chunk's words past b3 are padding)
    uint32_t const home = b.sbase + (i0 < OFF_W2   ? S_W1 + tile_off(i0 / IN_K, i0 % IN_K)
                                     : i0 < OFF_W3 ? S_W2 + tile_off((i0 - OFF_W2) / HID, (i0 - OFF_W2) % HID)
                                                   : S_F32 + 4u * uint32_t(i0 - OFF_W3));
    auto minibatch = [&](int s) {                       // step s of this launch
        Params p = a.p;
        int const in_epoch = (a.first_step + s) % a.steps_per_epoch;
        p.batch = min(a.p.batch, a.rows - in_epoch * a.p.batch);
        p.idx = a.p.idx + size_t(s) * a.p.batch;
        p.inv_batch = 1.0f / float(p.batch);
        return p;
    };
    auto tiles = [](Params const& p) { return (p.batch + ROWS - 1) / ROWS; };
    Params p = minibatch(0);
    // CTAs that ever take a tile: their weights stay in shared memory (a minibatch has no more rows than there
    // are, and the cluster no more CTAs than its tiles were checked for)
    int const most = (min(a.p.batch, a.rows) + ROWS - 1) / ROWS;
    if (rank < most) b.load_weights(p);
    if (rank < tiles(p)) b.load_rows(p, rank);
    for (int s = 0; s < a.steps; ++s) {
        int const n = tiles(p);
        float const c1 = __ldg(a.c1 + s), c2 = __ldg(a.c2 + s);
        if (rank < n) {
            b.start();
            b.run_tile(p, rank);
            b.write_partial(p.partial + size_t(rank) * PARTIAL);
        } else {
            cp_async_wait();                            // (weights on their way must not land on the update's)
        }
        Params const next = s + 1 < a.steps ? minibatch(s + 1) : p;
        if (s + 1 < a.steps && rank < tiles(next)) b.load_rows(next, rank);     // on their way during the update
        cluster_sync();
        if (*reinterpret_cast<volatile uint32_t*>(a.p.status)) break;           // (set before the barrier: all see it)
        if (i0 < NPARAM) {
            float g[OWN];
#pragma unroll
            for (int k = 0; k < OWN; ++k) g[k] = 0.f;
            for (int q = 0; q < n; ++q) {               // the partials in CTA order
                float const* const from = p.partial + size_t(q) * PARTIAL + i0;
                float4 const lo = __ldcg(reinterpret_cast<float4 const*>(from));
                float4 const hi = owned(4) ? __ldcg(reinterpret_cast<float4 const*>(from + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
                float const t[OWN] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int k = 0; k < OWN; ++k) g[k] += t[k];
            }
#pragma unroll
            for (int k = 0; k < OWN; ++k)
                if (owned(k) && !is_padding(i0 + k)) w[k] = a.adam.step(g[k], c1, c2, m[k], v[k], w[k]);
            for (int q = 0; q < most; ++q) {
                uint32_t const at = map_rank(home, q);
                if (i0 < OFF_W3) {
                    st_cluster128(at, pack_bf16(w[0], w[1]), pack_bf16(w[2], w[3]), pack_bf16(w[4], w[5]),
                                  pack_bf16(w[6], w[7]));
                } else {
                    st_cluster128(at, __float_as_uint(w[0]), __float_as_uint(w[1]), __float_as_uint(w[2]), __float_as_uint(w[3]));
                    if (owned(4))
                        st_cluster128(at + 16, __float_as_uint(w[4]), __float_as_uint(w[5]), __float_as_uint(w[6]),
                                      __float_as_uint(w[7]));
                }
            }
        }
        if (s + 1 == a.steps && rank == 0 && tid < 2) {
            float t = 0.f;
            for (int q = 0; q < n; ++q) t += __ldcg(p.partial + size_t(q) * PARTIAL + NPARAM + tid);
            a.loss_out[tid] = t;
        }
        cluster_sync();
        p = next;
    }
#pragma unroll
    for (int k = 0; k < OWN; ++k)
        if (owned(k)) {
            a.param[i0 + k] = w[k];
            a.m[i0 + k] = m[k];
            a.v[i0 + k] = v[k];
            if (!is_padding(i0 + k)) store_bf16(i0 + k, w[k], a.w1b, a.w2b);
        }
    cp_async_wait();
    b.close();
}

// Adam over the flat parameter vector; gradients summed over the CTA partials
// in a fixed order (deterministic). Refreshes the BF16 weight copies. The update
// of minibatches that one cluster cannot hold.
__global__ void adam_kernel(float* __restrict__ param, float* __restrict__ m, float* __restrict__ v,
                            float const* __restrict__ partial, int nparts, AdamConst ad, float c1, float c2,
                            __nv_bfloat16* __restrict__ w1b, __nv_bfloat16* __restrict__ w2b, float* __restrict__ loss_out) {
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= PARTIAL) return;
    float g = 0.f;
    for (int k = 0; k < nparts; ++k) g += partial[size_t(k) * PARTIAL + i];
    if (i >= NPARAM) {
        loss_out[i - NPARAM] = g;
        return;
    }
    if (is_padding(i)) return;
    float mi = m[i], vi = v[i];
    float const w = ad.step(g, c1, c2, mi, vi, param[i]);
    m[i] = mi;
    v[i] = vi;
    param[i] = w;
    store_bf16(i, w, w1b, w2b);
}

// a pass's gradient (and loss, rows) from the CTA partials, in CTA order
__global__ void sum_kernel(float const* __restrict__ partial, int nparts, float* __restrict__ out) {
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= PARTIAL) return;
    float g = 0.f;
    for (int k = 0; k < nparts; ++k) g += partial[size_t(k) * PARTIAL + i];
    out[i] = g;
}

// BF16 weight copies from the FP32 parameters
__global__ void refresh_kernel(float const* __restrict__ param, __nv_bfloat16* __restrict__ w1b,
                               __nv_bfloat16* __restrict__ w2b) {
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 128 * 128) {
        int const o = i / 128, c = i % 128;
        w1b[i] = __float2bfloat16_rn(c < IN ? param[OFF_W1 + o * IN_K + c] : 0.f);
        w2b[i] = __float2bfloat16_rn(param[OFF_W2 + i]);
    }
}

// standardised FP32 rows -> BF16 [rows][128]
__global__ void pack_kernel(float const* __restrict__ x, int rows, float const* __restrict__ mean,
                            float const* __restrict__ inv_std, __nv_bfloat16* __restrict__ xb) {
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * 128) return;
    int const r = i / 128, c = i % 128;
    float const v = c < IN ? (x[size_t(r) * IN + c] - mean[c]) * inv_std[c] : 0.f;
    xb[i] = __float2bfloat16_rn(v);
}

} // namespace ta3s

using namespace ta3s;

struct ta3s_model {
    int device = 0;
    int sms = 0;
    std::string err;
    std::mt19937 rng;
    float* d_param = nullptr;     // FP32 master parameters
    float* d_m = nullptr;
    float* d_v = nullptr;
    __nv_bfloat16* d_w1b = nullptr;
    __nv_bfloat16* d_w2b = nullptr;
    float* d_partial = nullptr;   // [sms][PARTIAL]
    uint32_t* d_status = nullptr;
    float* d_loss = nullptr;      // [2]
    // data
    size_t cap_rows = 0;
    float* d_xraw = nullptr;
    __nv_bfloat16* d_x = nullptr;
    float* d_y = nullptr;
    int32_t* d_idx = nullptr;
    size_t cap_idx = 0;
    float* d_grad = nullptr;      // [PARTIAL]: a pass's summed gradient, loss and rows
    float* d_stats = nullptr;     // mean[128], inv_std[128]
    // page-locked and mapped: the status word, then predictions [rows][2], which the kernel writes there
    // itself (two copies into pageable memory cost a prediction of 800 rows 20 of its 80 us)
    uint32_t* h_status = nullptr;
    bool unchecked = false;       // kernels launched whose status no call has found to be zero
    float* h_out = nullptr;
    size_t cap_out = 0;
    float* d_out = nullptr;       // predictions of more rows than kMappedRows
    size_t cap_dout = 0;
    float* d_corr = nullptr;      // a training call's bias corrections
    size_t cap_corr = 0;
    float y_mean = 0.f, y_std = 1.f;
    uint32_t rows = 0;
    uint64_t adam_t = 0;
    cudaStream_t stream = nullptr;
};

namespace {
thread_local std::string g_err;

#define TA3S_CUDA(m, call, what)                                                           \
    do {                                                                                   \
        cudaError_t const e_ = (call);                                                     \
        if (e_ != cudaSuccess) return fail(m, std::string(what) + ": " + cudaGetErrorString(e_)); \
    } while (0)

int fail(ta3s_model* m, std::string msg) {
    if (m) m->err = msg;
    g_err = msg;
    return 1;
}

template<class T>
int grow(ta3s_model* m, T*& ptr, size_t& cap, size_t n, char const* what) {
    if (n <= cap && ptr) return 0;
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    TA3S_CUDA(m, cudaMalloc(&ptr, n * sizeof(T)), what);
    cap = n;
    return 0;
}

// the status word is zero between calls; a call that failed between its kernels and check_status may have left a bit
int begin_kernels(ta3s_model* m) {
    if (m->unchecked) TA3S_CUDA(m, cudaMemsetAsync(m->d_status, 0, 4, m->stream), "status");
    m->unchecked = true;
    return 0;
}
// waits for the call's kernels
int check_status(ta3s_model* m) {
    TA3S_CUDA(m, cudaMemcpyAsync(m->h_status, m->d_status, 4, cudaMemcpyDeviceToHost, m->stream), "status");
    TA3S_CUDA(m, cudaStreamSynchronize(m->stream), "surrogate kernels");
    if (*m->h_status) return fail(m, "surrogate: a tensor-core wait timed out");
    m->unchecked = false;
    return 0;
}

// Predictions of up to this many rows go into page-locked memory, 8 bytes a row (2 MB at most); more of them through
// device memory and a copy. Page-locking saves the copy on every call but costs a model's first one: 200,000 rows
// take 5.7 ms (6.0 with the copy), the first time 7.4 (8.2); 300,000 rows 10.3 (10.6) and 13.8 (12.1); 1,000,000 rows
// 36.5 (37.1) and 45 (39).
constexpr uint32_t kMappedRows = 262144;

// page-locked room for n rows' predictions
int grow_out(ta3s_model* m, size_t n) {
    if (n <= m->cap_out) return 0;
    if (m->h_out) cudaFreeHost(m->h_out);
    m->h_out = nullptr;
    m->cap_out = 0;
    TA3S_CUDA(m, cudaHostAlloc(&m->h_out, n * 2 * sizeof(float), cudaHostAllocMapped), "alloc predictions");
    m->cap_out = n;
    return 0;
}

// the rows on the device, standardised in BF16 (with `standardize` by their own statistics, which stay for
// later predictions). They take the place of the training rows, also when it fails half-way: no training
// set from here until a set_data call is complete.
int upload_rows(ta3s_model* m, float const* x, uint32_t n, bool standardize) {
    m->rows = 0;
    if (n > m->cap_rows) {
        size_t c1 = 0, c2 = 0, c3 = 0;
        m->cap_rows = 0;      // (grow frees first: after a failure there is no room for any rows)
        if (grow(m, m->d_xraw, c1, size_t(n) * IN, "alloc rows") || grow(m, m->d_x, c2, size_t(n) * 128, "alloc rows") ||
            grow(m, m->d_y, c3, n, "alloc targets"))
            return 1;
        m->cap_rows = n;
    }
    TA3S_CUDA(m, cudaMemcpyAsync(m->d_xraw, x, size_t(n) * IN * 4, cudaMemcpyHostToDevice, m->stream), "copy rows");
    if (standardize)
        TA3S_CUDA(m, ta3_stats::column_stats(m->d_xraw, int(n), IN, IN, m->d_stats, m->d_stats + 128, m->stream),
                  "column statistics");
    pack_kernel<<<(n * 128 + 255) / 256, 256, 0, m->stream>>>(m->d_xraw, int(n), m->d_stats, m->d_stats + 128, m->d_x);
    TA3S_CUDA(m, cudaGetLastError(), "pack");
    return 0;
}

Params make_params(ta3s_model* m, int batch, int32_t const* d_idx, int train, float* out = nullptr) {
    Params prm{};
    prm.x = m->d_x;
    prm.y = m->d_y;
    prm.idx = d_idx;
    prm.batch = batch;
    prm.w1 = m->d_w1b;
    prm.w2 = m->d_w2b;
    prm.p32 = m->d_param;
    prm.out = out;
    prm.partial = m->d_partial;
    prm.status = m->d_status;
    prm.inv_batch = 1.0f / float(batch);
    prm.train = train;
    return prm;
}

int launch_mlp(ta3s_model* m, int batch, int32_t const* d_idx, int train, float* out = nullptr) {
    int const ntiles = (batch + ROWS - 1) / ROWS;
    int const grid = std::min(ntiles, m->sms);
    mlp_kernel<<<grid, THREADS, SMEM_BYTES, m->stream>>>(make_params(m, batch, d_idx, train, out));
    TA3S_CUDA(m, cudaGetLastError(), "surrogate mlp launch");
    return 0;
}

} // namespace

extern "C" {

uint32_t ta3s_num_params(void) { return NPARAM; }

ta3s_model* ta3s_create(int device, uint32_t seed) {
    auto* m = new ta3s_model;
    m->device = device;
    m->rng.seed(seed);
    auto bad = [&](char const* what, cudaError_t e) {
        g_err = std::string("ta3s_create: ") + what + ": " + cudaGetErrorString(e);
        delete m;
        return static_cast<ta3s_model*>(nullptr);
    };
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return bad("set device", e);
    cudaDeviceProp prop{};
    e = cudaGetDeviceProperties(&prop, device);
    if (e != cudaSuccess) return bad("device properties", e);
    if (prop.major != 10) {
        g_err = "ta3s_create: needs an sm_100 (B200) device";
        delete m;
        return nullptr;
    }
    m->sms = prop.multiProcessorCount;
    if ((e = cudaFuncSetAttribute(mlp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(SMEM_BYTES))) !=
            cudaSuccess ||
        (e = cudaFuncSetAttribute(train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(SMEM_BYTES))) !=
            cudaSuccess)
        return bad("smem attribute", e);
    if ((e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking)) != cudaSuccess) return bad("stream", e);
    size_t const part = size_t(m->sms) * PARTIAL;
    if ((e = cudaMalloc(&m->d_param, NPARAM * 4)) != cudaSuccess || (e = cudaMalloc(&m->d_m, NPARAM * 4)) != cudaSuccess ||
        (e = cudaMalloc(&m->d_v, NPARAM * 4)) != cudaSuccess ||
        (e = cudaMalloc(&m->d_w1b, 128 * 128 * 2)) != cudaSuccess ||
        (e = cudaMalloc(&m->d_w2b, 128 * 128 * 2)) != cudaSuccess ||
        (e = cudaMalloc(&m->d_partial, part * 4)) != cudaSuccess || (e = cudaMalloc(&m->d_status, 4)) != cudaSuccess ||
        (e = cudaMalloc(&m->d_loss, 8)) != cudaSuccess || (e = cudaMalloc(&m->d_stats, 256 * 4)) != cudaSuccess ||
        (e = cudaMalloc(&m->d_grad, PARTIAL * 4)) != cudaSuccess ||
        (e = cudaHostAlloc(&m->h_status, 16, cudaHostAllocDefault)) != cudaSuccess)
        return bad("alloc", e);
    // He-uniform init for the ReLU layers, small output layer; FP32 master copy
    std::vector<float> w(NPARAM, 0.f);
    auto uni = [&](float a) { return std::uniform_real_distribution<float>(-a, a)(m->rng); };
    for (int o = 0; o < HID; ++o)
        for (int i = 0; i < IN; ++i) w[OFF_W1 + o * IN_K + i] = uni(std::sqrt(6.f / IN));
    for (int k = 0; k < HID * HID; ++k) w[OFF_W2 + k] = uni(std::sqrt(6.f / HID));
    for (int k = 0; k < 2 * HID; ++k) w[OFF_W3 + k] = uni(std::sqrt(1.f / HID));
    if (ta3s_set_params(m, w.data())) {
        delete m;
        return nullptr;
    }
    std::vector<float> stats(256, 0.f);
    for (int c = 0; c < 128; ++c) stats[128 + c] = 1.f;
    // every copy and fill goes on the model's stream: its kernels run on a non-blocking stream, which
    // does not wait for work on the legacy default stream (a pageable cudaMemcpy can even return
    // before its DMA has landed)
    if (cudaMemcpyAsync(m->d_stats, stats.data(), 256 * 4, cudaMemcpyHostToDevice, m->stream) != cudaSuccess ||
        cudaMemsetAsync(m->d_status, 0, 4, m->stream) != cudaSuccess ||
        cudaStreamSynchronize(m->stream) != cudaSuccess) {
        g_err = "ta3s_create: initial copies failed";
        ta3s_destroy(m);
        return nullptr;
    }
    return m;
}

void ta3s_destroy(ta3s_model* m) {
    if (!m) return;
    cudaSetDevice(m->device);
    for (void* p : {(void*)m->d_param, (void*)m->d_m, (void*)m->d_v, (void*)m->d_w1b, (void*)m->d_w2b,
                    (void*)m->d_partial, (void*)m->d_status, (void*)m->d_loss, (void*)m->d_xraw, (void*)m->d_x,
                    (void*)m->d_y, (void*)m->d_idx, (void*)m->d_grad, (void*)m->d_out, (void*)m->d_stats, (void*)m->d_corr})
        if (p) cudaFree(p);
    if (m->h_status) cudaFreeHost(m->h_status);
    if (m->h_out) cudaFreeHost(m->h_out);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
}

const char* ta3s_last_error(const ta3s_model* m) { return m ? m->err.c_str() : g_err.c_str(); }

int ta3s_set_params(ta3s_model* m, const float* params) {
    if (!m || !params) return fail(m, "ta3s_set_params: null argument");
    TA3S_CUDA(m, cudaSetDevice(m->device), "set device");
    // on the model's (non-blocking) stream, ahead of the refresh kernel that reads them
    TA3S_CUDA(m, cudaMemcpyAsync(m->d_param, params, NPARAM * 4, cudaMemcpyHostToDevice, m->stream), "params");
    TA3S_CUDA(m, cudaMemsetAsync(m->d_m, 0, NPARAM * 4, m->stream), "adam m");
    TA3S_CUDA(m, cudaMemsetAsync(m->d_v, 0, NPARAM * 4, m->stream), "adam v");
    m->adam_t = 0;
    refresh_kernel<<<(128 * 128 + 255) / 256, 256, 0, m->stream>>>(m->d_param, m->d_w1b, m->d_w2b);
    TA3S_CUDA(m, cudaGetLastError(), "refresh");
    TA3S_CUDA(m, cudaStreamSynchronize(m->stream), "refresh");
    return 0;
}

int ta3s_get_params(ta3s_model* m, float* params_out) {
    if (!m || !params_out) return fail(m, "ta3s_get_params: null argument");
    TA3S_CUDA(m, cudaSetDevice(m->device), "set device");
    TA3S_CUDA(m, cudaStreamSynchronize(m->stream), "sync");
    TA3S_CUDA(m, cudaMemcpy(params_out, m->d_param, NPARAM * 4, cudaMemcpyDeviceToHost), "params");
    return 0;
}

int ta3s_set_data(ta3s_model* m, const float* x, const float* y, uint32_t n) {
    if (!m || !x || !y || n == 0) return fail(m, "ta3s_set_data: need n > 0 rows");
    TA3S_CUDA(m, cudaSetDevice(m->device), "set device");
    m->rows = 0;      // (until the call is complete)
    // per-column standardisation of the inputs and of the target, FP64 sums
    double s = 0, s2 = 0;
    for (uint32_t r = 0; r < n; ++r) s += y[r];
    double const mu = s / n;
    for (uint32_t r = 0; r < n; ++r) s2 += (y[r] - mu) * (y[r] - mu);
    m->y_mean = float(mu);
    m->y_std = s2 > 0 ? float(std::sqrt(s2 / n)) : 1.f;
    bool const host_stats = ta3_stats::stats_on_host(n, IN);
    std::vector<float> stats(256, 0.f);
    if (host_stats) {
        for (int c = 0; c < 128; ++c) stats[128 + c] = 1.f;
        ta3_stats::host_column_stats(x, n, IN, stats.data(), stats.data() + 128);
        TA3S_CUDA(m, cudaMemcpyAsync(m->d_stats, stats.data(), 256 * 4, cudaMemcpyHostToDevice, m->stream), "stats");
    }
    if (upload_rows(m, x, n, !host_stats)) return 1;
    std::vector<float> ys(n);
    for (uint32_t r = 0; r < n; ++r) ys[r] = (y[r] - m->y_mean) / m->y_std;
    TA3S_CUDA(m, cudaMemcpyAsync(m->d_y, ys.data(), size_t(n) * 4, cudaMemcpyHostToDevice, m->stream), "targets");
    TA3S_CUDA(m, cudaStreamSynchronize(m->stream), "set data");
    m->rows = n;
    return 0;
}

int ta3s_set_data_standardized(ta3s_model* m, const float* x, const float* y, uint32_t n) {
    if (!m || !x || !y || n == 0) return fail(m, "ta3s_set_data_standardized: need n > 0 rows");
    TA3S_CUDA(m, cudaSetDevice(m->device), "set device");
    std::vector<float> stats(256, 0.f);
    for (int c = 0; c < 128; ++c) stats[128 + c] = 1.f;
    m->rows = 0;      // (until the call is complete)
    m->y_mean = 0.f;
    m->y_std = 1.f;
    TA3S_CUDA(m, cudaMemcpyAsync(m->d_stats, stats.data(), 256 * 4, cudaMemcpyHostToDevice, m->stream), "stats");
    if (upload_rows(m, x, n, false)) return 1;
    TA3S_CUDA(m, cudaMemcpyAsync(m->d_y, y, size_t(n) * 4, cudaMemcpyHostToDevice, m->stream), "targets");
    TA3S_CUDA(m, cudaStreamSynchronize(m->stream), "set data");
    m->rows = n;
    return 0;
}

int ta3s_gradients(ta3s_model* m, float* grad_out, float* loss_out) {
    if (!m || !grad_out) return fail(m, "ta3s_gradients: null argument");
    if (m->rows == 0) return fail(m, "ta3s_gradients: no data");
    TA3S_CUDA(m, cudaSetDevice(m->device), "set device");
    if (begin_kernels(m) || launch_mlp(m, int(m->rows), nullptr, 1)) return 1;
    int const grid = std::min(int((m->rows + ROWS - 1) / ROWS), m->sms);
    sum_kernel<<<(PARTIAL + 255) / 256, 256, 0, m->stream>>>(m->d_partial, grid, m->d_grad);
    TA3S_CUDA(m, cudaGetLastError(), "gradient sum");
    if (check_status(m)) return 1;
    TA3S_CUDA(m, cudaMemcpy(grad_out, m->d_grad, NPARAM * 4, cudaMemcpyDeviceToHost), "gradients");
    if (loss_out) TA3S_CUDA(m, cudaMemcpy(loss_out, m->d_grad + NPARAM, 4, cudaMemcpyDeviceToHost), "loss");
    return 0;
}

int ta3s_train(ta3s_model* m, uint32_t epochs, uint32_t batch, float lr, float weight_decay, uint32_t seed,
               float* final_loss) {
    if (!m || batch == 0) return fail(m, "ta3s_train: batch must be positive");
    if (m->rows == 0) return fail(m, "ta3s_train: no data");
    TA3S_CUDA(m, cudaSetDevice(m->device), "set device");
    uint32_t const n = m->rows;
    batch = std::min(batch, n);          // (a minibatch has no more rows than there are, and fits an int)
    uint32_t const steps_per_epoch = (n + batch - 1) / batch;
    size_t const total = size_t(epochs) * steps_per_epoch * batch;
    std::vector<int32_t> idx(total);
    std::mt19937 rng(seed);
    std::vector<int32_t> perm(n);
    for (uint32_t e = 0; e < epochs; ++e) {
        std::iota(perm.begin(), perm.end(), 0);
        std::shuffle(perm.begin(), perm.end(), rng);
        for (uint32_t s = 0; s < steps_per_epoch; ++s)
            for (uint32_t b = 0; b < batch; ++b) {
                uint32_t const k = s * batch + b;
                idx[(size_t(e) * steps_per_epoch + s) * batch + b] = k < n ? perm[k] : -1;
            }
    }
    if (grow(m, m->d_idx, m->cap_idx, std::max<size_t>(total, 1), "alloc indices")) return 1;
    TA3S_CUDA(m, cudaMemcpyAsync(m->d_idx, idx.data(), total * 4, cudaMemcpyHostToDevice, m->stream), "indices");
    AdamConst const ad{lr, 0.9f, 0.999f, 1e-8f, weight_decay};
    uint64_t const steps = uint64_t(epochs) * steps_per_epoch;
    // bias corrections of every step
    std::vector<float> corr(2 * size_t(steps));
    for (uint64_t k = 0; k < steps; ++k) {
        float const t = float(m->adam_t + k + 1);
        corr[k] = 1.f - std::pow(ad.b1, t);
        corr[steps + k] = 1.f - std::pow(ad.b2, t);
    }
    if (begin_kernels(m)) return 1;
    if (batch <= uint32_t(CLUSTER * ROWS)) {
        // minibatches of one cluster: whole runs of steps in one launch, bounded so that a launch stays short
        constexpr uint64_t kStepsPerLaunch = 4096;
        if (steps && grow(m, m->d_corr, m->cap_corr, corr.size(), "alloc bias corrections")) return 1;
        if (steps)
            TA3S_CUDA(m, cudaMemcpyAsync(m->d_corr, corr.data(), corr.size() * 4, cudaMemcpyHostToDevice, m->stream),
                      "bias corrections");
        for (uint64_t k = 0; k < steps; k += kStepsPerLaunch) {
            TrainArgs a{};
            a.p = make_params(m, int(batch), m->d_idx + size_t(k) * batch, 1);
            a.steps = int(std::min(kStepsPerLaunch, steps - k));
            a.first_step = int(k % steps_per_epoch);
            a.steps_per_epoch = int(steps_per_epoch);
            a.rows = int(n);
            a.c1 = m->d_corr + k;
            a.c2 = m->d_corr + steps + k;
            a.param = m->d_param;
            a.m = m->d_m;
            a.v = m->d_v;
            a.w1b = m->d_w1b;
            a.w2b = m->d_w2b;
            a.adam = ad;
            a.loss_out = m->d_loss;
            train_kernel<<<CLUSTER, THREADS, SMEM_BYTES, m->stream>>>(a);
            TA3S_CUDA(m, cudaGetLastError(), "train launch");
            m->adam_t += uint64_t(a.steps);
        }
    } else {
        for (uint64_t k = 0; k < steps; ++k) {
            uint32_t const rows_here = std::min(batch, n - uint32_t(k % steps_per_epoch) * batch);
            if (launch_mlp(m, int(rows_here), m->d_idx + size_t(k) * batch, 1)) return 1;
            int const grid = std::min(int((rows_here + ROWS - 1) / ROWS), m->sms);
            adam_kernel<<<(PARTIAL + 255) / 256, 256, 0, m->stream>>>(m->d_param, m->d_m, m->d_v, m->d_partial, grid, ad,
                                                                      corr[k], corr[steps + k], m->d_w1b, m->d_w2b,
                                                                      m->d_loss);
            TA3S_CUDA(m, cudaGetLastError(), "adam launch");
            ++m->adam_t;
        }
    }
    if (check_status(m)) return 1;
    if (final_loss) {
        float l[2];
        TA3S_CUDA(m, cudaMemcpy(l, m->d_loss, 8, cudaMemcpyDeviceToHost), "loss");
        *final_loss = l[1] > 0 ? l[0] / l[1] : 0.f;
    }
    return 0;
}

int ta3s_predict(ta3s_model* m, const float* x, uint32_t n, float* mean_out, float* logvar_out) {
    if (!m || !x || !mean_out) return fail(m, "ta3s_predict: null argument");
    if (n == 0) return 0;
    TA3S_CUDA(m, cudaSetDevice(m->device), "set device");
    bool const mapped = n <= kMappedRows;
    if (mapped ? grow_out(m, n) : grow(m, m->d_out, m->cap_dout, size_t(n) * 2, "alloc predictions")) return 1;
    if (upload_rows(m, x, n, false) || begin_kernels(m) || launch_mlp(m, int(n), nullptr, 0, mapped ? m->h_out : m->d_out))
        return 1;
    std::vector<float> copied(mapped ? 0 : size_t(n) * 2);
    if (!mapped)
        TA3S_CUDA(m, cudaMemcpyAsync(copied.data(), m->d_out, copied.size() * 4, cudaMemcpyDeviceToHost, m->stream), "outputs");
    if (check_status(m)) return 1;
    float const* const out = mapped ? m->h_out : copied.data();
    for (uint32_t r = 0; r < n; ++r) {
        mean_out[r] = out[2 * r] * m->y_std + m->y_mean;
        if (logvar_out) logvar_out[r] = out[2 * r + 1] + 2.f * std::log(m->y_std);
    }
    return 0;
}

} // extern "C"
