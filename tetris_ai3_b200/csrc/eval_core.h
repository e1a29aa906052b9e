// Candidate evaluation core, shared by the CUDA kernel and a host build used
// only by the CPU tests (tests/test_core_host.py) to pin the incremental path
// against the oracle before it runs on a GPU.
//
// A candidate = (parent board, placement). Two exact paths:
//
// * full path: the reference algorithm as written -- spawn-collision + drop
//   over the columns (ta3_sim/incl/ta3/sim/board2.hpp:306-320), lock
//   (board2.hpp:322-327), line clear (board2.hpp:333-342), the v11 features
//   recomputed over the whole board (ta3_ai/incl/ta3/ai/models/metrics/
//   v_board_metrics.hpp:130-232) and the 10 -> 8 -> 1 MLP
//   (ta3_ai/incl/ta3/ai/models/models/model_v11.hpp:63-91,166-180).
//
// * fast path: the same integers and floats, derived incrementally from a
//   per-parent record built once per kept frontier node. It applies when the
//   drop touches no cell in the piece's own rows of the spawn area (no
//   collision possible) and completes no row (no clear); otherwise the
//   candidate is handed to the full path. With no clear, the clear-count
//   inputs of the MLP are the parent's, so the first four multiply-adds of
//   every hidden unit are folded into the record (P[o]); the remaining
//   operations run in the reference order with separate roundings.
//
// Floating-point rules (both paths, host and device): every multiply and add
// rounds separately (__fmul_rn / __fadd_rn on the device; the host build uses
// -ffp-contract=off); v11's surface input sqrt(s) / 100 comes from a table of
// correctly rounded values, the widened networks compute it (sqrtf correctly
// rounded); divisions by the feature constants 20, 200, 5 and 100 use the FMA-corrected reciprocal quotient (Markstein), which
// tests/test_exact_division.py proves equal to the IEEE quotient over every
// value the features can take.
#pragma once
#include "tables.h"

#include <cstdint>
#if !defined(__CUDA_ARCH__)
#include <cmath>
#endif

#if defined(__CUDACC__)
#define TA3B_HD __host__ __device__ __forceinline__
#else
#define TA3B_HD inline
#endif

namespace ta3b {

// ------------------------------------------------------- exact arithmetic ---
TA3B_HD float f_mul(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
TA3B_HD float f_add(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
TA3B_HD float f_fma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rn(a, b, c);
#else
    return std::fmaf(a, b, c);
#endif
}
TA3B_HD float f_sqrt(float x) {
#if defined(__CUDA_ARCH__)
    return __fsqrt_rn(x);
#else
    return std::sqrt(x);
#endif
}
TA3B_HD int b_ctz_nz(uint32_t v) {           // v != 0
#if defined(__CUDA_ARCH__)
    return __ffs(int(v)) - 1;
#else
    return __builtin_ctz(v);
#endif
}
TA3B_HD int b_popc(uint32_t v) {
#if defined(__CUDA_ARCH__)
    return __popc(v);
#else
    return __builtin_popcount(v);
#endif
}
TA3B_HD int b_msb_nz(uint32_t v) {           // index of the highest set bit, v != 0
#if defined(__CUDA_ARCH__)
    return 31 - __clz(int(v));
#else
    return 31 - __builtin_clz(v);
#endif
}

// x / d rounded to nearest (Markstein: q = x*r, e = fma(-q, d, x), q' = fma(e, r, q)),
// exact for the feature domains (holes <= 230, hole depths <= 2599, wells <= 10,
// sqrt(surface sum) for sums <= 4761).
TA3B_HD float div_exact(float x, float d, float r) {
    float const q = f_mul(x, r);
    float const e = f_fma(-q, d, x);
    return f_fma(e, r, q);
}
constexpr float R20 = 0.05f, R200 = 0.005f, R5 = 0.2f, R100 = 0.01f;

// The surface input sqrt(s) / 100 for every integer surface sum s, both operations rounded to
// nearest: one load instead of a conversion, a square root and a quotient per candidate. The root
// is exact integer arithmetic: m = floor(sqrt(s * 4^k)) with 24 bits, rounded up when the
// remainder exceeds m (a tie is impossible: (m + 1/2)^2 is not an integer).
constexpr int SURF_MAX = 4761;                                   // 9 * 23^2
struct SurfaceTable {
    float in[SURF_MAX + 1];
};
constexpr SurfaceTable make_surface_table() {
    SurfaceTable t{};
    uint64_t m = 1;
    int k = 23;                                                  // s * 4^k in [2^46, 2^48)
    for (int s = 1; s <= SURF_MAX; ++s) {
        while ((uint64_t(s) << (2 * k)) >= (uint64_t(1) << 48)) {
            --k;
            m >>= 1;
        }
        uint64_t const n = uint64_t(s) << (2 * k);
        uint64_t r = m < (uint64_t(1) << 23) ? (uint64_t(1) << 23) : m;
        for (int i = 0; i < 64; ++i) {                           // Newton's iteration, from any start
            uint64_t const q = (r + n / r) / 2;
            if (q == r || q == r + 1 || q + 1 == r) {
                r = q;
                break;
            }
            r = q;
        }
        while (r * r > n) --r;
        while ((r + 1) * (r + 1) <= n) ++r;
        m = r;
        uint64_t const root = n - r * r > r ? r + 1 : r;
        t.in[s] = float(root) / float(uint64_t(1) << k) / 100.0f;
    }
    return t;
}
#if defined(__CUDACC__)
__device__ SurfaceTable const g_surface = make_surface_table();
#endif
inline SurfaceTable const& host_surface() {
    static SurfaceTable const t = make_surface_table();
    return t;
}
TA3B_HD float surface_input(int s) {
#if defined(__CUDA_ARCH__)
    return __ldg(&g_surface.in[s]);
#else
    return host_surface().in[s];
#endif
}

TA3B_HD uint32_t ordered_bits(float v) {                         // beam.hpp:204-207
    uint32_t u;
#if defined(__CUDA_ARCH__)
    u = __float_as_uint(v);
#else
    __builtin_memcpy(&u, &v, 4);
#endif
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

TA3B_HD uint32_t clear_bump(int cleared) {                       // model_defs.hpp:177-183
    return cleared == 0 ? 0u : 1u << (8 * (cleared - 1));
}

TA3B_HD int column_top(uint32_t col) { return b_ctz_nz(col | FLOOR); }

// ------------------------------------------------------------ the weights ---
// Flat v11 layout (model_v11.hpp:166-180, utility.hpp:30-46): W1[o][i] at o*10+i,
// b1[o] at 80+o, W2[0][i] at 88+i, b2 at 96.
constexpr int WB1 = NIN * NHID, WW2 = WB1 + NHID, WB2 = WW2 + NHID;

// ----------------------------------------------------------- full path ---
// v_board_metrics.hpp:130-225 integer metrics of one board
struct BoardInts {
    uint32_t holes, hole_depths, max_height, wells;
    int surf_sq;
};

// The occupied cells' counts of empty cells below them, summed over the board: a column of n cells
// at rows r_i has sum (22 - r_i) cells below them, less the n (n - 1) / 2 occupied ones:
// n (45 - n) / 2 - sum r_i. The row indices are summed over all columns at once, from the number of
// occupied cells per row as bit planes (planes[p] bit y = bit p of row y's count).
TA3B_HD void row_planes(uint32_t const (&b)[W], uint32_t (&p)[4]) {
    // ten one-bit numbers per row: full adders (three of a weight -> sum, carry), then half adders
    auto sum3 = [](uint32_t x, uint32_t y, uint32_t z) { return x ^ y ^ z; };
    auto maj3 = [](uint32_t x, uint32_t y, uint32_t z) { return (x & y) | (z & (x | y)); };
    uint32_t const s1 = sum3(b[0], b[1], b[2]), c1 = maj3(b[0], b[1], b[2]);
    uint32_t const s2 = sum3(b[3], b[4], b[5]), c2 = maj3(b[3], b[4], b[5]);
    uint32_t const s3 = sum3(b[6], b[7], b[8]), c3 = maj3(b[6], b[7], b[8]);
    uint32_t const s4 = sum3(s1, s2, s3), c4 = maj3(s1, s2, s3);
    uint32_t const c5 = s4 & b[9];
    uint32_t const t1 = sum3(c1, c2, c3), d1 = maj3(c1, c2, c3);
    uint32_t const d2 = maj3(t1, c4, c5);
    p[0] = s4 ^ b[9];
    p[1] = sum3(t1, c4, c5);
    p[2] = d1 ^ d2;
    p[3] = d1 & d2;
}

TA3B_HD BoardInts board_ints(uint32_t const (&b)[W]) {
    BoardInts r{0, 0, 0, 0, 0};
    int h[W];
    uint32_t pairs = 0;                                // sum of n (45 - n)
#pragma unroll
    for (int x = 0; x < W; ++x) {
        uint32_t const n = uint32_t(b_popc(b[x]));
        h[x] = H - column_top(b[x]);
        r.holes += uint32_t(h[x]) - n;
        r.max_height = uint32_t(h[x]) > r.max_height ? uint32_t(h[x]) : r.max_height;
        pairs += n * (45u - n);
    }
    uint32_t p[4];
    row_planes(b, p);
    uint32_t rows = 0;                                 // sum of the occupied cells' row indices
#pragma unroll
    for (int q = 3; q >= 0; --q)
        rows = 2 * rows + uint32_t(b_popc(p[q] & 0x2AAAAAu) + 2 * b_popc(p[q] & 0x4CCCCCu) + 4 * b_popc(p[q] & 0x70F0F0u) +
                                   8 * b_popc(p[q] & 0x00FF00u) + 16 * b_popc(p[q] & 0x7F0000u));
    r.hole_depths = pairs / 2 - rows;
#pragma unroll
    for (int x = 1; x < W; ++x) r.surf_sq += (h[x] - h[x - 1]) * (h[x] - h[x - 1]);
    uint32_t wells = uint32_t(h[1] >= h[0] + 3) + uint32_t(h[W - 2] >= h[W - 1] + 3);
#pragma unroll
    for (int x = 1; x < W - 1; ++x) wells += uint32_t((h[x - 1] < h[x + 1] ? h[x - 1] : h[x + 1]) >= h[x] + 3);
    r.wells = wells;
    return r;
}

// search.hpp:61-70: returns legality; nb = resulting board, cleared = rows removed. src: the same
// board as b in memory (the piece's columns are read from it by index)
TA3B_HD bool apply_full(uint32_t const* src, uint32_t const (&b)[W], uint32_t cols, int col0, uint32_t (&nb)[W],
                        int& cleared) {
    uint32_t hit = 0;
    int drop = H;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t const nib = (cols >> (4 * i)) & 0xFu;
        uint32_t const col = src[col0 + i < W ? col0 + i : W - 1];
        hit |= col & nib;
        int const low = b_msb_nz(nib | 1u);
        int const dd = column_top(col & ~((2u << low) - 1u)) - low - 1;
        drop = (nib != 0u && dd < drop) ? dd : drop;
    }
    if (hit) return false;
    uint64_t const piece = uint64_t(cols) << (4 * col0);       // nibble x = board column x
    uint32_t full = FIELD;
#pragma unroll
    for (int x = 0; x < W; ++x) {
        nb[x] = b[x] | ((uint32_t(piece >> (4 * x)) & 0xFu) << drop);
        full &= nb[x];
    }
    cleared = b_popc(full);
    while (full) {                                             // the lowest set bit is the top row: rows above move down
        uint32_t const above = (full & (~full + 1u)) - 1u;
        full &= full - 1u;
#pragma unroll
        for (int x = 0; x < W; ++x) nb[x] = ((nb[x] & above) << 1) | (nb[x] & ~(2u * above + 1u));
    }
    return true;
}
TA3B_HD bool apply_full(uint32_t const (&b)[W], uint32_t cols, int col0, uint32_t (&nb)[W], int& cleared) {
    return apply_full(b, b, cols, col0, nb, cleared);
}

// model_v11.hpp:63-91 inputs + forward, every operation in the reference order
template <class WF>
TA3B_HD float value_full(uint32_t clear_bits, BoardInts const& bi, bool held_i, WF const& w) {
    float in[NIN];
#pragma unroll
    for (int k = 0; k < 4; ++k) in[k] = f_mul(float((clear_bits >> (8 * k)) & 0xFFu), 0.25f);
    in[4] = surface_input(bi.surf_sq);
    in[5] = div_exact(float(bi.holes), 20.0f, R20);
    in[6] = div_exact(float(bi.hole_depths), 200.0f, R200);
    in[7] = float(bi.max_height);
    in[8] = held_i ? 1.0f : 0.0f;
    in[9] = div_exact(float(bi.wells), 5.0f, R5);
    float hid[NHID];
#pragma unroll
    for (int o = 0; o < NHID; ++o) {
        float v = w(WB1 + o);
#pragma unroll
        for (int i = 0; i < NIN; ++i) v = f_add(v, f_mul(in[i], w(o * NIN + i)));
        hid[o] = v > 0.0f ? v : 0.0f;                  // std::max<float>(0, v)
    }
    float v = w(WB2);
#pragma unroll
    for (int i = 0; i < NHID; ++i) v = f_add(v, f_mul(hid[i], w(WW2 + i)));
    return v;
}

// ---------------------------------------------- widened value network ---
// The reference's dense layers (ta3_ai/incl/ta3/ai/models/models/utility.hpp:29-46)
// widened: the v11 inputs -> H ReLU -> H ReLU -> 1 for a compile-time width H, per
// layer [out][in] weights then [out] biases (H = 64: 704 + 4160 + 65 = 4,929 parameters).
template <int H>
struct WideNet {
    static constexpr int B1 = NIN * H, W2 = B1 + H, B2 = W2 + H * H, W3 = B2 + H, B3 = W3 + H, N = B3 + 1;
    // Device copy (STRIDE floats, 16-byte aligned): the same offsets, but layers 1 and 2
    // transposed to [in][out], so one input's weights to all H units are contiguous; the
    // word after the last bias is SKIP (the zero-term flag).
    static constexpr int W1T = 0, W2T = W2, SKIP = N, STRIDE = (N + 1 + 3) / 4 * 4;
    static_assert(H % 4 == 0 && B1 % 4 == 0 && W2 % 4 == 0 && B2 % 4 == 0 && W3 % 4 == 0 && STRIDE > SKIP,
                  "16-byte aligned blocks");
    // device-layout index of parameter j (reference order)
    static TA3B_HD int device_index(int j) {
        if (j < B1) return W1T + (j % NIN) * H + j / NIN;
        if (j >= W2 && j < B2) return W2T + ((j - W2) % H) * H + (j - W2) / H;
        return j;
    }
    static TA3B_HD bool is_bias(int j) { return (j >= B1 && j < W2) || (j >= B2 && j < W3) || j == B3; }
};
// the widths the kernels are built for: 64 (4,929 parameters, the 80k-sim widened generation) and 32 (1,441)
constexpr int WH = 64;
using Wide64 = WideNet<64>;
using Wide32 = WideNet<32>;
constexpr int NPARAMS_WIDE = Wide64::N, NPARAMS_WIDE32 = Wide32::N;
static_assert(NPARAMS_WIDE == 4929 && NPARAMS_WIDE32 == 1441 && Wide64::STRIDE == 4932, "10 -> H -> H -> 1");

TA3B_HD float relu(float v) { return v > 0.0f ? v : 0.0f; }    // std::max<float>(0, v)

// model_v11.hpp:63-91 inputs of the widened network. The surface input is computed: L1, which
// would hold its table, is full of the models' weights
TA3B_HD void wide_inputs(uint32_t clear_bits, BoardInts const& bi, bool held_i, float (&in)[NIN]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) in[k] = f_mul(float((clear_bits >> (8 * k)) & 0xFFu), 0.25f);
    in[4] = div_exact(bi.surf_sq > 0 ? f_sqrt(float(bi.surf_sq)) : 0.0f, 100.0f, R100);
    in[5] = div_exact(float(bi.holes), 20.0f, R20);
    in[6] = div_exact(float(bi.hole_depths), 200.0f, R200);
    in[7] = float(bi.max_height);
    in[8] = held_i ? 1.0f : 0.0f;
    in[9] = div_exact(float(bi.wells), 5.0f, R5);
}

// --------------------------------------------------------- packed FP32x2 ---
// Two independent, separately rounded FP32 operations per instruction on
// sm_100 (__fmul2_rn / __fadd2_rn / __ffma2_rn: per component identical to the
// scalar _rn intrinsics). The host build applies the scalar operation twice.
#if !defined(__CUDACC__)
struct float2 {
    float x, y;
};
inline float2 make_float2(float x, float y) { return float2{x, y}; }
#endif
TA3B_HD float2 f2_mul(float2 a, float2 b) {
#if defined(__CUDA_ARCH__)
    return __fmul2_rn(a, b);
#else
    return make_float2(f_mul(a.x, b.x), f_mul(a.y, b.y));
#endif
}
TA3B_HD float2 f2_add(float2 a, float2 b) {
#if defined(__CUDA_ARCH__)
    return __fadd2_rn(a, b);
#else
    return make_float2(f_add(a.x, b.x), f_add(a.y, b.y));
#endif
}
TA3B_HD float2 f2_fma(float2 a, float2 b, float2 c) {
#if defined(__CUDA_ARCH__)
    return __ffma2_rn(a, b, c);
#else
    return make_float2(f_fma(a.x, b.x, c.x), f_fma(a.y, b.y, c.y));
#endif
}
// The same two operations as inline PTX with the explicit .rn modifier, which
// PTX guarantees is never contracted into a fused multiply-add.
TA3B_HD float2 p2_mul(float2 a, float2 b) {
#if defined(__CUDA_ARCH__)
    unsigned long long ua, ub, ud;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ua) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(ub) : "f"(b.x), "f"(b.y));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(ud) : "l"(ua), "l"(ub));
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(ud));
    return d;
#else
    return make_float2(f_mul(a.x, b.x), f_mul(a.y, b.y));
#endif
}
TA3B_HD float2 p2_add(float2 a, float2 b) {
#if defined(__CUDA_ARCH__)
    unsigned long long ua, ub, ud;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ua) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(ub) : "f"(b.x), "f"(b.y));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(ud) : "l"(ua), "l"(ub));
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(ud));
    return d;
#else
    return make_float2(f_add(a.x, b.x), f_add(a.y, b.y));
#endif
}

// two correctly rounded quotients x / d (div_exact per component; -q * d = q * -d)
TA3B_HD float2 div2_exact(float2 x, float2 d, float2 r) {
    float2 const q = f2_mul(x, r);
    float2 const e = f2_fma(q, make_float2(-d.x, -d.y), x);
    return f2_fma(e, r, q);
}
TA3B_HD int dot4_s8(uint32_t a, uint32_t b, int c) {            // c + sum of 4 signed byte products
#if defined(__CUDA_ARCH__)
    return __dp4a(int(a), int(b), c);
#else
    int s = c;
    for (int i = 0; i < 4; ++i) s += int(int8_t(a >> (8 * i))) * int(int8_t(b >> (8 * i)));
    return s;
#endif
}

// ------------------------------------------------------ parent record ---
// One kept frontier node (or the committed board), in 68 u32 words (a 16-byte
// multiple; 68 = 4 mod 32 staggers the records across shared-memory banks, and
// eight lanes' 16-byte stores cover all 32):
constexpr int REC_WORDS = 68;
constexpr int R_P = 0;        // float[8]: hidden partial sums after the 4 clear inputs
constexpr int R_BOARD = 8;    // 10 bit-columns
constexpr int R_CLEARS = 18;  // path clear histogram (4 x 8-bit lanes)
constexpr int R_TOT = 20;     // holes (8) | max height (5) << 8 | hole depths (12) << 16
constexpr int R_RE = 21;      // 3 words: empty cells per row, 4 bits per row, rows 0..22; then rows 23.. as empty
constexpr int R_SPAN = 26;    // 4 pairs of words: column heights as bytes (byte x = column x), then
                              // (holes - height) per column as signed bytes; bytes 10..15 zero
constexpr int R_COMBO = 34;   // 34 words, per (c0, width) combo: height of column c0-1, 31 at the wall (5)
                              // | left-well precondition << 5 | height of column c0+w, 31 at the wall (5) << 8
                              // | right-well precondition << 13 | wells outside the window's columns (3) << 16
                              // | surface sum without the window's pairs (13) << 19
static_assert(R_COMBO + NCOMBO <= REC_WORDS && REC_WORDS % 4 == 0 && R_SPAN % 2 == 0, "record layout");
constexpr uint32_t WALL = 31; // height outside the board: satisfies every well-edge rule
constexpr uint32_t ROWS_EMPTY = 0xAAAAAAAAu;

TA3B_HD uint32_t fshr32(uint32_t lo, uint32_t hi, uint32_t sh) {     // low word of (hi:lo) >> sh, sh < 32
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, sh);
#else
    return sh ? (lo >> sh) | (hi << (32u - sh)) : lo;
#endif
}
TA3B_HD uint32_t dot4_u8(uint32_t a, uint32_t b, uint32_t c) {       // c + sum of 4 unsigned byte products
#if defined(__CUDA_ARCH__)
    return __dp4a(a, b, c);
#else
    for (int i = 0; i < 4; ++i) c += ((a >> (8 * i)) & 0xFFu) * ((b >> (8 * i)) & 0xFFu);
    return c;
#endif
}

TA3B_HD void store4(uint32_t* dst, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {   // dst 16-byte aligned
#if defined(__CUDA_ARCH__)
    *reinterpret_cast<uint4*>(dst) = make_uint4(a, b, c, d);
#else
    dst[0] = a; dst[1] = b; dst[2] = c; dst[3] = d;
#endif
}

template <class WF>
TA3B_HD uint32_t partial_word(uint32_t clear_bits, int o, WF const& w) {
    // hidden unit o through the 4 clear-count inputs (bias first, inputs ascending)
    float v = w(WB1 + o);
#pragma unroll
    for (int i = 0; i < 4; ++i) v = f_add(v, f_mul(f_mul(float((clear_bits >> (8 * i)) & 0xFFu), 0.25f), w(o * NIN + i)));
    uint32_t u;
#if defined(__CUDA_ARCH__)
    u = __float_as_uint(v);
#else
    __builtin_memcpy(&u, &v, 4);
#endif
    return u;
}

// PARTIALS: the v11 hidden partial sums (the widened network recomputes its own per candidate)
template <class WF, bool PARTIALS = true>
TA3B_HD void build_record(uint32_t const (&b)[W], uint32_t clear_bits, WF const& w, uint32_t* rec) {
    if (PARTIALS) {
        uint32_t p[NHID];
#pragma unroll
        for (int o = 0; o < NHID; ++o) p[o] = partial_word(clear_bits, o, w);
        store4(rec + R_P, p[0], p[1], p[2], p[3]);
        store4(rec + R_P + 4, p[4], p[5], p[6], p[7]);
    }
    store4(rec + R_BOARD, b[0], b[1], b[2], b[3]);
    store4(rec + R_BOARD + 4, b[4], b[5], b[6], b[7]);
    store4(rec + R_BOARD + 8, b[8], b[9], clear_bits, 0u);
    // per column: height, holes; h[x + 2] with walls
    int h[W + 4];
    h[0] = h[1] = h[W + 2] = h[W + 3] = int(WALL);
    uint32_t holes = 0, maxh = 0, pairs = 0, hb[3] = {0, 0, 0}, hmb[3] = {0, 0, 0};
#pragma unroll
    for (int x = 0; x < W; ++x) {
        uint32_t const n = uint32_t(b_popc(b[x]));
        uint32_t const hx = uint32_t(H - column_top(b[x]));
        h[x + 2] = int(hx);
        holes += hx - n;
        maxh = hx > maxh ? hx : maxh;
        pairs += n * (45u - n);
        hb[x >> 2] |= hx << (8 * (x & 3));
        hmb[x >> 2] |= ((0u - n) & 0xFFu) << (8 * (x & 3));          // holes - height = -cells
    }
    // cells per row as nibbles; the row indices of all cells (board_ints)
    uint32_t pl[4], cnt[3], rows = 0;
    row_planes(b, pl);
    auto spread = [](uint32_t v) {              // 8 bits -> bit 4t of a word
        v = (v | (v << 12)) & 0x000F000Fu;
        v = (v | (v << 6)) & 0x03030303u;
        v = (v | (v << 3)) & 0x11111111u;
        return v;
    };
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        cnt[q] = 0;
#pragma unroll
        for (int t = 3; t >= 0; --t) cnt[q] = 2 * cnt[q] + spread((pl[t] >> (8 * q)) & 0xFFu);
        rows = dot4_u8(cnt[q] & 0x0F0F0F0Fu, 0x06040200u + 0x08080808u * uint32_t(q), rows);
        rows = dot4_u8((cnt[q] >> 4) & 0x0F0F0F0Fu, 0x07050301u + 0x08080808u * uint32_t(q), rows);
    }
    store4(rec + R_TOT, holes | (maxh << 8) | ((pairs / 2 - rows) << 16), ROWS_EMPTY - cnt[0], ROWS_EMPTY - cnt[1],
           ROWS_EMPTY - cnt[2]);
    store4(rec + R_TOT + 4, ROWS_EMPTY, 0u, hb[0], hmb[0]);
    store4(rec + R_TOT + 8, hb[1], hmb[1], hb[2], hmb[2]);
    // a combo word is the sum of a word of its window's left edge (c0) and one of its right edge
    // (e = c0 + w): prefix sums up to the edges (pairs (x-1, x) and well flags) on the left, the
    // totals less the prefix sums on the right
    uint32_t pp[W + 1], left[W], right[W + 1];           // prefix: wells << 16 | surface sum << 19
    pp[0] = 0;
#pragma unroll
    for (int x = 0; x < W; ++x) {
        int const l = h[x + 1], m = h[x + 2], r = h[x + 3];
        uint32_t const step = x > 0 ? uint32_t((m - l) * (m - l)) << 19 : 0u;
        pp[x + 1] = pp[x] + step + (uint32_t((l < r ? l : r) >= m + 3) << 16);
    }
    constexpr uint32_t WELLS = 7u << 16, SURF = ~0u << 19;
#pragma unroll
    for (int c = 0; c < W; ++c)                          // wells among columns < c0 - 1, pairs before (c0 - 1, c0)
        left[c] = uint32_t(h[c + 1]) | (uint32_t(c > 0 && h[c] >= h[c + 1] + 3) << 5) |
                  (pp[c > 0 ? c - 1 : 0] & WELLS) | (pp[c > 1 ? c : 1] & SURF);
#pragma unroll
    for (int e = 1; e <= W; ++e)
        right[e] = (uint32_t(h[e + 2]) << 8) | (uint32_t(e < W && h[e + 3] >= h[e + 2] + 3) << 13) |
                   (pp[W] - pp[e + 1 < W ? e + 1 : W]);
    store4(rec + R_TOT + 12, 0u, 0u, left[0] + right[1], left[1] + right[2]);
    static_assert(R_COMBO + 2 == R_TOT + 16 && (NCOMBO - 2) % 4 == 0, "the first two combos share a vector");
#pragma unroll
    for (int id = 2; id < NCOMBO; id += 4) {
        uint32_t v[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            int const wd = id + t < 10 ? 1 : id + t < 19 ? 2 : id + t < 27 ? 3 : 4;
            int const c0 = id + t - (wd == 1 ? 0 : wd == 2 ? 10 : wd == 3 ? 19 : 27);
            v[t] = left[c0] + right[c0 + wd];
        }
        store4(rec + R_COMBO + id, v[0], v[1], v[2], v[3]);
    }
}

// ------------------------------------------------------------ fast path ---
// The weights the fast path needs, as pairs of hidden units (2q, 2q+1):
// W1[o][4..9], W2[o], plus b2; nz = -0 (see MLP_X2FMA), a value the compiler must not know.
struct FastW {
    float2 w4[NHID / 2], w5[NHID / 2], w6[NHID / 2], w7[NHID / 2], w8[NHID / 2], w9[NHID / 2], u[NHID / 2];
    float b2, nz;
};

template <class WF>
TA3B_HD void load_fast_weights(WF const& w, FastW& f, float nz = -0.0f) {
    f.nz = nz;
#pragma unroll
    for (int q = 0; q < NHID / 2; ++q) {
        int const a = 2 * q, b = 2 * q + 1;
        f.w4[q] = make_float2(w(a * NIN + 4), w(b * NIN + 4));
        f.w5[q] = make_float2(w(a * NIN + 5), w(b * NIN + 5));
        f.w6[q] = make_float2(w(a * NIN + 6), w(b * NIN + 6));
        f.w7[q] = make_float2(w(a * NIN + 7), w(b * NIN + 7));
        f.w8[q] = make_float2(w(a * NIN + 8), w(b * NIN + 8));
        f.w9[q] = make_float2(w(a * NIN + 9), w(b * NIN + 9));
        f.u[q] = make_float2(w(WW2 + a), w(WW2 + b));
    }
    f.b2 = w(WB2);
}

enum FastStatus { FAST_OK = 0, FAST_DEFER = 1 };

// The parent record words a fast candidate reads.
struct RecView {
    uint32_t const* rec;
    float P[NHID];
    uint32_t tot, h4, hm4, combo;
};

// the parent's words for one placement (P is the caller's: the widened network has none)
TA3B_HD void load_view(uint32_t const* rec, PlaceFast pf, RecView& r) {
    r.rec = rec;
    r.tot = rec[R_TOT];
    uint32_t const* const s = rec + R_SPAN + (pf.span & 0xFFu);
#if defined(__CUDA_ARCH__)
    uint2 const lo = *reinterpret_cast<uint2 const*>(s), hi = *reinterpret_cast<uint2 const*>(s + 2);
#else
    struct { uint32_t x, y; } const lo{s[0], s[1]}, hi{s[2], s[3]};
#endif
    uint32_t const sh = pf.span >> 8;
    r.h4 = fshr32(lo.x, hi.x, sh);
    r.hm4 = fshr32(lo.y, hi.y, sh);
    r.combo = rec[R_COMBO + pf.combo];
}

// The placement's effect on the parent, from the record alone (branch-free).
// Returns FAST_DEFER when a piece cell may meet the stack inside the spawn rows
// or a row completes; the value is then meaningless.
// MLP arithmetic: MLP_SCALAR = __fmul_rn / __fadd_rn per hidden unit;
// MLP_PTX_X2 = pairs of hidden units per packed PTX instruction (mul/add.rn.f32x2);
// MLP_X2 = the same pairs through the __fmul2_rn / __fadd2_rn intrinsics;
// MLP_X2MUL = packed multiplies (__fmul2_rn), scalar adds;
// MLP_X2FMA = packed multiplies as fused multiply-adds of -0, packed adds.
// Each packed instruction rounds both halves exactly like the scalar .rn operation, but a packed
// multiply feeding a packed add is compiled into a fused multiply-add (one rounding): on the B200 the
// PTX pair equals fma.rn on all of 1,048,576 probe samples. x * w + (-0) is x * w with one rounding,
// signed zeros included, and cannot be fused with the add that follows as long as the compiler does not
// know the -0 (a kernel parameter): MLP_X2FMA keeps the reference's two roundings with 24 packed adds in
// place of 48 scalar ones (0 of 16,777,216 probe samples differ). A packed instruction takes two cycles
// of the FP32 pipe, so it saves issue slots, not arithmetic.
enum MlpMode { MLP_SCALAR = 0, MLP_PTX_X2 = 1, MLP_X2 = 2, MLP_X2MUL = 3, MLP_X2FMA = 4 };

// The fast path's features of one placement (holes, hole depths, surface,
// wells, max height) from the parent record alone; true when the candidate
// must take the full path instead. Bound by issue slots (16 warps per SM, 65 % busy): the record and
// the placement data hold what it needs in the place where one instruction takes it (bytes, whole words,
// top fields, sums formed when the record is built), and the columns are handled four at a time as bytes.
struct FastFeat {
    int holes, hd, surf, wells, maxh, dr;
};

TA3B_HD int min3_s32(int a, int b, int c) {
#if defined(__CUDA_ARCH__)
    return __vimin3_s32(a, b, c);
#else
    int const m = a < b ? a : b;
    return m < c ? m : c;
#endif
}

TA3B_HD bool fast_features(RecView const& r, PlaceFast pf, FastFeat& f) {
    // byte i = 128 + how far piece column i can fall: 22 - lowest row - height (far above for i >= width)
    uint32_t const d = pf.d4 - r.h4;
    int const reach = min3_s32(int(d & 0xFFu), int((d >> 8) & 0xFFu),
                               min3_s32(int((d >> 16) & 0xFFu), int(d >> 24), 255)) - 128;
    bool defer = reach < 0;
    int const dr = reach < 0 ? 0 : reach;
    // rows dr..dr+3: a row whose empty cells are all the piece's is full (rows past the floor: 10 empty cells)
    uint32_t const* const re = r.rec + R_RE + (dr >> 3);
    uint32_t const left = fshr32(re[0], re[1], uint32_t(4 * dr) & 31u) - pf.rows;
    defer = defer || (((left - 0x1111u) & ~left & 0x8888u) != 0u);
    int const w = int(pf.tops >> 24);
    // holes gain the gaps under the piece; every new cell sits over (holes + gap) empty cells
    int const holes = dot4_s8(r.h4, pf.neg, int(r.tot & 0xFFu) + int(pf.adds & 0xFFu)) - w * dr;
    int const hd = dot4_s8(pf.c4, r.hm4, int(r.tot >> 16) + int((pf.adds >> 8) & 0xFFu)) - 4 * dr;
    // new heights of the first and last piece columns and of the piece's top
    uint32_t const tops = pf.tops - uint32_t(dr) * 0x010101u;
    int const n0 = int(tops & 0xFFu), nl = int((tops >> 8) & 0xFFu), top = int((tops >> 16) & 0xFFu);
    int const maxh0 = int((r.tot >> 8) & 0xFFu);
    int const maxh = maxh0 > top ? maxh0 : top;
    uint32_t const cb = r.combo;
    int const hl = int(cb & 31u), hr = int((cb >> 8) & 31u);
    int const tl = n0 - hl, tr = nl - hr;
    // surface: the window's pairs are replaced by the piece's inner steps and the two edge pairs
    int surf = int(cb >> 19) + int((pf.adds >> 16) & 0xFFu);
    surf += hl != int(WALL) ? tl * tl : 0;
    surf += hr != int(WALL) ? tr * tr : 0;
    // wells: only the two neighbour columns (and a one-column piece itself) can be wells now
    int wells = int((cb >> 16) & 7u);
    wells += int((cb & (1u << 5)) && tl >= 3);
    wells += int((cb & (1u << 13)) && tr >= 3);
    wells += int((pf.adds >> 24) && (tl > tr ? tl : tr) <= -3);
    f = FastFeat{holes, hd, surf, wells, maxh, dr};
    return defer;
}

template <int MLP = MLP_SCALAR>
TA3B_HD int fast_eval(RecView const& r, PlaceFast pf, bool held_i, FastW const& fw, float& value,
                      float* dbg = nullptr) {
    FastFeat ff;
    bool const defer = fast_features(r, pf, ff);
    int const holes = ff.holes, hd = ff.hd, surf = ff.surf, wells = ff.wells, maxh = ff.maxh, dr = ff.dr;
    // features (model_v11.hpp:63-91): pairs of correctly rounded quotients
    float const s4 = surface_input(defer ? 0 : surf);            // a deferred candidate's sum may be out of range
    float2 const q56 = div2_exact(make_float2(float(holes), float(hd)), make_float2(20.0f, 200.0f),
                                  make_float2(R20, R200));
    float const q9 = div_exact(float(wells), 5.0f, R5);
    float2 const x4 = make_float2(s4, s4), x5 = make_float2(q56.x, q56.x), x6 = make_float2(q56.y, q56.y);
    float const m7 = float(maxh), m8 = held_i ? 1.0f : 0.0f;
    float2 const x7 = make_float2(m7, m7), x8 = make_float2(m8, m8), x9 = make_float2(q9, q9);
    if (dbg) {                                   // diagnostics for the self-tests
        dbg[0] = float(holes); dbg[1] = float(hd); dbg[2] = float(surf); dbg[3] = float(wells);
        dbg[4] = float(maxh); dbg[5] = x4.x; dbg[6] = x5.x; dbg[7] = x6.x; dbg[8] = x9.x; dbg[9] = float(dr);
    }
    // hidden units in pairs, every multiply and add rounded separately, reference order
    float v = fw.b2;
#pragma unroll
    for (int q = 0; q < NHID / 2; ++q) {
        float2 a = make_float2(r.P[2 * q], r.P[2 * q + 1]);
        if (MLP == MLP_X2MUL) {
            float2 const m4 = f2_mul(x4, fw.w4[q]), m5 = f2_mul(x5, fw.w5[q]), m6 = f2_mul(x6, fw.w6[q]);
            float2 const m7 = f2_mul(x7, fw.w7[q]), m8 = f2_mul(x8, fw.w8[q]), m9 = f2_mul(x9, fw.w9[q]);
            a.x = f_add(a.x, m4.x);
            a.y = f_add(a.y, m4.y);
            a.x = f_add(a.x, m5.x);
            a.y = f_add(a.y, m5.y);
            a.x = f_add(a.x, m6.x);
            a.y = f_add(a.y, m6.y);
            a.x = f_add(a.x, m7.x);
            a.y = f_add(a.y, m7.y);
            a.x = f_add(a.x, m8.x);
            a.y = f_add(a.y, m8.y);
            a.x = f_add(a.x, m9.x);
            a.y = f_add(a.y, m9.y);
        } else if (MLP == MLP_X2FMA) {
            float2 const nz = make_float2(fw.nz, fw.nz);
            a = f2_add(a, f2_fma(x4, fw.w4[q], nz));
            a = f2_add(a, f2_fma(x5, fw.w5[q], nz));
            a = f2_add(a, f2_fma(x6, fw.w6[q], nz));
            a = f2_add(a, f2_fma(x7, fw.w7[q], nz));
            a = f2_add(a, f2_fma(x8, fw.w8[q], nz));
            a = f2_add(a, f2_fma(x9, fw.w9[q], nz));
        } else if (MLP == MLP_X2) {
            a = f2_add(a, f2_mul(x4, fw.w4[q]));
            a = f2_add(a, f2_mul(x5, fw.w5[q]));
            a = f2_add(a, f2_mul(x6, fw.w6[q]));
            a = f2_add(a, f2_mul(x7, fw.w7[q]));
            a = f2_add(a, f2_mul(x8, fw.w8[q]));
            a = f2_add(a, f2_mul(x9, fw.w9[q]));
        } else if (MLP == MLP_PTX_X2) {
            a = p2_add(a, p2_mul(x4, fw.w4[q]));
            a = p2_add(a, p2_mul(x5, fw.w5[q]));
            a = p2_add(a, p2_mul(x6, fw.w6[q]));
            a = p2_add(a, p2_mul(x7, fw.w7[q]));
            a = p2_add(a, p2_mul(x8, fw.w8[q]));
            a = p2_add(a, p2_mul(x9, fw.w9[q]));
        } else {
            a.x = f_add(a.x, f_mul(x4.x, fw.w4[q].x));
            a.y = f_add(a.y, f_mul(x4.y, fw.w4[q].y));
            a.x = f_add(a.x, f_mul(x5.x, fw.w5[q].x));
            a.y = f_add(a.y, f_mul(x5.y, fw.w5[q].y));
            a.x = f_add(a.x, f_mul(x6.x, fw.w6[q].x));
            a.y = f_add(a.y, f_mul(x6.y, fw.w6[q].y));
            a.x = f_add(a.x, f_mul(x7.x, fw.w7[q].x));
            a.y = f_add(a.y, f_mul(x7.y, fw.w7[q].y));
            a.x = f_add(a.x, f_mul(x8.x, fw.w8[q].x));
            a.y = f_add(a.y, f_mul(x8.y, fw.w8[q].y));
            a.x = f_add(a.x, f_mul(x9.x, fw.w9[q].x));
            a.y = f_add(a.y, f_mul(x9.y, fw.w9[q].y));
        }
        if (dbg) {
            dbg[10 + 2 * q] = a.x;
            dbg[11 + 2 * q] = a.y;
        }
        a.x = a.x > 0.0f ? a.x : 0.0f;                      // std::max<float>(0, v)
        a.y = a.y > 0.0f ? a.y : 0.0f;
        float2 const t = MLP == MLP_PTX_X2                  ? p2_mul(a, fw.u[q])
                         : (MLP == MLP_X2 || MLP == MLP_X2MUL || MLP == MLP_X2FMA) ? f2_mul(a, fw.u[q])
                                                               : make_float2(f_mul(a.x, fw.u[q].x),
                                                                             f_mul(a.y, fw.u[q].y));
        v = f_add(v, t.x);
        v = f_add(v, t.y);
    }
    value = v;
    return defer ? FAST_DEFER : FAST_OK;
}

// The fast path's inputs of the widened network: the same features, the parent's
// clear counts as the first four inputs (a fast candidate clears no row). Returns
// true when the candidate must take the full path instead (inputs then all zero).
TA3B_HD bool fast_wide_inputs(RecView const& r, uint32_t clear_bits, PlaceFast pf, bool held_i, float (&in)[NIN]) {
    FastFeat ff;
    bool const defer = fast_features(r, pf, ff);
    BoardInts bi;
    bi.surf_sq = ff.surf;
    bi.holes = ff.holes;
    bi.hole_depths = ff.hd;
    bi.max_height = ff.maxh;
    bi.wells = ff.wells;
    wide_inputs(clear_bits, bi, held_i, in);
    if (defer)
#pragma unroll
        for (int i = 0; i < NIN; ++i) in[i] = 0.0f;
    return defer;
}

} // namespace ta3b
