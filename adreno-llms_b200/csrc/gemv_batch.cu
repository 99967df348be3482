// Batched decode (2 <= M <= 16 activation rows), sm_100a: one launch per operator.
//
// The reference has no batched GEMV (quantised M > 1 is a loop of M = 1 calls, src/models/lfm2-5-350m/src/model.cpp:243-251); the
// arithmetic of a row is that of the single-token call (stream_core.cuh), on the same K parts added in the same order, so row m of
// a batch carries the bits of the single call on row m.
//
// It takes operators whose tiles split K (the layers of a model).  What bounds those: a projection moves 0.3 - 9 MB, a microsecond or two of HBM
// time at most; the rest is the way from the launch before to the first MMA and from the last MMA to the end of the launch, 4000 to 7000 clocks
// in chains of dependent steps, and a second launch for staging the activations was as long again.  Hence:
//   * the rows come into every block as they are, with one copy on a barrier of their own; the weights of the first stages are on
//     their way before (they do not depend on the launch before).  The RMSNorm is applied in place in shared memory, one or two rows
//     per warp (16 rows of 896 values: 2500 clocks), and the accumulator starts of Q4 blocks are summed there;
//   * eight consumer warps, one per K part of a tile: a warp multiplies every second unit of its K chunks;
//   * a stage's weights are one copy too where the rows are whole columns (a copy takes some 50 clocks to issue);
//   * what the waits do not hold up (places of operands, scales, biases) is worked out before them, and no register is spilled;
//   * int8 has eight rows of activations per block at most, and two blocks per tile for 9..16: its exact sums are 24 registers per
//     lane and eight rows (with 16 rows in a block, 48 registers of sums and some spills, the step below took 830 us).
// Steps of 16 rows of a 24-layer, 896-wide model (staging launch + streaming kernel before): int8 771 -> 620 us, fp16 1063 -> 610; 8 rows
// of a 16-layer, 1024-wide Q4 model 397 -> 360; 4 rows of a 30-layer, 576-wide int8 model 540 -> 449.
#include <cuda.h>
#include <cuda_fp16.h>

#include "kernels.h"
#include "plan.h"
#include "ptx.cuh"
#include "stream_core.cuh"

namespace nnb {

namespace {

constexpr int BCW = KPARTS;                  // consumer warps
constexpr int BATCH_THREADS = BCW * 32 + 32; // + the producer warp
constexpr int BATCH_STAGES = 6;              // ring stages at most
constexpr int OFF_BARS = 0;                  // full[], empty[], and one for the activations
constexpr int OFF_SCALE = 512;               // int8: 2^p of the 16 rows, then 2^-p
constexpr int OFF_ROW = 640;                 // int8: a tile's 32 weight-row scales, then what is added or the second weight's scales
constexpr int OFF_X = 1024;                  // (128-byte swizzle: 1 KB boundaries)
static_assert(OFF_BARS + (2 * BATCH_STAGES + 1) * 8 <= OFF_SCALE && OFF_SCALE + 128 <= OFF_ROW && OFF_ROW + 256 <= OFF_X, "header");

// Where the parts of a tile meet: fp32 sums as [part][token][row].  int8: a chunk's pair of warps adds its limb sums first, 24 (times NT)
// integers per lane in the region that then takes the pair's fp32 sums.
constexpr int PAIR_INTS = 3 * 2 * 4 * 32;    // (times NT)
__host__ __device__ constexpr int batch_part_words(int fmt, int nt) { return fmt == FMT_INT8 ? PAIR_INTS / 2 * nt : 8 * nt * RED_TS; }
__host__ __device__ constexpr int batch_red_bytes(int fmt, int nt) { return BCW * batch_part_words(fmt, nt) * 4; }
static_assert(2 * batch_part_words(FMT_INT8, 1) >= 8 * RED_TS, "a pair's sums fit where its integers were");
// (the norm weight lies there first, and is read in whole passes of 32 pieces)
static_assert(batch_red_bytes(FMT_FP16, 1) % 512 == 0 && batch_red_bytes(FMT_INT8, 1) % 512 == 0, "norm weight");

struct BatchSeg {
    const uint16_t* scale;
    const uint16_t* bias;
    uint16_t* out;
    int N, ld, tile0;
};
struct BatchArgs {
    BatchSeg seg[3];
    const uint16_t* scale2;
    const uint16_t* norm_w;
    int* status;
    float norm_eps;
    int M, K, epi, nseg, ntiles, tile_rows;
    int kcb, nchunks, groups, rowbytes;
    int halves;                   // blocks 2 i and 2 i + 1 share the tiles of block i, eight activation rows each
    int cols, wide;               // columns of 128 bytes of a weight's rows in a stage; whether one copy brings them all
    int xcols;                    // columns of 128 bytes of an activation row in shared memory
    int stages, stage_bytes, evict_first;
    int off_ctab, off_red, off_ring;
};
// (the maps' address is taken: they travel in a parameter of their own)
struct BatchMaps { alignas(64) CUtensorMap tm[4], x; };
struct BatchMapsQ4 { alignas(64) CUtensorMap tm[4], x, tm_s[4]; };
template <int FMT> struct BatchMapsFor { typedef BatchMaps type; };
template <> struct BatchMapsFor<FMT_Q4> { typedef BatchMapsQ4 type; };
__device__ __forceinline__ const CUtensorMap* batch_scale_map(const BatchMaps&, int) { return nullptr; }
__device__ __forceinline__ const CUtensorMap* batch_scale_map(const BatchMapsQ4& km, int i) { return &km.tm_s[i]; }

// Activation rows in shared memory: one after another, in columns of 128 bytes whose eight 16-byte pieces are swapped about by the copy
// (128-byte swizzle: piece q of column c of row n sits at q ^ ((n * columns + c) mod 8)).  The columns of a row are counted so that the
// rows of a fragment load lie in different banks: odd for ldmatrix (fp16), 2 or 6 modulo 8 for the 8-byte loads of the int8 path,
// 4 modulo 8 for the 16-byte loads of Q4.
__host__ __device__ inline int batch_xcols(int fmt, int K) {
    const int n = K / 64;
    if (fmt == FMT_FP16) return n | 1;
    if (fmt == FMT_INT8) return (n + 1) / 4 * 4 + 2;
    return (n + 3) / 8 * 8 + 4;
}

// Rows of activations that have room in shared memory: those there are, and one of zeros that stands for all absent ones.
__host__ __device__ inline int batch_xrows(int M, int nt) { return M < 8 * nt ? M + 1 : 8 * nt; }

// Keeps a value's computation where it stands: the compiler would move it past the waits to its first use.
__device__ __forceinline__ void pin(uint32_t& v) { asm volatile("" : "+r"(v)); }
__device__ __forceinline__ void pin(int& v) { asm volatile("" : "+r"(v)); }

__device__ __forceinline__ void batch_sync() { asm volatile("bar.sync 1, %0;" ::"n"(BCW * 32) : "memory"); }

// two fp32 operations at once
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long half2_to_float2(uint32_t h) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    return pack2(f.x, f.y);
}

// RMSNorm of one or two rows in shared memory, in place, by one warp (two at a time: a row alone is a chain of waits).  `row`, `x0`: where
// the rows start and n * columns of them; gamma: the lane's first piece of the norm weight (in shared memory, in order).  The sum of squares is taken in the order of
// rmsnorm_rows, whose four warps a lane stands for one after another: the same bits.
constexpr int NORM_PIECES = NCW;   // 16-byte pieces per lane and pass: rows of up to 1024 values in one
struct NormRow {
    uint32_t at[2];   // the lane's piece of a pass: even and odd ones (a pass is 32 pieces, four columns, which flips bit 2 of the place)
    __device__ __forceinline__ NormRow(uint32_t row, int x0, int lane) {
        const int c = lane >> 3;
        const uint32_t q = (uint32_t)((lane ^ (x0 + c)) & 7);
        at[0] = row + c * 128 + (q << 4);
        at[1] = row + c * 128 + ((q ^ 4u) << 4);
    }
};
__device__ __forceinline__ void lds_v4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void sts_v4(uint32_t addr, const uint32_t (&r)[4]) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
template <int ROWS>
__device__ __forceinline__ void norm_rows(const NormRow (&row)[ROWS], uint32_t gamma, float eps, int K, int lane) {
    const int per_row = K / 8;
    uint32_t xv[ROWS][NORM_PIECES][4];
    unsigned long long ss[ROWS][2];   // of warps 0 and 1, 2 and 3
#pragma unroll
    for (int r = 0; r < ROWS; ++r) ss[r][0] = ss[r][1] = 0ull;
    auto load = [&](int b) {   // b: first piece of a pass
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
            for (int i = 0; i < NORM_PIECES; ++i) {
                if (b + i * 32 + lane < per_row) lds_v4(row[r].at[i & 1] + (uint32_t)(b + i * 32) * 16u, xv[r][i]);
                else xv[r][i][0] = xv[r][i][1] = xv[r][i][2] = xv[r][i][3] = 0u;
            }
    };
    auto squares = [&]() {
#pragma unroll
        for (int i = 0; i < NORM_PIECES; i += 2)
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&xv[r][i][q])), h = __half22float2(*reinterpret_cast<const __half2*>(&xv[r][i + 1][q]));
                    const unsigned long long a = pack2(f.x, h.x), b = pack2(f.y, h.y);
                    ss[r][i >> 1] = fma2(a, a, ss[r][i >> 1]);
                    ss[r][i >> 1] = fma2(b, b, ss[r][i >> 1]);
                }
    };
    load(0);
    squares();
    int last = 0;   // the pass whose pieces are in registers
#pragma unroll 1
    for (int b = NORM_PIECES * 32; b < per_row; b += NORM_PIECES * 32) {
        load(b);
        squares();
        last = b;
    }
    float s4[ROWS][4];
    unsigned long long inv2[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const float2 s01 = unpack2(ss[r][0]), s23 = unpack2(ss[r][1]);
        s4[r][0] = s01.x; s4[r][1] = s01.y; s4[r][2] = s23.x; s4[r][3] = s23.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
            for (int v = 0; v < 4; ++v) s4[r][v] += __shfl_xor_sync(0xffffffffu, s4[r][v], o);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const float inv = 1.0f / sqrtf((((0.f + s4[r][0]) + s4[r][1]) + s4[r][2] + s4[r][3]) / (float)K + eps);
        inv2[r] = pack2(inv, inv);
    }
#pragma unroll 1
    for (int b = 0; b < per_row; b += NORM_PIECES * 32) {
        if (last != 0) load(b);   // (a row of one pass is still there)
#pragma unroll
        for (int i = 0; i < NORM_PIECES; ++i) {
            if (b + i * 32 >= per_row) continue;   // (the warp as one)
            uint32_t g4[4];
            lds_v4(gamma + (uint32_t)(b + i * 32) * 16u, g4);   // (past the row's end: room that is there, and not used)
            unsigned long long gf[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) gf[q] = half2_to_float2(g4[q]);
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 f = unpack2(mul2(mul2(half2_to_float2(xv[r][i][q]), inv2[r]), gf[q]));
                    const __half2 h = __floats2half2_rn(f.x, f.y);
                    xv[r][i][q] = *reinterpret_cast<const uint32_t*>(&h);
                }
                if (b + i * 32 + lane < per_row) sts_v4(row[r].at[i & 1] + (uint32_t)(b + i * 32) * 16u, xv[r][i]);
            }
        }
    }
}

// Q4: the value that the accumulator of a 32-weight block starts from, -72 times the sum of the block's activations, added up in the order
// of stage_x.  `at`: the row's column that holds the block, `h` which half of it, `x`: n * columns + column.
__device__ __forceinline__ float q4_start(const uint8_t* at, int h, int x) {
    uint4 v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = *reinterpret_cast<const uint4*>(at + (((4 * h + t) ^ (x & 7)) << 4));
    float bsum = 0.f;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const uint32_t vv[4] = {v[t].x, v[t].y, v[t].z, v[t].w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&vv[q]));
            bsum += f.x;
            bsum += f.y;
        }
    }
    return -Q4_BIAS * bsum;
}

// The warp's place in a stage and in the activations.  `parity`: of the units it takes (fp16, int8: 64 bytes; Q4: blocks of 16).
template <int NT>
struct BatchGeo {
    uint32_t a0, up;       // its first 16-row block, this lane's row, from the stage's start; from there to the second
    uint32_t a_off;        // fp16, int8: the lane's piece of the first 32 bytes of a unit (of the second: ^ 32)
    uint32_t col_bytes;    // from column to column of a stage
    uint32_t b, b_up;      // the lane's activation row, and how far it is to the one of the second token tile
    uint32_t b_x, b_q;     // n * columns of it; the lane's first piece of a unit
    const uint8_t* start[NT];   // Q4: this lane's accumulator starts, one per block
    int start_step;
    bool two;              // both row blocks
};

// int8: the scales 2^p and 2^-p of one row from its largest magnitude (stream_core.cuh), by one warp; the row is `bytes` long at `row`.
__device__ __forceinline__ void batch_row_scale(uint32_t row, int bytes, float* scale, int m, int lane) {
    uint32_t mx = 0u;
#pragma unroll 4
    for (int o = lane * 16; o < bytes; o += 512) {
        uint32_t v[4];
        lds_v4(row + o, v);
#pragma unroll
        for (int q = 0; q < 4; ++q) mx = half2_magnitude_max(mx, v[q]);
    }
    float up, down;
    int8_row_scale(__reduce_max_sync(0xffffffffu, max(mx & 0xFFFFu, mx >> 16)), up, down);
    if (lane == 0) {
        scale[m] = up;
        scale[16 + m] = down;
    }
}

// One unit (stream_core.cuh: step_fp16, block_q4; the same products in the same order): i counts the warp's units of the chunk,
// s the row's units.  Loads and arithmetic are apart so that two units' loads can be on their way together.
template <int NT>
struct BatchFrag {
    uint32_t w[2][2][4], b[2][NT][2];   // [32-byte half][row block]; [k16 step]
};
template <int NT>
__device__ __forceinline__ void batch_load(const BatchGeo<NT>& L, uint32_t sw, int i, int s, BatchFrag<NT>& f) {
    const uint32_t col = sw + (uint32_t)i * L.col_bytes;
#pragma unroll
    for (int h = 0; h < 2; ++h) ldsm_x4(col + L.a0 + (L.a_off ^ (32u * h)), f.w[h][0][0], f.w[h][0][1], f.w[h][0][2], f.w[h][0][3]);
    if (L.two) {
#pragma unroll
        for (int h = 0; h < 2; ++h) ldsm_x4(col + L.a0 + L.up + (L.a_off ^ (32u * h)), f.w[h][1][0], f.w[h][1][1], f.w[h][1][2], f.w[h][1][3]);
    }
    const uint32_t off = (uint32_t)(s >> 1) * 128u + ((L.b_q ^ ((L.b_x + (uint32_t)(s >> 1)) & 7u)) << 4);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) ldsm_x4(L.b + nt * L.b_up + off, f.b[0][nt][0], f.b[0][nt][1], f.b[1][nt][0], f.b[1][nt][1]);
}
template <int NT>
__device__ __forceinline__ void batch_mac(const BatchFrag<NT>& f, bool two, float (&ac)[2][NT][4]) {
#pragma unroll
    for (int rb = 0; rb < 2; ++rb) {
        if (rb == 1 && !two) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_16816(ac[rb][nt], f.w[h][rb][0], f.w[h][rb][1], f.w[h][rb][2], f.w[h][rb][3], f.b[h][nt][0], f.b[h][nt][1]);
    }
}
// int8: one unit of 64 values.  The codes go into the integer MMAs as they are; the limbs of the activations (stream_core.cuh: int8_limbs) are
// made here from the fp16 rows: each value belongs to one warp of the tile, and the limb planes of 16 rows would take half as much
// shared memory again as the rows.  Four neighbouring values are the four bytes of a lane's B register, so there is nothing to exchange.
template <int NT>
__device__ __forceinline__ void batch_unit_int8(const BatchGeo<NT>& L, uint32_t sw, int i, int s, const float (&up)[NT], int (&ac)[3][2][NT][4]) {
    const uint32_t col = sw + (uint32_t)i * L.col_bytes, x = (L.b_x + (uint32_t)s) & 7u, at = (uint32_t)s * 128u + (L.b_q & 1u) * 8u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t w[2][4], v[NT][2][2];
        ldsm_x4(col + L.a0 + (L.a_off ^ (32u * h)), w[0][0], w[0][1], w[0][2], w[0][3]);
        if (L.two) ldsm_x4(col + L.a0 + L.up + (L.a_off ^ (32u * h)), w[1][0], w[1][1], w[1][2], w[1][3]);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 2; ++j) lds_v2(L.b + nt * L.b_up + at + (((2u * (2 * h + j) + (L.b_q >> 1)) ^ x) << 4), v[nt][j][0], v[nt][j][1]);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            uint32_t b[2][3];
#pragma unroll
            for (int j = 0; j < 2; ++j) int8_limbs(v[nt][j][0], v[nt][j][1], up[nt], b[j]);
#pragma unroll
            for (int rb = 0; rb < 2; ++rb) {
                if (rb == 1 && !L.two) continue;
                imma_16832<true>(ac[0][rb][nt], w[rb][0], w[rb][1], w[rb][2], w[rb][3], b[0][0], b[1][0]);
                imma_16832<false>(ac[1][rb][nt], w[rb][0], w[rb][1], w[rb][2], w[rb][3], b[0][1], b[1][1]);
                imma_16832<false>(ac[2][rb][nt], w[rb][0], w[rb][1], w[rb][2], w[rb][3], b[0][2], b[1][2]);
            }
        }
    }
}
// Q4: one 16-byte block, number u of the chunk and s of the row; sc[rb]: the chunk's scales of the lane's row g of a row block, `sstr`
// bytes from row to row.  The activations of a block are 16 bytes per lane, paired here as a word's codes come out (k 8t + j, k 8t + j + 4).
template <int NT>
__device__ __forceinline__ void batch_block_q4(const BatchGeo<NT>& L, uint32_t sw, int u, int s, float (&ac)[2][NT][4], const uint8_t* const (&sc)[2], int sstr, uint32_t lane7) {
    uint32_t w[4], b[NT][4];
    float4 cq[NT];
    ldsm_x4(sw + (uint32_t)(u >> 3) * L.col_bytes + L.a0 + ((((uint32_t)u & 7u) ^ lane7) << 4), w[0], w[1], w[2], w[3]);
    const uint32_t off = (uint32_t)(s >> 1) * 128u + ((L.b_q ^ ((L.b_x + (uint32_t)(s >> 1)) & 7u)) << 4);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        uint32_t v[4];
        lds_v4(L.b + nt * L.b_up + off, v);
        b[nt][0] = __byte_perm(v[0], v[2], 0x5410);
        b[nt][1] = __byte_perm(v[0], v[2], 0x7632);
        b[nt][2] = __byte_perm(v[1], v[3], 0x5410);
        b[nt][3] = __byte_perm(v[1], v[3], 0x7632);
        cq[nt] = *reinterpret_cast<const float4*>(L.start[nt] + (size_t)s * L.start_step);
    }
#pragma unroll
    for (int rb = 0; rb < 2; ++rb) {
        if (rb == 1 && !L.two) continue;
        const float s_lo = __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t*>(sc[rb] + u * 2)));
        const float s_hi = __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t*>(sc[rb] + 8 * sstr + u * 2)));
        uint32_t p04, p15, p26, p37, q04, q15, q26, q37;
        q4x8_to_half2x4_biased(w[rb * 2], p04, p15, p26, p37);
        q4x8_to_half2x4_biased(w[rb * 2 + 1], q04, q15, q26, q37);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            float d[4];
            mma_16816_c(d, p04, q04, p15, q15, b[nt][0], b[nt][1], cq[nt]);
            mma_16816(d, p26, q26, p37, q37, b[nt][2], b[nt][3]);
            ac[rb][nt][0] = fmaf(d[0], s_lo, ac[rb][nt][0]);
            ac[rb][nt][1] = fmaf(d[1], s_lo, ac[rb][nt][1]);
            ac[rb][nt][2] = fmaf(d[2], s_hi, ac[rb][nt][2]);
            ac[rb][nt][3] = fmaf(d[3], s_hi, ac[rb][nt][3]);
        }
    }
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void* tmap, int x, int y, int z, uint32_t bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(dst),
        "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar), "l"(policy)
        : "memory");
}

template <int FMT, int NT>
__global__ void __launch_bounds__(BATCH_THREADS, 2) linear_batch_kernel(const __grid_constant__ typename BatchMapsFor<FMT>::type km, const BatchArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Token halves (int8, 9..16 rows): the second block of a pair takes the last eight rows, and stores those from the ninth on.
    const bool halves = FMT == FMT_INT8 && a.halves;
    const int bx = halves ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, gx = halves ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int m_off = halves && (blockIdx.x & 1u) ? a.M - 8 : 0, m_lo = m_off ? 8 - m_off : 0;   // first row here; first one that is stored
    const int M = halves ? 8 : a.M, K = a.K, stages = a.stages, ntiles = a.ntiles, groups = a.groups, kcb = a.kcb, rowbytes = a.rowbytes, nchunks = a.nchunks;
    const bool dual = a.epi == EPI_SWIGLU;
    const int tile_rows = a.tile_rows;
    const uint32_t base = (smem_u32(smem) + 1023u) & ~1023u;
    uint8_t* const sm = smem + (base - smem_u32(smem));
    const uint32_t full0 = base + OFF_BARS, empty0 = full0 + BATCH_STAGES * 8, xbar = empty0 + BATCH_STAGES * 8;
    const uint32_t ring = base + (uint32_t)a.off_ring, col_bytes = (uint32_t)tile_rows * 128u;
    const int xpitch = a.xcols * 128;
    if (tid < BATCH_STAGES) mbar_init(full0 + tid * 8, 1u);
    else if (tid < 2 * BATCH_STAGES) mbar_init(full0 + tid * 8, (uint32_t)BCW);
    else if (tid == 2 * BATCH_STAGES) mbar_init(xbar, 1u);
    if (FMT == FMT_INT8 && tid < 32) reinterpret_cast<float*>(sm + OFF_SCALE)[tid] = 1.f;   // (absent rows)
    mbar_init_fence();
    // Absent rows are zeros, but not by the copy: 128 bytes past the end take it five times as long as those that are there (a
    // step of 2 rows, 16-layer, 1024-wide Q4 model: 440 us with boxes of 8 rows, 316 so).
    for (uint32_t i = (uint32_t)(M * xpitch + tid * 16); i < (uint32_t)(batch_xrows(M, NT) * xpitch); i += BATCH_THREADS * 16) *reinterpret_cast<uint4*>(sm + OFF_X + i) = make_uint4(0, 0, 0, 0);
    __syncthreads();

    auto segment = [&](int tile) { return (a.nseg > 2 && tile >= a.seg[2].tile0) ? 2 : (a.nseg > 1 && tile >= a.seg[1].tile0) ? 1 : 0; };
    // (constant indexes into the parameter block: a run-time one would read it through generic loads)
    auto seg_at = [&](int si) { return si == 0 ? a.seg[0] : si == 1 ? a.seg[1] : a.seg[2]; };

    if (warp == BCW) {
        // ---- producer: the weights of the ring's first pass, the activations once the launch before is over, the rest ----
        pdl_launch_dependents();
        const uint64_t policy = a.evict_first ? l2_policy_evict_first() : l2_policy_evict_normal();
        const int per_block = (bx < ntiles ? (ntiles - bx + gx - 1) / gx : 0) * groups;
        const int ahead = min(stages, per_block), cols = a.cols;
        const int sw_bytes = (dual ? 2 : 1) * cols * (int)col_bytes, sc_row = cols * 16;   // sc_row: bytes of Q4 block scales per row of a stage
        int tile = bx, cg = 0, stage = 0;
        uint32_t phase = 1u;
#pragma unroll 1
        for (int it = 0; it <= per_block; ++it) {
            if (it == ahead) {
                pdl_wait_prior_grid();
                if (lane == 0) {
                    // One copy for all rows.  A copy takes some 50 clocks to issue, whatever its size: 16 rows of
                    // 896 values are there after 1330 clocks, as pieces of 1 KB after 2900 (155 KB: 2600 and 10000).
                    mbar_arrive_expect_tx(xbar, (uint32_t)(M * xpitch + (a.norm_w ? K * 2 : 0)));
                    tma_load_3d(base + OFF_X, &km.x, 0, 0, m_off, xbar, l2_policy_evict_normal());
                    if (a.norm_w) bulk_g2s(base + a.off_red, a.norm_w, (uint32_t)K * 2u, xbar, l2_policy_evict_normal());   // (the sums come later)
                }
            }
            if (it == per_block) break;
            if (it >= stages && !__all_sync(0xffffffffu, mbar_wait_bounded(empty0 + stage * 8, phase))) {
                *reinterpret_cast<volatile int*>(a.status) = 2;
                break;
            }
            if (lane == 0) {
                const uint32_t dst = ring + stage * a.stage_bytes, bar = full0 + stage * 8;
                const int si = dual ? 0 : segment(tile), row0 = (tile - seg_at(si).tile0) * tile_rows, c0 = cg * cols;
                const CUtensorMap* const m0 = &km.tm[si];
                // columns past the end of the rows come as zeros, or (one copy each) not at all
                const int n = a.wide ? cols : min(cols, (rowbytes + 127) / 128 - c0);
                mbar_arrive_expect_tx(bar, (uint32_t)((dual ? 2 : 1) * (n * (int)col_bytes + (FMT == FMT_Q4 ? tile_rows * sc_row : 0))));
                if (FMT == FMT_Q4) {
                    tma_load_2d(dst + sw_bytes, batch_scale_map(km, si), cg * sc_row, row0, bar, policy);
                    if (dual) tma_load_2d(dst + sw_bytes + tile_rows * sc_row, batch_scale_map(km, 3), cg * sc_row, row0, bar, policy);
                }
                if (a.wide) {
                    tma_load_3d(dst, m0, 0, row0, c0, bar, policy);
                    if (dual) tma_load_3d(dst + cols * col_bytes, &km.tm[3], 0, row0, c0, bar, policy);
                } else {
#pragma unroll 1
                    for (int i = 0; i < n; ++i) {
                        tma_load_2d(dst + i * col_bytes, m0, (c0 + i) * 128, row0, bar, policy);
                        if (dual) tma_load_2d(dst + (cols + i) * col_bytes, &km.tm[3], (c0 + i) * 128, row0, bar, policy);
                    }
                }
            }
            __syncwarp();
            if (++cg == groups) { cg = 0; tile += gx; }
            if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        return;
    }

    // ---- consumers: warp 2 j + set takes the units of parity `set` of the tile's K chunks j, j + 4, .. ----
    constexpr bool IMMA = FMT == FMT_INT8;
    constexpr int PART = batch_part_words(FMT, NT);   // one warp's sums, as [token][row]
    const int box = warp >> 1, set = warp & 1, g = lane >> 2, t = lane & 3;
    // the finish: a pair of neighbouring rows of one token per thread
    const int plog = 30 - __clz(tile_rows), pair = tid & ((1 << plog) - 1), m = tid >> plog;
    static_assert((BCW * 32) / (WARP_ROWS / 2) >= 16, "one pass over the rows of activations");
    const int prow = 2 * pair;   // in the tile
    const bool inplace = a.epi == EPI_RESIDUAL || a.epi == EPI_SILU_GATE;
    // what a tile's finish needs besides the sums: fetched ahead (raw bits: the loads are waited for where they are used)
    uint16_t p_sc = 0, p_add[2] = {0, 0}, p_old[2] = {0, 0};
    auto fetch_rows = [&](int tile) {
        const BatchSeg sg = seg_at(dual ? 0 : segment(tile));
        if (IMMA) {   // (one warp, a row per lane: the int8 sums leave few registers)
            const int n = min((tile - sg.tile0) * tile_rows + lane, sg.N - 1);
            if (warp == 1) {
                p_sc = sg.scale[n];
                if (dual) p_add[0] = a.scale2[n];
                else if (sg.bias) p_add[0] = sg.bias[n];
            }
            return;
        }
        const int n0 = (tile - sg.tile0) * tile_rows + prow;
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (sg.bias) p_add[i] = sg.bias[min(n0 + i, sg.N - 1)];
    };
    auto fetch_old = [&](int tile) {
        const BatchSeg sg = seg_at(segment(tile));
        const int n0 = (tile - sg.tile0) * tile_rows + prow;
#pragma unroll
        for (int i = 0; i < 2; ++i) p_old[i] = (n0 + i < sg.N && m < M && m >= m_lo) ? sg.out[(size_t)(m_off + m) * sg.ld + n0 + i] : (uint16_t)0;
    };
    int tile = bx;
    if (tile < ntiles) fetch_rows(tile);
    BatchGeo<NT> lg;
    {
        const int grp = box * (kcb / 128) * (int)col_bytes;
        lg.two = dual || tile_rows == WARP_ROWS;
        lg.col_bytes = col_bytes;
        const uint32_t up = dual ? (uint32_t)a.cols * col_bytes : 16u * 128u;   // from the first row block to the second
        // fp16, int8: ldmatrix over rows 0-7 and 8-15, a piece and the next; Q4: over both row blocks' rows, one piece
        lg.a0 = (uint32_t)(grp + (lane & 15) * 128) + (FMT == FMT_Q4 && (lane >> 4) && lg.two ? up : 0u);
        lg.up = up;
        lg.a_off = (uint32_t)(((4 * set + (lane >> 4)) ^ (lane & 7)) << 4);
        const int n = FMT == FMT_FP16 ? lane & 7 : g;
        lg.b_x = (uint32_t)(n * a.xcols) & 7u;
        lg.b_q = (uint32_t)(IMMA ? t : 4 * set + (FMT == FMT_FP16 ? lane >> 3 : t));
        lg.b = base + OFF_X + (uint32_t)(min(n, M) * xpitch);
        lg.b_up = (uint32_t)((min(n + 8, M) - min(n, M)) * xpitch);   // (eight rows of columns are whole turns of the swizzle)
        const int pairs = (M + 1) / 2;
        lg.start_step = pairs * 16;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) lg.start[nt] = sm + a.off_ctab + min(t + 4 * nt, pairs - 1) * 16;
    }
    uint32_t mine_off = (uint32_t)(a.off_red + (warp * PART + 2 * t * RED_TS + g) * 4), src_off = (uint32_t)(a.off_red + prow * 4);
    pin(lg.a0); pin(lg.a_off); pin(lg.b); pin(lg.b_x); pin(lg.b_q);
    pin(mine_off); pin(src_off);
    pdl_launch_dependents();
    pdl_wait_prior_grid();
    if (inplace && tile < ntiles) fetch_old(tile);
    bool failed = false;
    if (!mbar_wait_bounded(xbar, 0u)) {
        failed = true;
        *reinterpret_cast<volatile int*>(a.status) = 5;
    }
    if (a.norm_w) {
        if (warp + BCW < M) {
            const NormRow rows[2] = {NormRow(base + OFF_X + warp * xpitch, warp * a.xcols, lane), NormRow(base + OFF_X + (warp + BCW) * xpitch, (warp + BCW) * a.xcols, lane)};
            norm_rows<2>(rows, base + a.off_red + lane * 16, a.norm_eps, K, lane);
        } else if (warp < M) {
            const NormRow rows[1] = {NormRow(base + OFF_X + warp * xpitch, warp * a.xcols, lane)};
            norm_rows<1>(rows, base + a.off_red + lane * 16, a.norm_eps, K, lane);
        }
        if (IMMA) __syncwarp();   // (a warp's rows are its own until their scales are there)
        else batch_sync();
    }
    float *const scale = reinterpret_cast<float*>(sm + OFF_SCALE), *const rows = reinterpret_cast<float*>(sm + OFF_ROW);
    float up[NT];
    if (IMMA) {
        for (int m = warp; m < M; m += BCW) batch_row_scale(base + OFF_X + m * xpitch, K * 2, scale, m, lane);
        batch_sync();
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) up[nt] = scale[g + 8 * nt];
    }
    if (FMT == FMT_Q4) {
        const int pairs = (M + 1) / 2, blocks = K / 32;
#pragma unroll 1
        for (int i = tid; i < 2 * pairs * blocks; i += BCW * 32) {
            const int m = i / blocks, b = i - m * blocks;
            const float v = m < M ? q4_start(sm + OFF_X + m * xpitch + (b >> 1) * 128, b & 1, m * a.xcols + (b >> 1)) : 0.f;
            float* const cq = reinterpret_cast<float*>(sm + a.off_ctab) + ((size_t)b * pairs + (m >> 1)) * 4 + (m & 1);
            cq[0] = v;
            cq[2] = v;
        }
        batch_sync();
    }
    int stage = 0;
    uint32_t phase = 0u;
#pragma unroll 1
    for (; tile < ntiles; tile += gx) {
        float acc[2][NT][4];
        int iacc[IMMA ? 3 : 1][2][NT][4];
#pragma unroll
        for (int rb = 0; rb < 2; ++rb)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    acc[rb][nt][i] = 0.f;
#pragma unroll
                    for (int l = 0; l < (IMMA ? 3 : 1); ++l) iacc[l][rb][nt][i] = 0;
                }
#pragma unroll 1
        for (int cg = 0; cg < groups; ++cg) {
            const int c = cg * NCW + box;
            // A wait that runs out records an error and skips the arithmetic from then on; the warp still walks its items so that
            // the block's barriers stay matched, and still waits (not as long) for each copy, so that none is in flight when the block ends.
            if (!mbar_wait_bounded(full0 + stage * 8, phase, failed ? WAIT_CYCLES / 64 : WAIT_CYCLES)) {
                failed = true;
                *reinterpret_cast<volatile int*>(a.status) = 1;
            }
            failed = __any_sync(0xffffffffu, failed) != 0;   // (the warp agrees before its matrix instructions)
            const uint32_t sw = ring + stage * a.stage_bytes;
            const int cb = (failed || c >= nchunks) ? 0 : min(kcb, rowbytes - c * kcb);
            if constexpr (FMT == FMT_Q4) {
                const int sstr = a.cols * 16, s0 = c * kcb / 16;
                const uint8_t* const scb = sm + (sw - base) + (dual ? 2 : 1) * a.cols * (int)col_bytes + box * (kcb / 8);
                const uint8_t* const sc[2] = {scb + g * sstr, scb + (g + (dual ? tile_rows : 16)) * sstr};
#pragma unroll 1
                for (int u = set; u < cb / 16; u += 2) batch_block_q4<NT>(lg, sw, u, s0 + u, acc, sc, sstr, (uint32_t)lane & 7u);
            } else if constexpr (IMMA) {
                const int s0 = c * kcb / 64;
#pragma unroll 1
                for (int u = set; u < cb / 64; u += 2) batch_unit_int8<NT>(lg, sw, u >> 1, s0 + u, up, iacc);
            } else {
                const int s0 = c * kcb / 64;
                const int n = (cb / 64 - set + 1) >> 1;   // the warp's units
                constexpr bool PAIR = NT == 1;   // two units' operands fit in registers
#pragma unroll 1
                for (int i = 0; i < n; i += PAIR ? 2 : 1) {
                    BatchFrag<NT> f0, f1;
                    batch_load<NT>(lg, sw, i, s0 + 2 * i + set, f0);
                    if (PAIR && i + 1 < n) batch_load<NT>(lg, sw, i + 1, s0 + 2 * i + 2 + set, f1);
                    batch_mac<NT>(f0, lg.two, acc);
                    if (PAIR && i + 1 < n) batch_mac<NT>(f1, lg.two, acc);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + stage * 8);
            if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        // the parts meet in shared memory as [part][token][row]
        batch_sync();   // (the finish before this one has read them)
        float* const mine = reinterpret_cast<float*>(sm + mine_off);
        if (IMMA) {
            // a chunk's two sets as integers (exact, so their order does not matter), then one fp32 sum per chunk, as int8_recombine has it
            int* const pair = reinterpret_cast<int*>(sm + a.off_red) + box * 2 * PART + lane;
            if (warp == 1) {
                rows[lane] = __half2float(__ushort_as_half(p_sc));
                rows[32 + lane] = __half2float(__ushort_as_half(p_add[0]));
            }
            if (set == 1) {
#pragma unroll
                for (int l = 0; l < 3; ++l)
#pragma unroll
                    for (int i = 0; i < 8 * NT; ++i) pair[(l * 8 * NT + i) * 32] = iacc[l % (IMMA ? 3 : 1)][i / (4 * NT)][(i >> 2) % NT][i & 3];
            }
            asm volatile("bar.sync %0, 64;" ::"r"(2 + box) : "memory");
            if (set == 0) {
                const float* const down = scale + 16 + 2 * t;
#pragma unroll
                for (int i = 0; i < 8 * NT; ++i) {
                    auto limb = [&](int l) { return (float)(iacc[l % (IMMA ? 3 : 1)][i / (4 * NT)][(i >> 2) % NT][i & 3] + pair[(l * 8 * NT + i) * 32]); };
                    acc[i / (4 * NT)][(i >> 2) % NT][i & 3] = fmaf(limb(0), 65536.f, fmaf(limb(1), 256.f, limb(2))) * down[(i >> 2) % NT * 8 + (i & 1)];
                }
                __syncwarp();
            }
        }
        if (!IMMA || set == 0) {
#pragma unroll
            for (int rb = 0; rb < 2; ++rb)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int i = 0; i < 4; ++i) mine[(nt * 8 + (i & 1)) * RED_TS + rb * 16 + (i >> 1) * 8] = acc[rb][nt][i];
        }
        batch_sync();
        const BatchSeg sg = seg_at(dual ? 0 : segment(tile));
        const int n = (tile - sg.tile0) * tile_rows + prow;
        const bool two = n + 1 < sg.N, biased = sg.bias != nullptr;
        const float* const src = reinterpret_cast<const float*>(sm + src_off);
        if (n < sg.N && m < M && m >= m_lo) {
            auto sum = [&](int up) {   // a chunk's two sets first, then the chunks in order
                const float* const s = src + m * RED_TS + up;
                auto both = [&](int j) {
                    if (IMMA) return *reinterpret_cast<const float2*>(s + 2 * j * PART);
                    const float2 v = *reinterpret_cast<const float2*>(s + 2 * j * PART), o = *reinterpret_cast<const float2*>(s + (2 * j + 1) * PART);
                    return make_float2(v.x + o.x, v.y + o.y);
                };
                float2 v = both(0);
#pragma unroll
                for (int j = 1; j < NCW; ++j) {
                    const float2 o = both(j);
                    v.x += o.x;
                    v.y += o.y;
                }
                return v;
            };
            const float2 s0 = sum(0);
            const float2 s1 = dual ? sum(16) : make_float2(0.f, 0.f);
            uint16_t* const dst = sg.out + (size_t)(m_off + m) * sg.ld + n;
            const float2 sc = IMMA ? *reinterpret_cast<const float2*>(rows + prow) : make_float2(0.f, 0.f);
            const float2 add = IMMA ? *reinterpret_cast<const float2*>(rows + 32 + prow) : make_float2(__half2float(__ushort_as_half(p_add[0])), __half2float(__ushort_as_half(p_add[1])));
            uint16_t hv[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {   // roundings as in finish_row and finish_swiglu
                float v = i ? s0.y : s0.x;
                if (IMMA) v = __fmul_rn(v, i ? sc.y : sc.x);
                const float gt = dual ? v : __half2float(__ushort_as_half(p_old[i]));
                if (dual) {
                    float uv = i ? s1.y : s1.x;
                    if (IMMA) uv *= i ? add.y : add.x;
                    v = (gt / (1.0f + expf(-gt))) * uv;
                } else {
                    if (biased) v = __fadd_rn(__half2float(__float2half_rn(v)), i ? add.y : add.x);
                    if (a.epi == EPI_RESIDUAL) v = __fadd_rn(gt, v);
                    else if (a.epi == EPI_SILU_GATE) v = gt * (1.0f / (1.0f + expf(-gt))) * v;
                }
                hv[i] = __half_as_ushort(__float2half_rn(v));
            }
            if (two && (reinterpret_cast<uintptr_t>(dst) & 3) == 0) {
                *reinterpret_cast<uint32_t*>(dst) = (uint32_t)hv[0] | (uint32_t)hv[1] << 16;
            } else {
                dst[0] = hv[0];
                if (two) dst[1] = hv[1];
            }
        }
        const int next = tile + gx;
        if (next < ntiles) {
            fetch_rows(next);
            if (inplace) fetch_old(next);
        }
    }
}

template <int FMT, int NT>
cudaError_t launch_n(const typename BatchMapsFor<FMT>::type& km, const BatchArgs& a, const BatchPlan& p, cudaStream_t st, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.grid);
    cfg.blockDim = dim3((unsigned)BATCH_THREADS);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, linear_batch_kernel<FMT, NT>, km, a);
}

inline bool fill_scale_maps(BatchMaps&, const LinArgs&, int, int) { return true; }
inline bool fill_scale_maps(BatchMapsQ4& km, const LinArgs& a, int bw, int tile_rows) {
    const uint16_t* base[4];
    int pitch = 0;
    if (!q4_scale_views(a, base, &pitch)) return false;
    for (int i = 0; i < a.nseg; ++i)
        if (!make_scale_map(&km.tm_s[i], base[i], a.seg[i].N, pitch, bw, tile_rows)) return false;
    return a.epi != EPI_SWIGLU || make_scale_map(&km.tm_s[3], base[3], a.seg[0].N, pitch, bw, tile_rows);
}

template <int FMT>
cudaError_t launch_f(const LinArgs& a, const BatchPlan& p, cudaStream_t st, bool pdl) {
    const bool dual = a.epi == EPI_SWIGLU;
    const int tile_rows = p.tile_rows;
    typename BatchMapsFor<FMT>::type km;
    BatchArgs b = {};
    b.rowbytes = fmt_row_bytes(FMT, a.K);
    size_t wbytes = 0;
    int t0 = 0;
    // rows of whole columns: one copy per stage and weight; else one per column, whose map knows where the rows end
    const bool wide = b.rowbytes % 128 == 0;
    auto weight_map = [&](CUtensorMap* m, const uint8_t* W, int N) {
        return wide ? make_columns_map(m, W, N, b.rowbytes, tile_rows, p.cols) : make_weight_map(m, W, N, b.rowbytes, tile_rows);
    };
    for (int i = 0; i < a.nseg; ++i) {
        b.seg[i].scale = a.seg[i].scale;
        b.seg[i].bias = a.seg[i].bias;
        b.seg[i].out = a.seg[i].out;
        b.seg[i].N = a.seg[i].N;
        b.seg[i].ld = a.seg[i].ld_out;
        b.seg[i].tile0 = t0;
        t0 += (a.seg[i].N + tile_rows - 1) / tile_rows;
        wbytes += (size_t)a.seg[i].N * b.rowbytes;
        if (!weight_map(&km.tm[i], a.seg[i].W, a.seg[i].N)) return cudaErrorInvalidValue;
    }
    if (dual && !weight_map(&km.tm[3], a.W2, a.seg[0].N)) return cudaErrorInvalidValue;
    if (!make_rows_map(&km.x, a.x, a.M, a.K * 2, a.x_pitch ? a.x_pitch : a.K * 2, p.xcols, p.halves ? 8 : a.M)) return cudaErrorInvalidValue;
    if (!fill_scale_maps(km, a, p.cols * 16, tile_rows)) return cudaErrorInvalidValue;
    b.scale2 = a.scale2;
    b.norm_w = a.norm_w;
    b.norm_eps = a.norm_eps;
    b.status = a.status;
    b.M = a.M;
    b.K = a.K;
    b.halves = p.halves ? 1 : 0;
    b.cols = p.cols;
    b.wide = wide ? 1 : 0;
    b.xcols = p.xcols;
    b.epi = a.epi;
    b.nseg = a.nseg;
    b.ntiles = t0;
    b.tile_rows = tile_rows;
    b.kcb = p.kcb;
    b.nchunks = (b.rowbytes + p.kcb - 1) / p.kcb;
    b.groups = (b.nchunks + NCW - 1) / NCW;
    b.stages = p.stages;
    b.stage_bytes = p.stage_bytes;
    b.evict_first = wbytes > ((size_t)96 << 20) ? 1 : 0;   // weights that cannot stay in L2 anyway are streamed evict-first
    b.off_ctab = p.off_ctab;
    b.off_red = p.off_red;
    b.off_ring = p.off_ring;
    if constexpr (FMT != FMT_INT8) {
        if (a.M > 8) return launch_n<FMT, 2>(km, b, p, st, pdl);
    }
    return launch_n<FMT, 1>(km, b, p, st, pdl);
}

}  // namespace

cudaError_t batch_configure() {
    cudaError_t e = cudaSuccess;
#define SET_SMEM(F, N) \
    if (e == cudaSuccess) e = cudaFuncSetAttribute(linear_batch_kernel<F, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    SET_SMEM(FMT_FP16, 1) SET_SMEM(FMT_FP16, 2) SET_SMEM(FMT_INT8, 1) SET_SMEM(FMT_Q4, 1) SET_SMEM(FMT_Q4, 2)
#undef SET_SMEM
    return e;
}

// Where the streaming kernel is the faster one although its tiles split K too: there the rows are staged by a launch before (small Q4 batches
// without a norm: by each block), here they come into every block, which applies the norm and builds the Q4 starts or the int8 limbs anew.
// The more tiles and the longer the rows, the more of that, and the less a launch counts.  All times in us, "here / there", of recorded
// operators one after another over weights that come from memory.
static bool stream_is_faster(int fmt, const LinArgs& a, BatchNorm norm, int sm_count) {
    const int tiles = count_tiles(a, a.epi == EPI_SWIGLU ? 16 : WARP_ROWS), M = a.M, K = a.K;
    const int two_per_sm = 2 * sm_count + 8;   // (with a few blocks that take a second tile: 4864 x 896, gate and up, has 304)
    if (norm == BatchNorm::staged && tiles * K <= 100 * 1024) return false;   // two launches both ways, and the host is what counts: q/k/v 2048 x 1024: 6.5 / 7.2
    const bool two_waves = tiles > two_per_sm - sm_count / 3 && tiles <= two_per_sm;   // int8 above 8 rows: a wave is a tile per SM
    if (fmt == FMT_Q4) {
        if (norm == BatchNorm::staged) return true;            // gate and up 8192 x 1536, 2 rows: 12.2 / 8.4
        if (norm == BatchNorm::here) {
            if (K > 1536) return true;                         // 2048 x 2048, 2 rows: 6.1 / 5.5; 1024 x 1024: 3.5 / 4.2
            if (M > 8) return M * K > 9216 || tiles > 48;      // two rows to normalise per warp: 1536 x 576, gate and up, 16 rows: 5.6 / 5.0; 896 x 896, 9 rows: 4.6 / 4.8
            // gate and up 4608 x 1024, 8 rows: 6.6 / 5.7; 4864 x 896, 5 rows: 6.2 / 6.9; 9461 x 384, 6 rows: 5.7 / 5.1
            if (tiles > sm_count) return M * K > 4608 || tiles > two_per_sm || (M >= 4 && K <= 640);
            // 4494 x 832, 5 rows: 5.1 / 4.7; 576 x 1536, 8 rows: 5.1 / 4.9; gate and up 719 x 1536, 5 rows: 5.6 / 5.3
            return M * K > 8192 || (M >= 4 && K > 768 && tiles > 110) || (M >= 5 && K > 1408 && tiles > 40);
        }
        if (M * K < 12288) {                                   // one launch there too
            if (K <= 384) return M > 4 || tiles > 48;          // q/k/v 5625 x 384, 8 rows: 4.4 / 3.4; gate and up 970 x 320, 9 rows: 3.4 / 3.0
            if (K <= 640 && M >= 6 && tiles > 140) return true;   // 8770 x 448, 8 rows: 4.8 / 4.0
        }
        if (tiles <= 48) return M > 14 && K > 2048 && K <= 2816;   // 896 x 4864, 8 rows: 7.1 / 8.4; 896 x 896: 2.9 / 3.1; 500 x 2624, 16 rows: 7.1 / 6.3
        if (K > 4096) return tiles > sm_count;                 // 2048 x 8192, 8 rows: 10.7 / 13.9; q/k/v 6000 x 8192, 4 rows: 18.0 / 16.9
        if (K <= 1024 && M >= 6) return tiles > (M <= 8 ? two_per_sm : sm_count);   // 4864 x 896, 8 rows: 4.1 / 4.7; gate and up, 16 rows: 7.3 / 7.1
        return true;                                           // 2048 x 2048, 5 rows: 5.6 / 4.8; 9400 x 1024, 2 rows: 4.9 / 3.9
    }
    if (fmt == FMT_INT8) {
        // limbs: three bytes per value, which must leave room for the ring there
        const bool roomy = 3ll * M * K <= (M <= 8 ? 40000 : 147456);
        if (norm == BatchNorm::staged || (norm == BatchNorm::here && K > 1536))
            return roomy || tiles <= 3 * sm_count;             // 3000 x 2048, gate and up, 5 rows: 7.7 / 6.5; 9000 x 4096, 8 rows: 20.6 / 27.0
        if (norm == BatchNorm::here) {
            // gate and up 4608 x 1024, 5 rows: 5.9 / 5.2; 3757 x 1152, 4 rows: 5.3 / 4.9; q/k/v 2203 x 1472, 8 rows: 6.0 / 5.2; 2048 x 1024: 4.5 / 4.7
            if (M <= 8) return tiles > (K <= 928 ? 200 : K <= 1408 ? 110 : 60);
            if (M > 12 && K <= 960 && two_waves) return false; // gate and up 4864 x 896, 16 rows: 8.7 / 9.3; 6764 x 960, 212 tiles: 7.9 / 7.2
            // two blocks per tile: 4864 x 896, 9 rows: 6.7 / 5.7; 4318 x 512, 9 rows: 5.1 / 4.6; q/k/v 1152 x 896: 4.4 / 4.6; gate and up 532 x 1216, 14 rows: 5.4 / 4.7
            return tiles > (K <= 384 ? sm_count : K <= 640 ? 128 : K <= 1088 ? 48 : 32);
        }
        if (!roomy) return false;                              // 28672 x 4096, 8 rows: 27.7 / 35.5, 16 rows: 47.4 / 75.4
        if (M <= 8) {                                          // 18900 x 1024, 8 rows: 8.7 / 7.4; gate and up 14000 x 2048, 5 rows: 14.1 / 15.0; 4534 x 4288, 2 rows: 15.2 / 11.9
            const bool parts = K >= 2048 && K % 128 != 0;      // (a copy per column)
            return K >= 512 && (parts ? tiles > sm_count : K < 2048 && tiles > two_per_sm);
        }
        if (tiles > 2 * two_per_sm) return true;               // 30000 x 320, 16 rows: 14.0 / 10.1
        // 17167 x 448, 9 rows: 9.9 / 6.6; 9543 x 384, 12 rows: 6.5 / 6.8; gate and up 7162 x 384, 9 rows: 7.1 / 6.6 (16 weight rows a tile)
        if (K < 512) return a.epi != EPI_SWIGLU && tiles > 160 && !two_waves;
        // 4096 x 4096, 9 rows: 10.5 / 9.3; 9400 x 1536, 12 rows: 16.6 / 12.7; 5323 x 768, 12 rows: 5.9 / 5.5; q/k/v 13939 x 576, 14 rows: 11.6 / 8.4; 4864 x 896, 16 rows: 5.7 / 6.7
        if (M <= 12) return tiles > (M < 12 && K > 640 ? 120 : sm_count);
        return tiles * K > 450000 || (K <= 640 && tiles > two_per_sm);
    }
    if (norm == BatchNorm::staged)   // gate and up 4864 x 896, 2 rows: 7.7 / 6.9; 2048 x 2048, 2 rows: 7.4 / 8.7, 9 rows: 8.0 / 6.3; gate and up 9000 x 4096, 8 rows: 29.5 / 48.5
        return K < 4096 && (tiles > sm_count ? M * K <= 16384 : K < 2048 || M > 8);
    if (norm == BatchNorm::here)
        return (K >= 1024 && K <= 1088 && tiles > 200 && tiles <= 2 * sm_count) ||             // gate and up 4608 x 1024, 8 rows: 6.9 / 6.1; 4864 x 896: 6.5 / 8.2
               (M <= 8 && K >= 448 && K <= 768 && tiles > 3 * sm_count) ||                     // q/k/v 11903 x 768, 4 rows: 8.5 / 7.1
               (a.epi == EPI_SWIGLU && M > 8 && K < 512 && tiles > sm_count) ||                // gate and up 12522 x 384, 16 rows: 8.8 / 7.7
               (M > 8 && M * K >= 16384 && K < 4096 && tiles >= 32 && tiles <= sm_count);      // 2048 x 2048, 12 rows: 8.1 / 6.4
    return false;                                              // 576 x 576, 2 rows: 2.1 / 3.3; 28672 x 4096, 16 rows: 52 / 69
}

// Which batched calls this kernel takes: those that the streaming kernel takes with K split, whose activations are whole 128-byte columns and fit
// in shared memory beside two stages of weights, and (Q4) whose block scales can be reached by tensor copies.  The K parts are the single call's.
// Not those that are faster there (above), unless it would take other K parts than the single call's: a batch's rows have the single call's
// bits, and a recorded call those of the eager one, whichever way each goes.
// Nor whole-row tiles (an lm_head): the finish there needs no meeting of warps in the streaming kernel (16 rows of 151936 x 896 in fp16: 48 us in
// both; 8 rows of 65536 x 1024 in Q4 20.6 against 16.5).
BatchPlan batch_plan(int fmt, const LinArgs& a, BatchNorm norm, int sm_count, size_t smem_limit) {
    BatchPlan p = {};
    if (a.M < 2 || a.npeer > 0 || a.sig.world > 0 || a.argmax_slot || !stream_supported(fmt, a.M, a.K, a)) return p;
    for (int i = 0; i < a.nseg; ++i)
        if (!a.seg[i].out) return p;
    const uint16_t* base[4];
    int pitch = 0;
    if (fmt == FMT_Q4 && !q4_scale_views(a, base, &pitch)) return p;
    const StreamPart part = stream_part(fmt, a, sm_count);
    if (part.kw == 1) return p;
    p.streams = stream_is_faster(fmt, a, norm, sm_count) && stream_keeps_parts(fmt, a, part, smem_limit);
    if (p.streams) return p;
    const bool dual = a.epi == EPI_SWIGLU;
    p.halves = fmt == FMT_INT8 && a.M > 8;
    const int rb = fmt_row_bytes(fmt, a.K), nt = a.M > 8 && !p.halves ? 2 : 1, warp_rows = dual ? 16 : WARP_ROWS;
    p.kcb = part.kcb;
    p.tile_rows = warp_rows;
    const int nchunks = (rb + p.kcb - 1) / p.kcb, groups = (nchunks + NCW - 1) / NCW;
    // Few tiles of long rows: half tiles on twice the SMs, whose warps have half the weights each (tiles do not enter the sums): Q4
    // 1024 x 4608, 8 rows, 8.4 -> 7.4 us.  Rows of one stage gain nothing (1024 x 1024: 3.3 against 3.5 us).
    if (!dual && groups > 1 && count_tiles(a, WARP_ROWS) * (p.halves ? 4 : 2) <= sm_count) p.tile_rows = 16;
    p.ntiles = count_tiles(a, p.tile_rows);
    p.cols = groups == 1 ? (rb + 127) / 128 : NCW * (p.kcb / 128);   // (not more than there are: what lies past the end takes a copy long)
    p.xcols = batch_xcols(fmt, a.K);
    if (a.K % 64 != 0 || p.xcols > 256 || p.cols * 16 > 256) return p;   // one copy's reach
    if (a.norm_w && a.K * 2 > batch_red_bytes(fmt, nt)) return p;       // the norm weight lies where the sums will
    const int sets = dual ? 2 : 1;
    p.stage_bytes = (sets * p.tile_rows * p.cols * (128 + (fmt == FMT_Q4 ? 16 : 0)) + 1023) / 1024 * 1024;
    const int xrow = p.xcols * 128;
    p.off_ring = OFF_X + (batch_xrows(p.halves ? 8 : a.M, nt) * xrow + 1023) / 1024 * 1024;
    // Two blocks per SM where that leaves each at least two stages (or all of its items): a block of the next launch can then be resident, with
    // its weights on their way, before this one's is done.  With long rows one block and a deep ring are better, also for so few rows of
    // activations that two blocks would fit (fp16 2048 x 8192, 3 rows: 14.4 us as two blocks, 10.5 as one); so are few tiles, where it asks for
    // so much shared memory that the next launch's blocks go to SMs that are idle (Q4 1024 x 4608, 3 rows: 6.9 and 6.0 us).
    const bool deep = groups > 4 || p.ntiles * (p.halves ? 2 : 1) * 2 <= sm_count;
    const int ctab = ctab_bytes_of(fmt, a.M, a.K), red = batch_red_bytes(fmt, nt), rest = ctab + red;
    for (int ps = 2; ps >= 1; --ps) {
        const long long budget = (long long)((smem_limit + 1024) / ps) - 1024 - 1024 - rest;   // 1 KB to align the start
        const int resident = sm_count * ps / (p.halves ? 2 : 1), waves = (p.ntiles + resident - 1) / resident, items = waves * groups;
        const int least = items < 2 ? 1 : 2;
        if (budget - (ps == 2 && deep ? OFF_X + 8 * nt * xrow : p.off_ring) < (long long)least * p.stage_bytes) continue;
        int st = (int)((budget - p.off_ring) / p.stage_bytes);
        if (st > items) st = items;
        if (st > BATCH_STAGES) st = BATCH_STAGES;
        p.stages = st;
        p.grid = (p.ntiles < resident ? p.ntiles : resident) * (p.halves ? 2 : 1);
        p.off_ctab = p.off_ring + st * p.stage_bytes;
        p.off_red = p.off_ctab + ctab;
        p.smem = (size_t)p.off_red + red + 1024;
        if (ps == 1 && p.smem < (smem_limit + 1024) / 2) p.smem = (smem_limit + 1024) / 2;
        p.ok = true;
        break;
    }
    return p;
}

cudaError_t launch_batch(int fmt, const LinArgs& a, const BatchPlan& p, cudaStream_t st, bool pdl) {
    if (fmt == FMT_FP16) return launch_f<FMT_FP16>(a, p, st, pdl);
    if (fmt == FMT_INT8) return launch_f<FMT_INT8>(a, p, st, pdl);
    if (fmt == FMT_Q4) return launch_f<FMT_Q4>(a, p, st, pdl);
    return cudaErrorInvalidValue;
}

}  // namespace nnb
