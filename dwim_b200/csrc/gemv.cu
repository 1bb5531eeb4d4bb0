// The small-M product (decode and speculative verify): out[t][r] = w[r] . x[t]
// for up to eight tokens, bound by how fast the packed weights stream from HBM.
//
// Replaces the reference's matmul_tile16_* / matmul_rows* kernels for few
// tokens (matmul_tile.cu:94-258, matmul_rows.cu:29-184; dispatch at
// gpu/cuda/mod.rs:1084-1131).
//
// Shape of the kernel
//   - Persistent grid, one CTA per SM.  A CTA walks tiles of R = 16*RT weight
//     rows; for each tile it streams the rows' packed blocks, K in chunks of
//     `kc` units of 256 weights, through a ring of shared-memory stages.
//   - One producer warp fills the ring with cp.async.bulk (the TMA engine's
//     untiled copy): a stage of whole rows is one contiguous run of HBM and one
//     copy (plus one for the rows' scales where the format keeps them apart);
//     longer rows are cut in chunks, one box of a tensor map each (Q8_0, whose
//     units would all start in the same bank: a swizzled box per 128 bytes).  Stages are
//     handed over with mbarriers (full: transaction bytes; empty: one arrival
//     per consumer warp).  Every wait is bounded.
//   - RT*KS consumer warps.  Warp (rt, ks) owns row tile rt and every KS-th
//     unit of a chunk.  The quants stay integers: nibbles (Q4_K) are masked
//     four at a time, Q6_K's six bits assembled into signed bytes, Q8_0's bytes
//     used as they are, and multiplied on the tensor cores (mma.sync int8,
//     weight rows on the M side) with the activations' signed base-256 digit
//     planes as columns (prologue.cu).  The integer sums of a sub-block are
//     weighted by its scale (integer multiply-add for the 6-bit and 8-bit
//     sub-scales, fp32 for Q8_0's f16 ones), and the unit's d and the plane's
//     worth scale once per unit in fp32: the result differs from the CPU's by
//     fp32 summation order and the planes' rounding (2^-31 or 2^-23 of a unit's
//     largest activation).
//   - The K-split warps of a row tile are summed through shared memory in a
//     fixed order (deterministic), then the epilogue stores, adds to, or
//     SwiGLU-combines the output (modes after prelude.cu:29-35).
#include <cuda_fp16.h>
#include <stdlib.h>

#include <atomic>

#include "common.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace dwim {

constexpr int MAX_STAGES = 8;

struct GemvArgs {
    WeightView w;
    const uint8_t *panels;   // [units][i8_unit_bytes(ncols)]: the activations' digit planes (prologue.cu)
    int xunit;               // bytes of one unit's panels for this launch
    int xsrc_stride;         // bytes between units in the panel array
    // SwiGLU in one launch (int8 routine): `w` is the gate matrix, these the quants and scales of
    // the up matrix of the same shape; a CTA takes a row tile of the one, then of the other, and
    // writes silu(gate . x) * (up . x).  Null: an ordinary product.
    const uint8_t *up_quants;
    const __half *up_scales;
    int ncols;               // digit-plane columns: planes * tokens
    int n_tokens;            // tokens of this launch
    size_t t0;               // first token's index in out
    size_t group_panels;     // bytes from a group's panels to the next's; blockIdx.y is the group
    OutSpec out;
    const float *aux;        // EPI_SWIGLU: the `up` product, token-major [n][rows]
    int epi;
    int units;               // ceil(cols / 256)
    int kc;                  // units per stage
    int n_tiles;
    int stages;
    int q_stride;            // bytes between rows of a stage's quant region
    int s_off, s_stride;     // scale region
    int x_off;               // panel region (when the panels travel with the stages)
    int stage_bytes;
    int whole_rows;          // 1: a stage holds whole rows (kc == units): one copy for the tile's quants, one for its scales
    int boxed;               // 1: a chunk is one box of the tensor map, rows kc units apart in the stage, with the rows' scales whole
    int x_resident;          // 1: the launch's panels sit in shared memory for the CTA's whole life
    int xres_bytes;
    uint32_t *status;
    int groups;              // groups of n_tokens tokens (host side: the grid's second extent)
};


// The formats as the int8 tensor-core routines read them.
constexpr int Q4K_I8 = 1012;
constexpr int Q8_I8 = 1008;
constexpr int Q6K_I8 = 1014;
constexpr bool is_i8(int fmt) { return fmt == Q4K_I8 || fmt == Q8_I8 || fmt == Q6K_I8; }
constexpr int base_of(int fmt) { return fmt == Q4K_I8 ? (int)Q4_K : fmt == Q8_I8 ? (int)Q8_0 : fmt == Q6K_I8 ? (int)Q6_K : fmt; }

template <int FMT> struct Traits;
template <> struct Traits<Q4K_I8> { static constexpr int UNIT_Q = 144; };
template <> struct Traits<Q8_I8> { static constexpr int UNIT_Q = 256; };
template <> struct Traits<Q6K_I8> { static constexpr int UNIT_Q = 208; };

// What a consumer lane needs to know about the stage it reads.
struct Lane {
    int g, c;                // row within the 8-row group; k-quarter
    uint32_t row_a, row_b;   // shared addresses of rows g and g+8 (quant region)
    uint32_t srow_a, srow_b; // shared addresses of the rows' scales
    // Q8_0: a unit's halves of 128 bytes `half` apart, units `unit` apart; `byte0` is the lane's place in a
    // half (its bytes of block j: (32 j) ^ byte0, which a swizzled half's 16-byte chunks need)
    uint32_t unit, half, byte0;
    uint32_t xbase;          // shared address of the launch's panels (unit 0 of the stage, or of the row when resident)
};

// ---------------------------------------------------------------------------
// the unit routines
// ---------------------------------------------------------------------------
// Q4_K's nibbles stay integers: four of them per AND, multiplied on the tensor
// cores (mma.sync m16n8k32 u8 x s8 -> s32) with the activations' signed
// base-256 digit planes as columns (prologue.cu).
// One MMA covers one 32-weight sub-block of 16 rows; its sums are weighted by
// the sub-block's 6-bit scale with integer multiply-adds, so a whole unit is an
// exact integer per (row, column), which d and the plane's worth then scale.
// High nibbles are masked in place (16*q: no shift), the low ones' scales are
// 16 times larger instead, and the unit's sum is divided by 16 in d.  The minimums
// use the digits' per-sub-block sums (dp4a).
// c = a * b (the accumulator operand is zero, not a register that has to be cleared first)
__device__ __forceinline__ void imma_u8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {   // a unsigned bytes, b signed bytes
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ float2 lds64f2(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}

__device__ __forceinline__ void imma_s8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
// 16 rows x 16 k: one 16-weight scale group of Q6_K
__device__ __forceinline__ void imma16_s8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ float lds32f(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}

// The digit planes' columns as the int8 routines see them: NTILE column tiles
// of the MMA (8 columns each).  Tile p's column g is blob column
// p*tile_stride + g, present when g < tile_cols.
//   one and two tokens:  one tile, column = 4*token + plane, tile_cols = 4n
//   three to five:       two tiles, the first eight of the blob's 3n columns and the last eight, so that
//                        neither reads past them (plane p of token t is column p*n + t): a third fewer MMAs
//                        and multiplies than a tile per plane ([17408, 5120] Q4_K by five tokens 25.0 us,
//                        21.4 like this); a token's planes meet after the K-split sums
//   six to eight:        a tile per plane, column g = token g, tile_stride = tile_cols = n
// In all a lane's accumulators are (row a | row b) x (tile column 2c, 2c+1).
// One token of Q6_K fills half a tile, so its columns 4..7 take a second scale group: B is block
// diagonal over K (columns 0..3 hold the planes' digits in the first 16 of an MMA's K and zeros in the
// rest, columns 4..7 the other way round), two groups share an MMA's results and their scales' multiplies
// ([151936, 5120] with norm and arg-max 160 us without, 147 with; Q8_0, built the same way, gained nothing).
struct I8Cols {
    int nc;           // columns in a unit's blob
    int tile_stride;
    int tile_cols;
    // the column a lane's B fragment of tile 0 comes from: the sums of columns that are not there are not used
    __host__ __device__ constexpr int lane_col(int g) const { return g < tile_cols ? g : 0; }
};
template <int NTILE> __host__ __device__ constexpr I8Cols i8_cols(int nc, int n_tokens) {
    return I8Cols{nc, NTILE == 1 ? 0 : NTILE == 2 ? nc - 8 : n_tokens, NTILE == 1 ? nc : NTILE == 2 ? 8 : n_tokens};
}
// Column tiles of n tokens (of any format): one (4 planes x 1-2 tokens), two (3 planes x 3-5 tokens), one per plane.
__host__ __device__ constexpr int i8_tiles(int n) { return n <= 2 ? 1 : n <= 5 ? 2 : 3; }
// Every lane's column of every tile is one of the blob's.
template <int NTILE> constexpr bool i8_columns_exist() {
    for (int n = 1; n <= I8_MAX_TOKENS; n++) {
        if (i8_tiles(n) != NTILE) continue;
        const I8Cols X = i8_cols<NTILE>(i8_planes(n) * n, n);
        for (int g = 0; g < 8; g++)
            for (int p = 0; p < NTILE; p++)
                if (X.lane_col(g) + p * X.tile_stride >= X.nc) return false;
    }
    return true;
}
static_assert(i8_columns_exist<1>() && i8_columns_exist<2>() && i8_columns_exist<3>(), "a lane reads past a unit's planes");

// Q4_K.  Lane (g, c) owns bytes [8c, 8c+8) of each 32-byte group of its two rows: MMA
// k-slots 4c..4c+3 and 16+4c..16+4c+3, matched by the same eight digits of the
// lane's column.  acc: (row a, col 2c), (row a, col 2c+1), (row b, ..), (row b, ..),
// summed over the tiles (the planes of a token, in the layout of three to eight tokens).
template <int NTILE>
__device__ __forceinline__ void unit_q4k_i8(const Lane &L, const I8Cols X, int ul, int xu, float (&acc)[NTILE == 2 ? 8 : 4]) {
    const uint32_t ba = L.row_a + ul * 144, bb = L.row_b + ul * 144;
    const uint4 ha = lds128(ba), hb = lds128(bb);
    const uint32_t blob = L.xbase + xu * i8_unit_bytes(X.nc);
    // the 6-bit scales and minimums as bytes: entries 0..3 and 4..7
    const uint32_t sa[2] = {ha.y & 0x3f3f3f3fu, (ha.w & 0x0f0f0f0fu) | ((ha.y >> 2) & 0x30303030u)};
    const uint32_t sb[2] = {hb.y & 0x3f3f3f3fu, (hb.w & 0x0f0f0f0fu) | ((hb.y >> 2) & 0x30303030u)};
    int is[NTILE][4];   // at most 4 * (16 * 63) * (32 * 15 * 128) + 4 * 63 * (32 * 240 * 128) < 2^29
#pragma unroll
    for (int p = 0; p < NTILE; p++)
#pragma unroll
        for (int i = 0; i < 4; i++) is[p][i] = 0;
    const uint32_t qa = ba + 16 + 8 * L.c, qb = bb + 16 + 8 * L.c;
    uint32_t xcol = blob + X.lane_col(L.g) * 32 + 8 * L.c;   // this lane's column of tile 0, sub-block 0
    const uint32_t xstep = 32 * X.nc;                // a sub-block further on
    const uint32_t tstep = 32 * X.tile_stride;       // a tile further on
#pragma unroll
    for (int G = 0; G < 4; G++) {   // group G: low nibbles = sub-block 2G, high nibbles = 2G+1
        const uint2 wa = lds64(qa + 32 * G), wb = lds64(qb + 32 * G);
        // the two sub-blocks' scales: bytes 2(G&1) and 2(G&1)+1 of the word, each by one byte permute
        const int s0a = (int)prmt(sa[G >> 1], 0u, 0x4440u + 2 * (G & 1)) << 4, s1a = (int)prmt(sa[G >> 1], 0u, 0x4441u + 2 * (G & 1));
        const int s0b = (int)prmt(sb[G >> 1], 0u, 0x4440u + 2 * (G & 1)) << 4, s1b = (int)prmt(sb[G >> 1], 0u, 0x4441u + 2 * (G & 1));
#pragma unroll
        for (int p = 0; p < NTILE; p++) {
            const uint2 x0 = lds64(xcol + p * tstep), x1 = lds64(xcol + p * tstep + xstep);
            int c0[4], c1[4];
            imma_u8s8(c0, wa.x & 0x0f0f0f0fu, wb.x & 0x0f0f0f0fu, wa.y & 0x0f0f0f0fu, wb.y & 0x0f0f0f0fu, x0.x, x0.y);
            imma_u8s8(c1, wa.x & 0xf0f0f0f0u, wb.x & 0xf0f0f0f0u, wa.y & 0xf0f0f0f0u, wb.y & 0xf0f0f0f0u, x1.x, x1.y);
            is[p][0] += s0a * c0[0]; is[p][1] += s0a * c0[1]; is[p][2] += s0b * c0[2]; is[p][3] += s0b * c0[3];
            is[p][0] += s1a * c1[0]; is[p][1] += s1a * c1[1]; is[p][2] += s1b * c1[2]; is[p][3] += s1b * c1[3];
        }
        xcol += 2 * xstep;
    }
    // minimums: sum_j m_j * (128*a_j + b_j) per column
    const uint32_t ma[2] = {ha.z & 0x3f3f3f3fu, ((ha.w >> 4) & 0x0f0f0f0fu) | ((ha.z >> 2) & 0x30303030u)};
    const uint32_t mb[2] = {hb.z & 0x3f3f3f3fu, ((hb.w >> 4) & 0x0f0f0f0fu) | ((hb.z >> 2) & 0x30303030u)};
    const float da = h2f_lo(ha.x) * 0.0625f, dma = h2f_hi(ha.x), db = h2f_lo(hb.x) * 0.0625f, dmb = h2f_hi(hb.x);
    if constexpr (NTILE == 1) {
        // one tile of 4n columns: the lane's two columns exist together, their sums and worths sit side by side
        uint4 t0 = make_uint4(0, 0, 0, 0), t1 = t0;
        float2 worth = make_float2(0.0f, 0.0f);
        if (2 * L.c < X.tile_cols) {
            t0 = lds128(blob + 256 * X.nc + (2 * L.c) * 16);
            t1 = lds128(blob + 256 * X.nc + (2 * L.c + 1) * 16);
            worth = lds64f2(blob + 272 * X.nc + 8 * L.c);
        }
        const int m0 = (dp4a_us(ma[1], t0.y, dp4a_us(ma[0], t0.x, 0)) << 7) + dp4a_us(ma[1], t0.w, dp4a_us(ma[0], t0.z, 0));
        const int m1 = (dp4a_us(ma[1], t1.y, dp4a_us(ma[0], t1.x, 0)) << 7) + dp4a_us(ma[1], t1.w, dp4a_us(ma[0], t1.z, 0));
        const int m2 = (dp4a_us(mb[1], t0.y, dp4a_us(mb[0], t0.x, 0)) << 7) + dp4a_us(mb[1], t0.w, dp4a_us(mb[0], t0.z, 0));
        const int m3 = (dp4a_us(mb[1], t1.y, dp4a_us(mb[0], t1.x, 0)) << 7) + dp4a_us(mb[1], t1.w, dp4a_us(mb[0], t1.z, 0));
        acc[0] += worth.x * (da * (float)is[0][0] - dma * (float)m0);
        acc[1] += worth.y * (da * (float)is[0][1] - dma * (float)m1);
        acc[2] += worth.x * (db * (float)is[0][2] - dmb * (float)m2);
        acc[3] += worth.y * (db * (float)is[0][3] - dmb * (float)m3);
    } else {
#pragma unroll
        for (int p = 0; p < NTILE; p++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                uint4 t = make_uint4(0, 0, 0, 0);
                float worth = 0.0f;
                const int col = p * X.tile_stride + 2 * L.c + i;
                if (NTILE == 2 || 2 * L.c + i < X.tile_cols) {
                    t = lds128(blob + 256 * X.nc + col * 16);
                    worth = lds32f(blob + 272 * X.nc + 4 * col);
                }
                const int m_a = (dp4a_us(ma[1], t.y, dp4a_us(ma[0], t.x, 0)) << 7) + dp4a_us(ma[1], t.w, dp4a_us(ma[0], t.z, 0));
                const int m_b = (dp4a_us(mb[1], t.y, dp4a_us(mb[0], t.x, 0)) << 7) + dp4a_us(mb[1], t.w, dp4a_us(mb[0], t.z, 0));
                acc[(NTILE == 2 ? 4 * p : 0) + i] += worth * (da * (float)is[p][i] - dma * (float)m_a);
                acc[(NTILE == 2 ? 4 * p : 0) + 2 + i] += worth * (db * (float)is[p][2 + i] - dmb * (float)m_b);
            }
    }
}

// Q8_0.  A 32-weight block is one MMA (s8 x s8); its f16 scale weighs the block's
// integer sums in fp32.  Lane c owns bytes [8c, 8c+8) of each block.
template <int NTILE>
__device__ __forceinline__ void unit_q8_i8(const Lane &L, const I8Cols X, int ul, int xu, float (&acc)[NTILE == 2 ? 8 : 4]) {
    const uint32_t qa = L.row_a + ul * L.unit, qb = L.row_b + ul * L.unit;
    const uint4 sa = lds128(L.srow_a + ul * 16), sb = lds128(L.srow_b + ul * 16);
    const uint32_t sca[4] = {sa.x, sa.y, sa.z, sa.w}, scb[4] = {sb.x, sb.y, sb.z, sb.w};
    const uint32_t blob = L.xbase + xu * i8_unit_bytes(X.nc);
    float fs[NTILE][4];
#pragma unroll
    for (int p = 0; p < NTILE; p++)
#pragma unroll
        for (int i = 0; i < 4; i++) fs[p][i] = 0.0f;
    uint32_t xcol = blob + X.lane_col(L.g) * 32 + 8 * L.c;
    const uint32_t xstep = 32 * X.nc, tstep = 32 * X.tile_stride;
#pragma unroll
    for (int blk = 0; blk < 8; blk++) {
        const uint32_t at = (blk >> 2) * L.half + ((32u * (blk & 3)) ^ L.byte0);
        const uint2 wa = lds64(qa + at), wb = lds64(qb + at);
        const float da = (blk & 1) ? h2f_hi(sca[blk >> 1]) : h2f_lo(sca[blk >> 1]);
        const float db = (blk & 1) ? h2f_hi(scb[blk >> 1]) : h2f_lo(scb[blk >> 1]);
#pragma unroll
        for (int p = 0; p < NTILE; p++) {
            const uint2 x = lds64(xcol + p * tstep);
            int c[4];
            imma_s8s8(c, wa.x, wb.x, wa.y, wb.y, x.x, x.y);
            fs[p][0] += da * (float)c[0];
            fs[p][1] += da * (float)c[1];
            fs[p][2] += db * (float)c[2];
            fs[p][3] += db * (float)c[3];
        }
        xcol += xstep;
    }
#pragma unroll
    for (int p = 0; p < NTILE; p++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            float worth = 0.0f;
            const int col = p * X.tile_stride + 2 * L.c + i;
            if (NTILE == 2 || 2 * L.c + i < X.tile_cols) worth = lds32f(blob + 272 * X.nc + 4 * col);
            acc[(NTILE == 2 ? 4 * p : 0) + i] += worth * fs[p][i];
            acc[(NTILE == 2 ? 4 * p : 0) + 2 + i] += worth * fs[p][2 + i];
        }
}

// Q6_K.  One MMA of k = 16 per 16-weight scale group: lane c holds weights
// 4c..4c+3 of the group as signed bytes; the group's i8 sub-scale weighs its
// integer sums, d the unit's.  A lane's share of a row is three 128-bit loads: word j of
// the four sets of four groups, from which nine instructions a set make the groups' bytes,
// 4 * q each (formats.cuh); d takes the 4 back.  (Bound by issue: with the file's nibbles and bit pairs, twelve
// 32-bit loads and sixteen instructions, the [151936, 5120] product took 108 us at one token, 131 at two and 201 at
// eight; 100, 118 and 194 like this, 101, 110 and 168 to 174 with launch_shape's row tiles.)
__device__ __forceinline__ uint32_t word_of(const uint4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
template <int NTILE, bool ONE>
__device__ __forceinline__ void unit_q6k_i8(const Lane &L, const I8Cols X, int ul, int xu, int d_index, float (&acc)[NTILE == 2 ? 8 : 4]) {
    const uint32_t ba = L.row_a + ul * 208, bb = L.row_b + ul * 208;
    const uint4 ta = lds128(ba + 192), tb = lds128(bb + 192);
    const uint32_t sca[4] = {ta.x, ta.y, ta.z, ta.w}, scb[4] = {tb.x, tb.y, tb.z, tb.w};
    const float da = 0.25f * __half2float(__ushort_as_half((uint16_t)lds16(L.srow_a + 2 * d_index)));
    const float db = 0.25f * __half2float(__ushort_as_half((uint16_t)lds16(L.srow_b + 2 * d_index)));
    const uint32_t blob = L.xbase + xu * i8_unit_bytes(X.nc);
    int is[NTILE][4];
#pragma unroll
    for (int p = 0; p < NTILE; p++)
#pragma unroll
        for (int i = 0; i < 4; i++) is[p][i] = 0;
    uint4 wa[3], wb[3];      // word j of the four sets of four groups
#pragma unroll
    for (int j = 0; j < 3; j++) {
        wa[j] = lds128(ba + 64 * j + 16 * L.c);
        wb[j] = lds128(bb + 64 * j + 16 * L.c);
    }
    if constexpr (ONE) {
        const uint32_t first = L.g < 4 ? 0xffffffffu : 0u, mine = 0x8880u + (uint32_t)(L.c >> 1) * 0x1111u;
        const uint32_t x0 = blob + (L.g & 3) * 32 + 16 * (L.g >> 2) + 4 * L.c;      // four columns: 128 bytes a sub-block
#pragma unroll
        for (int t = 0; t < 4; t++) {
            uint32_t qa[4], qb[4];
            q6k_bytes(word_of(wa[0], t), word_of(wa[1], t), word_of(wa[2], t), qa);
            q6k_bytes(word_of(wb[0], t), word_of(wb[1], t), word_of(wb[2], t), qb);
#pragma unroll
            for (int k = 0; k < 2; k++) {
                // the groups 4 t + 2 k and + 1: this lane's results are of the one its columns belong to
                const int fa = (int)prmt(sca[t], 0u, mine + 2 * k * 0x1111u);
                const int fb = (int)prmt(scb[t], 0u, mine + 2 * k * 0x1111u);
                const uint32_t x = lds32(x0 + (2 * t + k) * 128);
                int c[4];
                imma_s8s8(c, qa[2 * k], qb[2 * k], qa[2 * k + 1], qb[2 * k + 1], x & first, x & ~first);
                is[0][0] += fa * c[0];
                is[0][1] += fa * c[1];
                is[0][2] += fb * c[2];
                is[0][3] += fb * c[3];
            }
        }
        const float2 worth = lds64f2(blob + 272 * 4 + 8 * (L.c & 1));
        acc[0] += worth.x * (da * (float)is[0][0]);
        acc[1] += worth.y * (da * (float)is[0][1]);
        acc[2] += worth.x * (db * (float)is[0][2]);
        acc[3] += worth.y * (db * (float)is[0][3]);
        return;
    }
    const uint32_t xlane = blob + X.lane_col(L.g) * 32 + 4 * L.c;
    const uint32_t xstep = 32 * X.nc, tstep = 32 * X.tile_stride;
#pragma unroll
    for (int t = 0; t < 4; t++) {
        uint32_t qa[4], qb[4];
        q6k_bytes(word_of(wa[0], t), word_of(wa[1], t), word_of(wa[2], t), qa);
        q6k_bytes(word_of(wb[0], t), word_of(wb[1], t), word_of(wb[2], t), qb);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            // byte k of the word, sign-extended (a selector nibble of 8 + b replicates byte b's sign)
            constexpr uint32_t SEXT = 0x8880u;
            const int fa = (int)prmt(sca[t], 0u, SEXT + k * 0x1111u);
            const int fb = (int)prmt(scb[t], 0u, SEXT + k * 0x1111u);
            // group 4 t + k: its half of the sub-block, digits 4c .. +3
            const uint32_t xo = (2 * t + (k >> 1)) * xstep + 16 * (k & 1);
#pragma unroll
            for (int p = 0; p < NTILE; p++) {
                const uint32_t x = lds32(xlane + xo + p * tstep);
                int c[4];
                imma16_s8s8(c, qa[k], qb[k], x);
                is[p][0] += fa * c[0];
                is[p][1] += fa * c[1];
                is[p][2] += fb * c[2];
                is[p][3] += fb * c[3];
            }
        }
    }
#pragma unroll
    for (int p = 0; p < NTILE; p++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            float worth = 0.0f;
            const int col = p * X.tile_stride + 2 * L.c + i;
            if (NTILE == 2 || 2 * L.c + i < X.tile_cols) worth = lds32f(blob + 272 * X.nc + 4 * col);
            acc[(NTILE == 2 ? 4 * p : 0) + i] += worth * (da * (float)is[p][i]);
            acc[(NTILE == 2 ? 4 * p : 0) + 2 + i] += worth * (db * (float)is[p][2 + i]);
        }
}

// ---------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------
__device__ __forceinline__ float silu_mul(float g, float u) {
    // gpu/cpu.rs:238-242, 425-427: g * (1 / (1 + exp(-g))) * u
    return g * (1.0f / (1.0f + expf(-g))) * u;
}

__device__ __forceinline__ void emit(const GemvArgs &a, size_t t, size_t r, float v) {
    if (r >= a.w.rows) return;
    if (a.out.scatter_per) {
        // a K-sharded product's partial sum: to the row's owner alone, into its slot for this rank
        const size_t owner = r / a.out.scatter_per, local = r - owner * a.out.scatter_per;
        float *d = a.out.dst[0];
#pragma unroll
        for (int p = 1; p < DWIM_MAX_WORLD; p++)
            if ((size_t)p == owner) d = a.out.dst[p];
        d[t * a.out.pitch + a.out.row0 + local] = v;
        return;
    }
    const size_t i = t * a.out.pitch + a.out.row0 + r;
    if (a.epi == EPI_ADD) v += a.out.dst[0][i];
    else if (a.epi == EPI_SWIGLU) v = silu_mul(v, a.aux[t * a.w.rows + r]);
    a.out.dst[0][i] = v;
    // a shared result: the same element of every peer's copy (plain stores over NVLink).  The
    // parameter array is indexed by constants only: a variable index would make the compiler keep
    // a copy of the kernel's parameters in local memory.
    if (a.out.world > 1) {
#pragma unroll
        for (int p = 1; p < DWIM_MAX_WORLD; p++)
            if (p < a.out.world) a.out.dst[p][i] = v;
    }
}

// The tensor maps of a boxed launch: quants and (Q8_0) scales of the matrix and of the up matrix.
struct BoxMaps {
    CUtensorMap q[2], s[2];
};

// NT: the column tiles of the MMA; 0: the one-token form of Q6_K (one tile, block diagonal).
template <int FMT, int NT, int RT, int KS>
__global__ void __launch_bounds__((RT * KS + 1) * 32, 1) dwim_smallm_kernel(const __grid_constant__ GemvArgs a, const __grid_constant__ BoxMaps maps) {
    constexpr int NW = RT * KS;
    constexpr int R = RT * 16;
    constexpr int UNIT_Q = Traits<FMT>::UNIT_Q;
    constexpr int BASE = base_of(FMT);
    constexpr bool HAS_SCALES = BASE == Q6_K || BASE == Q8_0;   // scales kept apart from the quants
    // a lane's four accumulators (two rows by two columns); the unit routines sum a token's planes as they
    // go, but for NT = 2, whose tiles are kept apart
    constexpr int NACC = NT == 2 ? 8 : 4;
    constexpr int RED_FLOATS = KS > 1 ? 2 * KS * RT * NACC * 32 : 0;

    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);   // full[MAX_STAGES], empty[MAX_STAGES], panels
    float *red = reinterpret_cast<float *>(smem + 256);
    uint8_t *xres = smem + 256 + ((RED_FLOATS * 4 + 127) & ~127);
    // boxes land on 128-byte boundaries, swizzled ones on 1024-byte ones
    constexpr uint32_t ALIGN = BASE == Q8_0 ? 1024 : 128;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = a.stages;
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + MAX_STAGES), xbar = smem_u32(bars + 2 * MAX_STAGES);
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, NW);
        }
        mbar_init(xbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // The next launch in the stream may start as soon as SMs free up: what it
    // does before its own griddep_wait() (streaming its weights) depends on
    // nothing this kernel writes.
    griddep_launch();

    const int n_chunks = (a.units + a.kc - 1) / a.kc;
    const uint8_t *const panels = a.panels + blockIdx.y * a.group_panels;
    const size_t t0 = a.t0 + (size_t)blockIdx.y * a.n_tokens;
    const uint32_t stage0 = (smem_u32(xres) + a.xres_bytes + ALIGN - 1) & ~(ALIGN - 1);

    if (warp == NW) {
        // ------------------------------ producer ------------------------------
        // Weights are written by uploads only, which are ordinary launches long
        // complete: their copies may start before the kernel ahead has finished.
        // The panels come from the prologue that may be that very kernel.
        // So: the first ring-full of weight stages is requested at once, then the
        // warp waits for the kernel ahead and requests the panels.
        uint32_t it = 0;
        const int my_tiles = (int)blockIdx.x < a.n_tiles ? (a.n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
        const int n_mats = a.up_quants ? 2 : 1;
        const uint32_t ahead = (uint32_t)min(S, my_tiles * n_mats * n_chunks);   // stages that need no free slot
        bool waited = false;
        for (int tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x)
        for (int mat = 0; mat < n_mats; mat++) {
            const uint8_t *wq = mat ? a.up_quants : a.w.quants;
            const __half *wsc = mat ? a.up_scales : a.w.scales;
            const size_t row0 = (size_t)tile * R;
            const int nrows = (int)min((size_t)R, a.w.rows - row0);
            for (int ch = 0; ch < n_chunks; ch++, it++) {
                const int s = it % S;
                const uint32_t ph = (it / S) & 1;
                mbar_wait(empty0 + 8 * s, ph ^ 1, a.status, 0x1u);
                const int u0 = ch * a.kc, kcc = min(a.kc, a.units - u0);
                const uint32_t qbytes = UNIT_Q * kcc;
                uint32_t sbytes = 0;
                size_t s_first = 0;   // first f16 of the row's scales to copy
                if (BASE == Q8_0) { sbytes = 16 * kcc; s_first = (size_t)8 * u0; }
                if (BASE == Q6_K) {
                    s_first = (size_t)(u0 & ~7);
                    size_t s_end = min((size_t)pad8(u0 + kcc), a.w.srow);
                    sbytes = (uint32_t)(s_end - s_first) * 2;
                }
                const uint32_t xbytes = a.x_resident ? 0u : (uint32_t)a.xunit;
                const uint32_t bar = full0 + 8 * s;
                if (a.whole_rows) {
                    if (lane == 0)
                        mbar_expect_tx(bar, nrows * (uint32_t)(a.w.qpitch + (HAS_SCALES ? a.w.srow * 2 : 0)) + kcc * xbytes);
                } else if (a.boxed) {   // a box counts whole, its rows and units past the matrix's end read as zeros
                    if (lane == 0)
                        mbar_expect_tx(bar, BASE == Q8_0 ? R * (kcc * UNIT_Q + a.kc * 16) + kcc * xbytes
                                                         : R * a.kc * UNIT_Q + (HAS_SCALES ? nrows * (uint32_t)a.w.srow * 2 : 0) + kcc * xbytes);
                } else if (lane == 0) {
                    mbar_expect_tx(bar, nrows * (qbytes + sbytes) + kcc * xbytes);
                }
                __syncwarp();
                const uint32_t st = stage0 + s * a.stage_bytes;
                if (a.whole_rows) {
                    // consecutive rows are one contiguous run (rows sit qpitch apart, and so do the stage's)
                    if (lane == 0) bulk_g2s(st, wq + row0 * a.w.qpitch, nrows * (uint32_t)a.w.qpitch, bar);
                    if (HAS_SCALES && lane == 1)
                        bulk_g2s(st + a.s_off, wsc + row0 * a.w.srow, nrows * (uint32_t)a.w.srow * 2, bar);
                } else if (a.boxed) {
                    const CUtensorMap *qm = mat ? &maps.q[1] : &maps.q[0], *sm = mat ? &maps.s[1] : &maps.s[0];
                    if (BASE == Q8_0) {
                        if (lane < 2 * kcc) tma_load_2d(st + lane * R * 128, qm, u0 * 256 + lane * 128, (int)row0, bar);
                        if (lane == 31) tma_load_2d(st + a.s_off, sm, u0 * 8, (int)row0, bar);
                    } else if (lane == 0) {
                        tma_load_2d(st, qm, u0 * (UNIT_Q / 8), (int)row0, bar);
                    }
                    if (BASE == Q6_K && lane == 1)
                        bulk_g2s(st + a.s_off, wsc + row0 * a.w.srow, nrows * (uint32_t)a.w.srow * 2, bar);
                } else {
                    for (int r = lane; r < nrows; r += 32) {
                        bulk_g2s(st + r * a.q_stride, wq + (row0 + r) * a.w.qpitch + (size_t)u0 * UNIT_Q, qbytes, bar);
                        if (HAS_SCALES)
                            bulk_g2s(st + a.s_off + r * a.s_stride, wsc + (row0 + r) * a.w.srow + s_first, sbytes, bar);
                    }
                }
                if (!waited && (!a.x_resident || it + 1 == ahead)) {
                    griddep_wait();
                    waited = true;
                    if (a.x_resident && lane == 0) {
                        // the launch's panels are one contiguous run
                        mbar_expect_tx(xbar, a.xres_bytes);
                        bulk_g2s(smem_u32(xres), panels, a.xres_bytes, xbar);
                    }
                }
                for (int u = lane; u < kcc && !a.x_resident; u += 32)
                    bulk_g2s(st + a.x_off + u * xbytes, panels + (size_t)(u0 + u) * a.xsrc_stride, xbytes, bar);
            }
        }
        // Drain: the copies this warp issued must have landed before the CTA's
        // shared memory is given up.  Normally the consumers have already
        // waited on every stage and this returns at once.
        if (*(volatile uint32_t *)a.status != 0) {
            uint64_t start = globaltimer();
            uint32_t first = it > (uint32_t)S ? it - S : 0;
            for (uint32_t i = first; i < it; i++) {
                while (!mbar_try(full0 + 8 * (i % S), (i / S) & 1))
                    if (globaltimer() - start > WAIT_LIMIT_NS) break;
            }
        }
        return;
    }

    // -------------------------------- consumers --------------------------------
    const int rt = warp % RT, ks = warp / RT;
    Lane L;
    L.g = lane >> 2;
    L.c = lane & 3;
    // The int8 routine reads 8 bytes per lane and row: with rows an odd number
    // of 16-byte steps apart, the four rows of a half-warp must be two steps
    // apart to cover all banks, so lanes g = 0..3 take rows 0, 2, 4, 6 of the
    // eight and g = 4..7 rows 1, 3, 5, 7.
    const int grow = (FMT == Q4K_I8 || FMT == Q8_I8) ? ((L.g & 3) * 2 + (L.g >> 2)) : (L.g >> 1) + (L.g & 1) * 4;
    constexpr bool ONE = NT == 0, PACKED = NT <= 1;
    const I8Cols X = i8_cols<PACKED ? 1 : NT>(a.ncols, a.n_tokens);

    uint32_t it = 0;
    int tile_parity = 0;
    bool out_ready = false;
    if (a.x_resident && (int)blockIdx.x < a.n_tiles) mbar_wait(xbar, 0, a.status, 0x4u);
    const int n_mats = a.up_quants ? 2 : 1;
    float gate[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // SwiGLU in one launch: the gate's sums of this lane, kept until up's arrive
    for (int tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x)
    for (int mat = 0; mat < n_mats; mat++, tile_parity ^= 1) {
        float acc[NACC];
#pragma unroll
        for (int i = 0; i < NACC; i++) acc[i] = 0.0f;

        for (int ch = 0; ch < n_chunks; ch++, it++) {
            const int s = it % S;
            const uint32_t ph = (it / S) & 1;
            mbar_wait(full0 + 8 * s, ph, a.status, 0x2u);
            const int u0 = ch * a.kc, kcc = min(a.kc, a.units - u0);
            const uint32_t st = stage0 + s * a.stage_bytes;
            L.row_a = st + (rt * 16 + grow) * a.q_stride;
            L.row_b = L.row_a + 8 * a.q_stride;
            L.srow_a = st + a.s_off + (rt * 16 + grow) * a.s_stride;
            L.srow_b = L.srow_a + 8 * a.s_stride;
            if (BASE == Q8_0) {
                L.unit = a.boxed ? 2 * R * 128 : 256;
                L.half = a.boxed ? R * 128 : 128;
                L.byte0 = a.boxed ? (((L.c >> 1) ^ (grow & 7)) << 4) | (L.c & 1) << 3 : 8 * L.c;
            }
            L.xbase = a.x_resident ? smem_u32(xres) : st + a.x_off;
            const int xu0 = a.x_resident ? u0 : 0;
            // units are dealt to the K-split warps round-robin over the whole row,
            // so every warp gets the same number whatever the chunking
            for (int ul = (ks + KS - u0 % KS) % KS; ul < kcc; ul += KS) {
                if constexpr (FMT == Q4K_I8) unit_q4k_i8<NT>(L, X, ul, xu0 + ul, acc);
                else if constexpr (FMT == Q8_I8) unit_q8_i8<NT>(L, X, ul, xu0 + ul, acc);
                else unit_q6k_i8<ONE ? 1 : NT, ONE>(L, X, ul, xu0 + ul, (a.whole_rows || a.boxed ? u0 : (u0 & 7)) + ul, acc);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + 8 * s);
        }

        // ---- sum the K-split warps of this row tile, in warp order ----
        if (KS > 1) {
            float *buf = red + tile_parity * (KS * RT * NACC * 32);
#pragma unroll
            for (int i = 0; i < NACC; i++) buf[((ks * RT + rt) * NACC + i) * 32 + lane] = acc[i];
            asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory");
            if (ks != 0) continue;
#pragma unroll
            for (int i = 0; i < NACC; i++) {
                float v = 0.0f;
#pragma unroll
                for (int k2 = 0; k2 < KS; k2++) v += buf[((k2 * RT + rt) * NACC + i) * 32 + lane];
                acc[i] = v;
            }
        }

        if (!out_ready) {   // the kernel ahead may still be writing `out` or `aux`
            griddep_wait();
            out_ready = true;
        }
        // ---- epilogue: lane (g, c) holds rows g, g+8 and columns 2c, 2c+1 of each group ----
        const size_t r0 = (size_t)tile * R + rt * 16 + grow, r1 = r0 + 8;
        if constexpr (PACKED) {
            // a token's four planes are columns 4t..4t+3: lanes c = 2t, 2t+1 (ONE: both halves are token 0's)
            float va = acc[0] + acc[1], vb = acc[2] + acc[3];
            va += __shfl_xor_sync(0xffffffffu, va, 1);
            vb += __shfl_xor_sync(0xffffffffu, vb, 1);
            if (ONE) {
                va += __shfl_xor_sync(0xffffffffu, va, 2);
                vb += __shfl_xor_sync(0xffffffffu, vb, 2);
            }
            const int t = L.c >> 1;
            if (n_mats == 2 && mat == 0) {
                gate[0] = va;
                gate[2] = vb;
            } else if (!(L.c & 1) && t < a.n_tokens) {
                emit(a, t0 + t, r0, n_mats == 2 ? silu_mul(gate[0], va) : va);
                emit(a, t0 + t, r1, n_mats == 2 ? silu_mul(gate[2], vb) : vb);
            }
        } else if constexpr (NT == 2) {
            // Lane c of a row's four finishes tokens c and c + 4: their planes' columns are p*n + t; a tile's
            // column i is in lane i >> 1, the even or odd one of its pair.
            float v[4];
#pragma unroll
            for (int s = 0; s < 2; s++) {
                const int t = L.c + 4 * s;
                v[s] = v[2 + s] = 0.0f;
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    const int col = t < a.n_tokens ? p * a.n_tokens + t : 0, i2 = col < 8 ? col : col - X.tile_stride;
                    const int from = (lane & ~3) | (i2 >> 1);
                    float x[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) x[i] = __shfl_sync(0xffffffffu, acc[i], from);
                    const float ra = col < 8 ? ((i2 & 1) ? x[1] : x[0]) : ((i2 & 1) ? x[5] : x[4]);
                    const float rb = col < 8 ? ((i2 & 1) ? x[3] : x[2]) : ((i2 & 1) ? x[7] : x[6]);
                    v[s] += ra;
                    v[2 + s] += rb;
                }
            }
            if (n_mats == 2 && mat == 0) {
#pragma unroll
                for (int i = 0; i < 4; i++) gate[i] = v[i];
            } else {
#pragma unroll
                for (int s = 0; s < 2; s++) {
                    const int t = L.c + 4 * s;
                    if (t < a.n_tokens) {
                        emit(a, t0 + t, r0, n_mats == 2 ? silu_mul(gate[s], v[s]) : v[s]);
                        emit(a, t0 + t, r1, n_mats == 2 ? silu_mul(gate[2 + s], v[2 + s]) : v[2 + s]);
                    }
                }
            }
        } else {
            // a tile per plane, summed by the unit routine: this lane holds tokens 2c and 2c+1 of its two rows
            if (n_mats == 2 && mat == 0) {
#pragma unroll
                for (int i = 0; i < 4; i++) gate[i] = acc[i];
            } else {
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int t = 2 * L.c + i;
                    if (t < a.n_tokens) {
                        emit(a, t0 + t, r0, n_mats == 2 ? silu_mul(gate[i], acc[i]) : acc[i]);
                        emit(a, t0 + t, r1, n_mats == 2 ? silu_mul(gate[2 + i], acc[2 + i]) : acc[2 + i]);
                    }
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// A CTA's shared memory (one CTA per SM): barriers, the K-split warps' sums, then resident planes and stages.
template <int FMT, int NT, int RT, int KS> struct Smem {
    static constexpr int LIMIT = 227 * 1024;
    static constexpr int FIXED = 256 + (KS > 1 ? 2 * KS * RT * (NT == 2 ? 8 : 4) * 32 * 4 : 0);
    static constexpr int ALIGN = base_of(FMT) == Q8_0 ? 1024 : 128;     // the stages' start is rounded up
    static constexpr int BUDGET = LIMIT - FIXED - (ALIGN - 128);
    static int pad(int b) { return (b + ALIGN - 1) & ~(ALIGN - 1); }
    // bytes of a stage of whole rows without planes
    static int whole(const GemvArgs &a) { return (int)(16 * RT * (a.w.qpitch + a.w.srow * 2)); }
    // the planes and two stages of whole rows
    static bool two_whole_fit(const GemvArgs &a) { return pad(a.units * a.xunit) + 2 * pad(whole(a)) <= BUDGET; }
};

template <int FMT, int NT, int RT, int KS>
static int launch(dwim_b200_ctx *ctx, GemvArgs &a) {
    constexpr int R = RT * 16;
    constexpr int UNIT_Q = Traits<FMT>::UNIT_Q;
    constexpr int BASE = base_of(FMT);
    using S = Smem<FMT, NT, RT, KS>;
    // K per stage.  Whole rows when two stages of them fit: the tile is then one contiguous run of
    // HBM and moves with a single bulk copy (issuing a bulk copy costs the producer on the order of a
    // hundred cycles, so a stage made of one copy per row starves the consumers).  Longer rows are cut
    // in even chunks, a box of a tensor map each: the stage's rows then lie the chunk's units apart,
    // an odd number of 16-byte steps for an odd number of units.  The digit planes stay resident in
    // shared memory when they are small next to the ring or when enough stages fit beside them: those of
    // eight tokens of a 5120-wide row are 132 KB, beside which two whole rows' stages do not fit and
    // three boxes of seven units do (planes that travel with the stages are twice the weights' bytes:
    // the [151936, 5120] head by eight tokens 350 us so, 287 in boxes).
    auto pad = [](int b) { return S::pad(b); };
    const int xall = a.units * a.xunit, srow_bytes = (int)a.w.srow * 2;
    const int whole = S::whole(a);
    // odd: a box of 256 elements of 8 bytes; Q8_0: a lane for each half unit and one for the scales
    constexpr int MAX_BOX = BASE == Q8_0 ? 15 : (2048 / UNIT_Q - 1) / 2 * 2 + 1;
    auto box_units = [&](int chunks) { return ((a.units + chunks - 1) / chunks) | 1; };
    a.x_resident = xall <= 80 * 1024 || S::two_whole_fit(a);
    a.whole_rows = 2 * pad(whole + (a.x_resident ? 0 : xall)) <= S::BUDGET - (a.x_resident ? pad(xall) : 0);
    a.boxed = 0;
    // scale bytes of a row in a box's stage: Q8_0's own box, Q6_K's whole row
    auto box_scales = [&](int kc) { return BASE == Q8_0 ? kc * 16 : srow_bytes; };
    if (!(a.whole_rows && a.x_resident)) {
        // the fewest chunks that a box takes and of which three stages fit (two where planes travel with them)
        for (int pass = 0; pass < 2 && !a.boxed; pass++) {
            const int resident = pass == 0, want = resident ? 3 : 2;
            if (resident && pad(xall) + 3 * pad(R * (UNIT_Q + box_scales(1))) > S::BUDGET) continue;
            for (int chunks = (a.units + MAX_BOX - 1) / MAX_BOX; chunks <= a.units; chunks++) {
                const int kc = box_units(chunks);
                if (kc > MAX_BOX) continue;
                const int bytes = pad(R * (kc * UNIT_Q + box_scales(kc)) + (resident ? 0 : kc * a.xunit));
                if (want * bytes > S::BUDGET - (resident ? pad(xall) : 0)) {
                    if (kc == 1) break;
                    continue;
                }
                if (resident && kc < 3) break;       // too little a copy: rather the planes with the stages
                a.boxed = 1;
                a.whole_rows = 0;
                a.x_resident = resident;
                a.kc = kc;
                a.q_stride = BASE == Q8_0 ? 128 : kc * UNIT_Q;
                a.s_off = R * kc * UNIT_Q;
                a.s_stride = box_scales(kc);
                a.x_off = a.s_off + R * a.s_stride;
                a.stage_bytes = bytes;
                break;
            }
        }
    }
    a.xres_bytes = a.x_resident ? xall : 0;
    const int budget = S::BUDGET - pad(a.xres_bytes);
    if (a.boxed) {
        a.stages = budget / a.stage_bytes;
    } else if (a.whole_rows) {
        a.kc = a.units;
        a.q_stride = (int)a.w.qpitch;
        a.s_off = R * a.q_stride;
        a.s_stride = srow_bytes;
        a.x_off = a.s_off + R * a.s_stride;
        a.stage_bytes = pad(whole + (a.x_resident ? 0 : xall));
        a.stages = budget / a.stage_bytes;
    } else {
        int chunks = 2;
        for (;; chunks++) {
            a.kc = (a.units + chunks - 1) / chunks;
            int qs = UNIT_Q * a.kc;
            if ((qs / 16) % 2 == 0) qs += 16;   // an odd number of 16-byte steps between rows: no bank conflicts
            a.q_stride = qs;
            a.s_off = R * qs;
            a.s_stride = BASE == Q8_0 ? 16 * a.kc + 16 : BASE == Q6_K ? ((2 * (a.kc + 14) + 15) & ~15) + 16 : 0;
            a.x_off = a.s_off + R * a.s_stride;
            a.stage_bytes = pad(a.x_off + (a.x_resident ? 0 : a.kc * a.xunit));
            a.stages = budget / a.stage_bytes;
            if (a.stages >= 2 || a.kc == 1) break;
        }
    }
    if (a.stages > MAX_STAGES) a.stages = MAX_STAGES;
    if (a.stages < 2) return fail(ctx, DWIM_B200_EINVAL, "small-M kernel: a stage of %d bytes does not fit", a.stage_bytes);
    a.n_tiles = (int)((a.w.rows + R - 1) / R);
    const int smem = S::LIMIT - S::BUDGET + pad(a.xres_bytes) + a.stages * a.stage_bytes;
    auto kern = dwim_smallm_kernel<FMT, NT, RT, KS>;
    static std::atomic<bool> configured[64] = {};   // per instantiation, per device; contexts of several threads share it
    if (!configured[ctx->device & 63]) {
        DWIM_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::LIMIT));
        configured[ctx->device & 63] = true;
    }
    int grid = a.n_tiles < ctx->sm_count ? a.n_tiles : ctx->sm_count;
    const int nwarps = RT * KS + 1;
    BoxMaps maps = {};
    for (int i = 0; i < (a.boxed ? a.up_quants ? 2 : 1 : 0); i++) {
        const uint8_t *q = i ? a.up_quants : a.w.quants;
        int rc;
        if (BASE == Q8_0) {
            rc = encode_2d(ctx, &maps.q[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, q, a.w.qpitch, a.w.rows, a.w.qpitch, 128, R, CU_TENSOR_MAP_SWIZZLE_128B,
                           "weight");
            if (!rc)
                rc = encode_2d(ctx, &maps.s[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, i ? a.up_scales : a.w.scales, a.w.srow, a.w.rows, a.w.srow * 2,
                               (uint32_t)(a.kc * 8), R, CU_TENSOR_MAP_SWIZZLE_NONE, "scale");
        } else {
            rc = encode_2d(ctx, &maps.q[i], CU_TENSOR_MAP_DATA_TYPE_INT64, q, a.w.qpitch / 8, a.w.rows, a.w.qpitch, (uint32_t)(a.kc * UNIT_Q / 8), R,
                           CU_TENSOR_MAP_SWIZZLE_NONE, "weight");
        }
        if (rc) return rc;
    }
    const bool dependent = !ctx->weights_written;   // see dwim_b200_ctx::weights_written
    ctx->weights_written = false;
    DWIM_CUDA(ctx, launch_dependent(dependent, kern, dim3((unsigned)grid, (unsigned)a.groups), dim3((unsigned)(nwarps * 32)), (size_t)smem, ctx->stream, a,
                                    maps));
    DWIM_LAUNCHED(ctx);
    return 0;
}

template <int FMT, int NT>
static int launch_shape(dwim_b200_ctx *ctx, GemvArgs &a) {
    // Row tiles per CTA (RT) x K-split warps per row tile (KS).  A CTA's tiles last rounds * (RT + c) in times of 16
    // rows: every round has its reduction, epilogue and, where the planes travel with the stages, one load of all planes,
    // which weigh the more the shorter the rows are; wide tiles save rounds, narrow ones fill the last.  c * cols was
    // fitted to these and others, us for RT = 1, 2, 3, 4:
    //   Q4_K, one token: [17408, 5120] 15.7 13.4 12.6 12.5, [10240, 5120] 11.1 10.4 8.8 10.2, [6144, 5120] 7.5 7.0 6.8
    //   7.2, [5120, 6144] 7.3 7.9 7.2 8.3, [1024, 5120] 3.4 4.2 5.1 5.8, [5120, 17408] 15.7 19.5 14.6 16.7; five tokens
    //   [17408, 5120] 22.5 19.2 18.6 18.4, [10240, 5120] 14.9 14.0 13.3 16.9, [5120, 17408] 24.6 24.0 16.8 21.5
    //   Q6_K: the [151936, 5120] head by one 107 99 101, by two 125 112 112, by five 251 171 167 147, by eight 234 211 186
    //   168; [12288, 5120] by one 12.4 12.3 11.5, by five 22.9 18.4 18.5 19.4
    //   Q8_0: [17408, 2048] by one 12.6 9.5 9.4 8.8, by eight 16.5 11.8 13.8 11.9; [5120, 5120] by eight 14.3 14.7 10.3
    // (with c = 0.3 throughout, [10240, 5120] took one row tile and [17408, 2048] whole rows of one).  Four K-split warps
    // leave a thread more registers than five: Q4_K by one token with three row tiles [10240, 5120] 9.3 us with five,
    // 8.8 with four, by five [5120, 6144] 10.8 and 9.5; two row tiles 20.1 and 19.2.  Q6_K and Q8_0 by three tokens and
    // more are a percent better with five.  Q8_0 by one or two tokens: whole rows of one row tile, where those of two do
    // not fit, beat its boxes, two swizzled ones a unit, unless the boxes take a single round ([12288, 5120] 13.0 and 14.0;
    // [5120, 5120] 7.5 and 8.5 one product behind the other, but 10.1 and 9.4 with the conversion before each).
    // Rows beyond 65536 columns keep one row tile: the stage with the fewest units is the narrowest then.
    constexpr bool FEW = NT <= 1;
    constexpr int MOST = FMT == Q4K_I8 || (FMT == Q6K_I8 && !FEW) ? 4 : 3;
    constexpr int KS3 = FMT == Q4K_I8 || FEW ? 4 : 5, KS4 = FMT == Q4K_I8 ? 4 : 3;
    int rt = 1;
    if (a.w.cols <= 65536) {
        const bool whole = FMT == Q8_I8 && FEW && Smem<FMT, NT, 1, 8>::two_whole_fit(a) && !Smem<FMT, NT, 2, 4>::two_whole_fit(a);
        const double c = (FMT == Q4K_I8 ? 4300.0 : FMT == Q8_I8 ? 1900.0 : FEW ? 1540.0 : 2560.0) / (double)a.w.cols;
        double best = 0;
        for (int t = 1; t <= MOST; t++) {
            const size_t tiles = (a.w.rows + 16 * t - 1) / (16 * t);
            const size_t rounds = (tiles + ctx->sm_count - 1) / ctx->sm_count;
            const double cost = (double)rounds * (t + c);
            if (t == 1 || (cost < best && !(whole && rounds > 1))) {
                best = cost;
                rt = t;
            }
        }
    }
    if (rt == 2) return launch<FMT, NT, 2, 4>(ctx, a);
    if (rt == 3) return launch<FMT, NT, 3, KS3>(ctx, a);
    if constexpr (MOST == 4)
        if (rt == 4) return launch<FMT, NT, 4, KS4>(ctx, a);
    return launch<FMT, NT, 1, 8>(ctx, a);
}

// Whether the small-M kernel takes a product of n tokens: up to eight tokens of
// any format (Q8_0 rows need not be whole 256-weight units: their scale rows are
// padded with zeros).
bool gemv_takes_i8(const WeightView &w, size_t n) {
    if (n < 1 || n > I8_MAX_TOKENS) return false;
    return w.fmt == Q8_0 || ((w.fmt == Q4_K || w.fmt == Q6_K) && w.cols % 256 == 0);
}

// Up to eight tokens through the int8 routines; `panels` from build_panels_i8.
// `up`, when given, makes it the SwiGLU of the pair (w = gate) in one launch.
int gemv_small_i8(dwim_b200_ctx *ctx, const WeightView &w, const uint8_t *panels, int n_tokens, size_t t0, const OutSpec &out,
                  const float *aux, int epilogue, const WeightView *up, size_t groups) {
    if (w.rows == 0 || n_tokens == 0) return 0;
    if (!gemv_takes_i8(w, (size_t)n_tokens))
        return fail(ctx, DWIM_B200_EINVAL, "int8 small-M kernel: format %d, %d tokens", w.fmt, n_tokens);
    GemvArgs a{};
    a.w = w;
    a.panels = panels;
    a.ncols = i8_planes(n_tokens) * n_tokens;
    a.n_tokens = n_tokens;
    a.t0 = t0;
    a.out = out;
    a.aux = aux;
    a.epi = epilogue;
    a.units = (int)((w.cols + 255) / 256);
    a.xunit = a.xsrc_stride = i8_unit_bytes(a.ncols);
    a.group_panels = (size_t)a.units * a.xunit;
    a.groups = (int)groups;
    if (up) {
        if (up->fmt != w.fmt || up->rows != w.rows || up->cols != w.cols || up->qpitch != w.qpitch || epilogue != EPI_STORE)
            return fail(ctx, DWIM_B200_EINVAL, "int8 small-M kernel: gate and up differ");
        a.up_quants = up->quants;
        a.up_scales = up->scales;
    }
    a.status = ctx->status;
    const int tiles = i8_tiles(n_tokens);
    switch (w.fmt) {
    case Q4_K: return tiles == 1 ? launch_shape<Q4K_I8, 1>(ctx, a) : tiles == 2 ? launch_shape<Q4K_I8, 2>(ctx, a) : launch_shape<Q4K_I8, 3>(ctx, a);
    case Q8_0: return tiles == 1 ? launch_shape<Q8_I8, 1>(ctx, a) : tiles == 2 ? launch_shape<Q8_I8, 2>(ctx, a) : launch_shape<Q8_I8, 3>(ctx, a);
    case Q6_K:
        return n_tokens == 1 ? launch_shape<Q6K_I8, 0>(ctx, a)
               : tiles == 1  ? launch_shape<Q6K_I8, 1>(ctx, a)
               : tiles == 2  ? launch_shape<Q6K_I8, 2>(ctx, a)
                             : launch_shape<Q6K_I8, 3>(ctx, a);
    default: return fail(ctx, DWIM_B200_EFORMAT, "unknown weight format %d", w.fmt);
    }
}

}  // namespace dwim
