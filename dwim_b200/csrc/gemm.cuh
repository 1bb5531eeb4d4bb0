// What the tensor-core kernels share (gemm.cu, gemm_few.cu): tile and role constants, the MMA's wrappers, where
// results go, Q4_K's decoding, and how many blocks share a tile.
#pragma once
#include <cuda.h>
#include <stdlib.h>

#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"
#include "tc.cuh"
#include "tmap.cuh"

namespace dwim {

constexpr int TILE_M = 128;   // weight rows per CTA
constexpr int BK = 64;        // K per stage: one 128-byte swizzled row of f16
constexpr int KBLOCKS = 4;    // K blocks per unit; each is a stage of the A ring and a hand-over of its own
constexpr int SCALE_SLOTS = 4;
constexpr int N_WORKERS = 16;                                      // warps 0..15: four per TMEM lane quadrant
constexpr int X_WARP = 16, MMA_WARP = 17, RAW_WARP = 18;           // the activations' producer, the issuer, the weights' producer
constexpr int GEMM_THREADS = 640;                                  // whole warpgroups (one warp has no role)
// A thread's registers are 96 at launch (65536 / 640, whole eights); the four warps without sums give some of theirs to
// the workers.  The dense kernel's workers take all there are ([12288, 5120] Q6_K by 512 f32 tokens 213 us with the
// Q4_K kernel's shares, 208 with these); the Q4_K kernel's issuer wants more than 32 (375 and 387 us).
constexpr int WORKER_REGS = 104, OTHER_REGS = 56, DENSE_WORKER_REGS = 112, DENSE_OTHER_REGS = 32;
static_assert(512 * WORKER_REGS + 128 * OTHER_REGS <= 640 * 96 && 512 * DENSE_WORKER_REGS + 128 * DENSE_OTHER_REGS <= 640 * 96,
              "a warpgroup would wait for registers that nobody gives up");
constexpr int RAW_BYTES = ((TILE_M * 144 + 1023) / 1024) * 1024;   // 18 KB
constexpr int A_BYTES = TILE_M * BK * 2;                           // 16 KB
constexpr int AMIN_BYTES = TILE_M * 16 * 4;                        // 8 KB: [K group of 8][row][16 B], four groups
constexpr int MAX_SMEM = 227 * 1024;
constexpr int BAR_BYTES = 1024;
constexpr int MAX_SPLIT = 8;                                       // blocks of a portable cluster

// ---- tcgen05 wrappers -----------------------------------------------------------
// D[tmem] (+)= A[smem desc] * B[smem desc]; f16 inputs, f32 accumulate.
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same with the descriptors given as (low word, shared high word) and the
// accumulate flag fixed at compile time: the issuing thread has about one
// instruction slot per five cycles, so every instruction between two MMAs counts.
template <int ACC>
__device__ __forceinline__ void umma_f16_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "n"(ACC)
        : "memory");
}
__device__ __forceinline__ void umma_f16_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"((uint32_t)acc)
        : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y) {
    asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void sts32f(uint32_t a, float x) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(x) : "memory"); }
__device__ __forceinline__ float lds32f(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
// Two floats rounded to f16, `lo` in the low half.
__device__ __forceinline__ uint32_t f16x2_rn(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ float silu_mul_f(float g, float u) { return g * (1.0f / (1.0f + expf(-g))) * u; }

// Where a thread's results go: its row of one destination; or (SHARED kernels) of every rank's
// copy of a shared result; or (a K-sharded product's partial sums) of its owner's slot alone.
// The pointers are read from the kernel's parameters by constant index, once, ahead of the
// stores' loop: indexing the parameter array by a variable, or reading a parameter after every
// store, cost the 256-column kernel half its speed.  The many-destination stores live in kernel
// instantiations of their own, so that the usual kernel's code stays small (an epilogue with
// eight predicated stores per value stalled the main loop on instruction fetch).
struct EmitTo {
    float *own;              // the first (or only) destination's element (token 0, this thread's row)
    size_t offset;           // the same element's offset in every other destination
    size_t pitch;
    const float *aux_row;
    const OutSpec *out;
    int world, epi;
};
__device__ __forceinline__ EmitTo emit_to(const OutSpec &out, const float *aux, int epi, size_t row) {
    EmitTo e;
    float *d = out.dst[0];
    e.offset = out.row0 + row;
    if (out.scatter_per) {
        // the row's owner alone, its slot for this rank; the owner is picked by constant indices
        const size_t owner = row / out.scatter_per;
        e.offset = out.row0 + row - owner * out.scatter_per;
#pragma unroll
        for (int p = 1; p < DWIM_MAX_WORLD; p++)
            if ((size_t)p == owner) d = out.dst[p];
    }
    e.own = d + e.offset;
    e.pitch = out.pitch;
    e.aux_row = aux ? aux + row : nullptr;
    e.out = &out;
    e.world = out.scatter_per ? 1 : out.world;
    e.epi = epi;
    return e;
}
constexpr uint32_t H2_1024 = 0x64006400u, H2_M1024 = 0xE400E400u, H2_64 = 0x54005400u, H2_M64 = 0xD400D400u;

// ---- dequantizer: the 64 weights of one row and K block as exact sc*q halves ----------
// K block g (0..3 inside the unit) is group g of the block's quants: 32 bytes
// whose low nibbles are sub-block 2g (k = 0..31 of the K block) and high
// nibbles sub-block 2g+1 (k = 32..63).  A word's bytes come out in the order
// (0, 2, 1, 3); the activations are stored in the same order.
// A row's unit is drained as s * S, with S the one accumulator both operands
// add into, and s = d * 2^e.  The main operand is sc*q*2^-e (still exact in
// f16, subnormals included, for e <= 24) and the minimums enter as
// -(32*dmin/s)*m_j.  e = 0 unless dmin is more than ~32 times d: it is chosen
// from the two exponents so that 63 * 32*dmin/s stays below f16's maximum.
// When d is zero, or e would pass 24 (the sc*q term is then below 2^-19 of the
// other), s = 32*dmin, the main operand is zero and the minimums enter as -m_j.
struct Q4kFold {
    int e;        // the main operand is scaled by 2^-e
    bool zero;    // the main operand is dropped
};
template <bool CENTRED = false>
__device__ __forceinline__ Q4kFold q4k_fold(uint32_t d_dmin) {
    const float d = h2f_lo(d_dmin), dmin = h2f_hi(d_dmin);
    const int ed = (int)((__float_as_uint(d) >> 23) & 0xffu), em = (int)((__float_as_uint(dmin) >> 23) & 0xffu);
    Q4kFold f;
    // (centred, and where d and dmin differ in sign, the minimums' two parts add up: twice the room)
    if (CENTRED) f.e = max(0, em - ed - 4 + (int)((d_dmin ^ (d_dmin << 16)) >> 31));
    else f.e = max(0, em - ed - 4);
    f.zero = d == 0.0f || f.e > 24;
    if (f.zero) f.e = 0;
    return f;
}

struct Q4kBlock {
    uint32_t words[8];                 // the 32 bytes of group g
    uint32_t mul[2], add[2];           // per nibble half: x*mul + add turns the magic-number halves into sc*q
};
__device__ __forceinline__ void load_q4k_block(const uint4 &hdr, uint32_t raw_row, int g, Q4kBlock &b) {
    const uint4 q0 = lds128(raw_row + 16 + 32 * g), q1 = lds128(raw_row + 32 + 32 * g);
    b.words[0] = q0.x; b.words[1] = q0.y; b.words[2] = q0.z; b.words[3] = q0.w;
    b.words[4] = q1.x; b.words[5] = q1.y; b.words[6] = q1.z; b.words[7] = q1.w;
    const int sh = (g & 1) * 16;
    const uint32_t y = (hdr.y >> sh) & 0xffffu, w = (hdr.w >> sh) & 0xffffu;
    const uint32_t sc2 = g < 2 ? (y & 0x3f3fu) : ((w & 0x0f0fu) | ((y >> 2) & 0x3030u));
    const uint32_t sa = sc2 & 0xffu, sb = sc2 >> 8;
    const Q4kFold f = q4k_fold(hdr.x);      // (passed in instead, the 256-column form spills 96 bytes, 32 like this)
    // 2^-e as a half: normal down to 2^-14, subnormal below; zero drops the operand
    const uint32_t p1 = f.zero ? 0u : (f.e <= 14 ? (uint32_t)(15 - f.e) << 10 : 1u << (24 - f.e));
    const uint32_t p2 = p1 | (p1 << 16);
    const uint32_t spa = hmul2(hsub2(0x64006400u | sa | (sa << 16), H2_1024), p2);   // half2 of sc_2g * 2^-e
    const uint32_t spb = hmul2(hsub2(0x64006400u | sb | (sb << 16), H2_1024), p2);   // half2 of sc_2g+1 * 2^-e
    // low nibbles: (1024 + q)*sc - 1024*sc; high nibbles: (64 + q)*sc - 64*sc
    b.mul[0] = spa; b.add[0] = hmul2(spa, H2_M1024);
    b.mul[1] = spb; b.add[1] = hmul2(spb, H2_M64);
}
// Four of the row's eight 6-bit minimums (m_0..m_3 for part 0, m_4..m_7 for
// part 1), each times f, as two f16 terms (value and rounding remainder):
// b[t] holds term t of the four values, two per word.
__device__ __forceinline__ void mins_q4k_terms(const uint4 &hdr, int part, float f, uint32_t (&b)[2][2]) {
    const uint32_t m4 = part ? (((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u)) : (hdr.z & 0x3f3f3f3fu);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        // byte -> float through the 2^23 magic number
        const float p0 = (__uint_as_float(prmt(m4, 0x4B000000u, 0x7650 + 2 * i)) - 8388608.0f) * f;
        const float p1 = (__uint_as_float(prmt(m4, 0x4B000000u, 0x7651 + 2 * i)) - 8388608.0f) * f;
        const uint32_t hi = f16x2_rn(p0, p1);
        b[0][i] = hi;
        b[1][i] = f16x2_rn(p0 - h2f_lo(hi), p1 - h2f_hi(hi));
    }
}

// Blocks that share a tile's K.  A block is alone on its SM, so tiles run in waves of as many
// clusters as the device holds; a wave lasts a block's units and what a tile costs besides, in units:
// three for ramp and epilogue, six and a half with the exchange (fitted to every split from 1 to 8 of
// six shapes by 48 to 2048 tokens; the choice is within 3 % of the best of them but for [1024, 5120] by
// 2048).  Without it 40 tiles left 108 of 148 SMs idle: [5120, 17408] by 131 bf16 tokens 134 us, 67 with three
// blocks a tile; by 512 f32 tokens (160 tiles) 299 and 236.  The few-token kernel's use of it: gemm_few.cu.
// The dense kernel's units are twice as long, so a tile's other costs are fewer of them: two, and four and
// a half with the exchange.  Over every split of twelve products (rows 1024 to 17408, K 5120 and 12288, 80 to 2048
// tokens) the choice is within 3 % of the best, but for [5120, 5120] by 131 f32 tokens (63.6 us alone, 60.4 by three).
struct SplitCost {
    double tile, shared;      // what a tile costs besides its units: alone, shared
};
// known: clusters of so many blocks that a device holds at once (0: not asked yet); contexts of several threads share it.
template <typename Kernel, typename Fits>
int pick_split(dwim_b200_ctx *ctx, Kernel kern, int threads, size_t smem, Fits fits, SplitCost cost,
               std::atomic<int> (&known)[64][MAX_SPLIT + 1], long tiles, int units, double unit, double *time = nullptr) {
    int best = 1;
    double t_best = 0;
    for (int s = 1; s <= MAX_SPLIT && s <= units; s++) {
        if (!fits(s)) continue;
        int k = known[ctx->device & 63][s];
        if (!k) {
            int n = ctx->sm_count;
            if (s > 1) {
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3((unsigned)(ctx->sm_count / s * s));
                cfg.blockDim = dim3((unsigned)threads);
                cfg.dynamicSmemBytes = smem;
                cudaLaunchAttribute at;
                at.id = cudaLaunchAttributeClusterDimension;
                at.val.clusterDim.x = (unsigned)s;
                at.val.clusterDim.y = at.val.clusterDim.z = 1;
                cfg.attrs = &at;
                cfg.numAttrs = 1;
                cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
                    cudaGetLastError();
                    n = 1;
                }
            }
            known[ctx->device & 63][s] = k = n;
        }
        const double t = (double)((tiles + k - 1) / k) * ((units + s - 1) / s * unit + (s > 1 ? cost.shared : cost.tile));
        if (s == 1 || t < 0.97 * t_best) {
            t_best = t;
            best = s;
        }
    }
    if (time) *time = t_best;
    return best;
}

// Once per kernel and device: its shared memory, and that it was compiled to be launched with the registers that its
// warpgroups trade (a warpgroup waits for its share without a limit).
template <typename Kernel>
int configure_gemm(dwim_b200_ctx *ctx, Kernel kern, int smem, int threads, int shares, std::atomic<bool> &done) {
    if (done) return 0;
    cudaFuncAttributes at;
    DWIM_CUDA(ctx, cudaFuncGetAttributes(&at, kern));
    if (at.numRegs * threads < shares)
        return fail(ctx, DWIM_B200_ECUDA, "a kernel of %d registers a thread cannot give its warpgroups their shares", at.numRegs);
    DWIM_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    done = true;
    return 0;
}

// Up to 32 tokens of Q4_K for one destination (gemm_few.cu).
int gemm_few(dwim_b200_ctx *ctx, const WeightView &w, const __half *operand, size_t n, int terms, const OutSpec &out, const float *aux,
             int epi);

}  // namespace dwim
