// The large-M product (prefill, long verify batches) for Q4_K: a dense
// contraction on the 5th-generation tensor cores whose weight products are
// exact.  Replaces the reference's matmul_tile64_* kernels
// (matmul_tile.cu:94-258; host side gpu/cuda/mod.rs:402-442).
//
// out[t][r] = sum_k W[r][k] x[t][k], with W[r][k] = d*(sc_j*q) - dmin*m_j
// (d, dmin per 256-weight unit and row; sc_j, m_j per 32-weight sub-block).
// The integer sc_j*q <= 945 is exact in f16, so for every unit u of K
//     S_u[r][t] = sum_k (sc*q)[r][k] * x[t][k]                    16 MMAs of K=16
//               - sum_j (32*dmin/d * m_j)[r] * mean_j(x[t])         2 MMAs of K=16
// is accumulated in the tensor cores' fp32 accumulators and
//     out[r][t] = sum_u d_u[r] * S_u[r][t]
// is applied by CUDA cores in fp32.  The first sum's products are exact; the
// second's factors travel as f16 value + rounding remainder on both sides (22
// bits each), and a power of two moves between d and the operands when dmin/d
// is large (q4k_fold, gemm.cuh).  The reference's tile kernel rounds every
// dequantized weight to f16 instead (matmul_tile.cu:66-74): 2e-4 of rms error
// against 5e-7 here.  An f32 activation travels as two f16 terms, value and
// rounding remainder; a bf16 one is exact in one.  The terms share a token's
// decoded weights and its minimums (whose means are of the activations
// themselves), and from 129 tokens on its accumulator.  (As two columns with
// sums, minimums and an epilogue of their own, a tile was half as many tokens:
// [17408, 5120] by 2048 f32 tokens 827 us then, 690 now.)
//
// A CTA owns 128 weight rows (one TMEM lane each) by BN columns (32..256):
//   warp 16       activations' producer (one thread): per K block of 64 the f16
//                 tile [BN][64] (TMA, 128-byte swizzle) into the B ring; per
//                 unit the sub-block means' hi and lo parts.
//   warp 17       MMA issuer: tcgen05.mma M=128 N=BN K=16 into the unit's
//                 accumulator buffer (two buffers, so unit u+1 multiplies
//                 while unit u drains).  The whole warp runs the loop and one
//                 lane issues: that thread has about one instruction slot per
//                 five cycles, and an N=128 MMA leaves it 64 cycles.
//   warps 0-15    workers.  Warp w owns TMEM lane quadrant w % 4 (weight rows
//                 32*(w % 4) + lane) and K block w / 4 of every unit:
//                 thread = row turns the block's 64 nibbles into sc*q halves
//                 (lop3 magic number + one HFMA2 per two weights) and stores
//                 them into the stage's A tile in the K-major 128-byte-
//                 swizzled layout of the MMA's descriptor; then it drains a
//                 quarter of the previous unit's columns: tcgen05.ld, acc +=
//                 d*S in registers.  K blocks 2 and 3's warps also write the
//                 unit's minimums operand and the row scales.  After the last
//                 unit: the operator's epilogue (store / add / SwiGLU),
//                 coalesced over rows.
//   warp 18       packed weights' producer (one thread): per unit the tile's
//                 blocks [128 rows][144 B] from HBM into the raw ring.
// Where the tiles do not fill the chip, a cluster's blocks share a tile's K and add up
// through each other's shared memory (pick_split).
// Warp 19 makes whole warpgroups of them, which trade registers at 256 columns: 96 a thread
// at launch, 104 for a worker then.  (At 96 the 256-column form spilled in its main loop: [17408,
// 5120] by 2048 bf16 tokens 391 us, 375 like this; with 100 bytes of spills 442.)
// Every mbarrier wait is bounded (ptx.cuh); a kernel that gave up says so in
// the context's status word.
#include "gemm.cuh"

namespace dwim {

namespace {

struct GemmArgs {
    size_t rows, n, units;          // weight rows, tokens, 256-weight units of K
    int terms;                      // f16 terms of an activation: 1, or 2 (value and rounding remainder)
    OutSpec out;
    const float *tok_scale;         // per token: the power of two its activations were divided by (prologue.cu)
    const float *aux;               // EPI_SWIGLU: the `up` product, token-major [n][rows]
    int epi;
    int split_k;                    // blocks of a cluster that share a tile's K
    uint32_t *status;
};

// The terms of an activation: one alone; up to two, the second's columns beside the first's, one MMA for both
// (while that is at most 256 columns); or two that take turns on one accumulator.
enum Mode : int { ONE_TERM, SIDE_BY_SIDE, TWO_PASSES };

// Per tile width.  Up to 192 columns of one MMA the B ring has as many stages as the A
// ring.  Up to 128 these are one and a quarter to one and a half units deep, so that the
// workers decode a unit while the one before multiplies ([17408, 5120] by 48 tokens 39.1
// with K blocks handed over in pairs, one unit deep, and 37.4 one by one like this).
// At 256 columns a decoded weight is used twice
// as often, an MMA takes 128 cycles, and shared memory is the limit: three B
// stages, two raw stages, one stage of the minimums' operands (a B stage is
// reloaded as soon as its own K block is done).
template <int BN, int MODE> struct Cfg {
    static constexpr int A_STAGES = BN <= 32 ? 6 : BN <= (MODE == SIDE_BY_SIDE ? 64 : 128) ? 5 : KBLOCKS;
    static constexpr int B_STAGES = BN > 192 || (BN == 128 && MODE == SIDE_BY_SIDE) ? 3 : A_STAGES;
    static constexpr int RAW_STAGES = BN == 32 ? 3 : 2;
    static constexpr int MIN_STAGES = BN > 128 ? 1 : 2;
    static constexpr bool WIDE = MODE == SIDE_BY_SIDE;
    // Whether the warpgroups trade registers: at 192 columns and less 96 are enough ([2090, 16896] by 571 bf16 tokens 57.0 us
    // with the trade, 55.1 without).
    static constexpr bool TRADE = BN > 192;
    static constexpr int TERM_BYTES = BN * BK * 2, B_BYTES = TERM_BYTES * (WIDE ? 2 : 1), ACC_COLS = BN * (WIDE ? 2 : 1);
    static constexpr int BMIN_BYTES = BN * 16 * 2;                 // [K group of 8][column][16 B]: the means' hi and lo parts
    static constexpr int MIN_BYTES = AMIN_BYTES + ((BMIN_BYTES + 1023) / 1024) * 1024;
    static constexpr int SCALE_BYTES = SCALE_SLOTS * TILE_M * 4;   // the unit's scale per row
    static constexpr int TOK_BYTES = BN * 4;                       // the columns' token scales, for the epilogue
    static constexpr int SMEM = BAR_BYTES + A_STAGES * A_BYTES + B_STAGES * B_BYTES + MIN_STAGES * MIN_BYTES +
                                RAW_STAGES * RAW_BYTES + SCALE_BYTES + TOK_BYTES + 1024;   // + alignment slack
    static_assert(SMEM <= MAX_SMEM, "the tile does not fit shared memory");
    static constexpr int TMEM_COLS = BN > 128 ? 512 : 2 * ACC_COLS;   // two accumulator buffers, a power of two
    static constexpr int DRAIN_COLS = BN / 4 < 16 ? 16 : BN / 4;   // accumulator columns per draining warp
    static constexpr int DRAINERS = BN / DRAIN_COLS;               // draining warps per lane quadrant (4, or 2 at BN=32)
    static constexpr int RINGS = A_STAGES * A_BYTES + B_STAGES * B_BYTES + MIN_STAGES * MIN_BYTES + RAW_STAGES * RAW_BYTES;
    // A split tile's exchange: columns that one of s blocks owns of a draining warp's, and whether the
    // blocks' sums of them fit the rings.
    static constexpr int owned(int s) { return (DRAIN_COLS / 8 + s - 1) / s * 8; }
    static constexpr bool split_fits(int s) { return s * 4 * owned(s) * TILE_M * 4 <= RINGS; }
};

// NV finished elements of a row, tokens t0 .. t0 + NV - 1: the operator's epilogue, then the
// stores.  What the epilogue reads (the residual; the `up` product) is loaded for the whole
// batch first: loads and stores taken turn by turn are one trip to L2 per element, and cost the
// [17408, 5120] product by 2048 tokens 236 us on top of 384.
template <bool SHARED, int NV>
__device__ __forceinline__ void gemm_emit(const EmitTo &e, size_t rows, size_t n, size_t t0, float (&v)[NV]) {
    float *o = e.own + t0 * e.pitch;
    if (!SHARED && e.epi != EPI_STORE) {
        const float *src = e.epi == EPI_ADD ? o : e.aux_row + t0 * rows;
        const size_t step = e.epi == EPI_ADD ? e.pitch : rows;
        float y[NV];
#pragma unroll
        for (int j = 0; j < NV; j++) y[j] = t0 + j < n ? src[j * step] : 0.0f;
        if (e.epi == EPI_ADD) {
#pragma unroll
            for (int j = 0; j < NV; j++) v[j] += y[j];
        } else {
#pragma unroll
            for (int j = 0; j < NV; j++) v[j] = silu_mul_f(v[j], y[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < NV; j++)
        if (t0 + j < n) {
            o[j * e.pitch] = v[j];
            if (SHARED) {
#pragma unroll
                for (int p = 1; p < DWIM_MAX_WORLD; p++)
                    if (p < e.world) e.out->dst[p][e.offset + (t0 + j) * e.pitch] = v[j];
            }
        }
}

// A split tile's exchange.  Eight columns at a time belong to the cluster's blocks in turn: the others' sums
// of them go into their owner's rings (whose last unit is done when the blocks have met), by rank, draining
// warp group, column and row ...
template <int COLS>
__device__ __forceinline__ void push_shares(const float (&acc)[COLS], uint32_t rings, int own, int g, int rl, int rank, int split_k) {
    cluster_sync();
#pragma unroll
    for (int q = 0; q < COLS / 8; q++) {
        if (q % split_k == rank) continue;
        const uint32_t to = cluster_addr(rings + (((rank * 4 + g) * own + q / split_k * 8) * TILE_M + rl) * 4, q % split_k);
#pragma unroll
        for (int j = 0; j < 8; j++)
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + j * TILE_M * 4), "f"(acc[8 * q + j]) : "memory");
    }
    cluster_sync();
}
// ... and the owner of columns 8q .. 8q + 7 adds its blocks' sums in rank order.
template <int COLS>
__device__ __forceinline__ void sum_shares(const float (&acc)[COLS], int q, uint32_t rings, int own, int g, int rl, int rank, int split_k,
                                           float (&v)[8]) {
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = 0.0f;
    for (int r = 0; r < split_k; r++) {
        const uint32_t from = rings + (((r * 4 + g) * own + q / split_k * 8) * TILE_M + rl) * 4;
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] += r == rank ? acc[8 * q + j] : lds32f(from + j * TILE_M * 4);
    }
}

// Writes the row's 128 bytes of the stage's A tile (K-major, 128-byte swizzle:
// 16-byte chunk c of row r sits at chunk c ^ (r & 7)).  `a_row_sw` is the row's
// address with (r & 7) << 4 or-ed in (rows are 128-byte aligned), so chunk c
// is at a_row_sw ^ (c << 4).
__device__ __forceinline__ void store_q4k_block(const Q4kBlock &b, uint32_t a_row_sw) {
#pragma unroll
    for (int c = 0; c < 4; c++) {   // words 2c, 2c+1: weights 8c .. 8c+7 of either sub-block
        const uint32_t w0 = b.words[2 * c], w1 = b.words[2 * c + 1], s0 = w0 >> 8, s1 = w1 >> 8;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            // 0x6400 | q = 1024 + q; 0x5400 | q << 4 = 64 + q (the ulp of 64.0 is 1/16)
            const uint32_t mask = h ? 0x00f000f0u : 0x000f000fu, magic = h ? H2_64 : H2_1024;
            const uint32_t o0 = hfma2(lop3_and_or(w0, mask, magic), b.mul[h], b.add[h]);   // bytes 0, 2
            const uint32_t o1 = hfma2(lop3_and_or(s0, mask, magic), b.mul[h], b.add[h]);   // bytes 1, 3
            const uint32_t o2 = hfma2(lop3_and_or(w1, mask, magic), b.mul[h], b.add[h]);
            const uint32_t o3 = hfma2(lop3_and_or(s1, mask, magic), b.mul[h], b.add[h]);
            sts128(a_row_sw ^ ((4 * h + c) << 4), o0, o1, o2, o3);
        }
    }
}

// One map per destination of a shared result, for the form of the kernel that writes it with TMA:
// this rank's rows of destination p as [tokens][rows], box [a draining warp group's tokens][128 rows].
struct OutMaps {
    CUtensorMap m[DWIM_MAX_WORLD];
};

// OUT: 0 = one destination (or a scattered one); 1 = a result shared by several ranks, every value
// stored to each copy from registers; 2 = the same through shared memory and one TMA store per
// destination and group of columns (whole 512-byte runs over NVLink instead of 4-byte stores).
template <int BN, int OUT, int MODE>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_q4k_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                const __grid_constant__ CUtensorMap tmap_m, const __grid_constant__ GemmArgs a,
                const __grid_constant__ OutMaps maps) {
    constexpr bool SHARED = OUT == 1;
    using C = Cfg<BN, MODE>;
    // One pass over a unit's K blocks: a K block's A and B stages are handed over and released together.
    constexpr int PASSES = MODE == TWO_PASSES ? 2 : 1;
    constexpr bool JOINT = PASSES == 1;
    constexpr bool TRADE = C::TRADE;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;   // the swizzled tiles want 1024-byte alignment
    // barriers, 8 bytes each
    const uint32_t afull0 = base, aempty0 = base + 64, bfull0 = base + 128, bempty0 = base + 192, minfull0 = base + 256;
    const uint32_t rawfull0 = base + 288, rawempty0 = base + 320, accfull0 = base + 352, accempty0 = base + 368;
    const uint32_t tmem_slot = base + 384;
    const uint32_t astage0 = base + BAR_BYTES;
    const uint32_t bstage0 = astage0 + C::A_STAGES * A_BYTES;
    const uint32_t min0 = bstage0 + C::B_STAGES * C::B_BYTES;
    const uint32_t raw0 = min0 + C::MIN_STAGES * C::MIN_BYTES;
    const uint32_t scale0 = raw0 + C::RAW_STAGES * RAW_BYTES;
    const uint32_t tok0 = scale0 + C::SCALE_BYTES;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split_k = OUT == 0 ? a.split_k : 1, rank = OUT == 0 ? (int)(blockIdx.x % split_k) : 0;
    const int row0 = (int)(blockIdx.x / split_k) * TILE_M, col0 = blockIdx.y * BN;
    // this block's share of K: units ub .. ub + units - 1
    const int ub = (int)a.units * rank / split_k, units = (int)a.units * (rank + 1) / split_k - ub;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::A_STAGES; s++) {
            mbar_init(afull0 + 8 * s, JOINT ? 1 + 4 : 4);   // (the producer's expect_tx arrival +) the K block's worker warps
            mbar_init(aempty0 + 8 * s, 1);               // the MMA warp's commit
        }
        for (int s = 0; s < C::B_STAGES; s++) {
            mbar_init(bfull0 + 8 * s, 1);                // the producer's expect_tx arrival
            mbar_init(bempty0 + 8 * s, 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(minfull0 + 8 * s, 1 + 8);          // the producer + the eight warps that write the minimums
            mbar_init(accfull0 + 8 * s, 1);              // also says that the unit's minimums and means have been read
            mbar_init(accempty0 + 8 * s, 4 * C::DRAINERS);
        }
        for (int s = 0; s < C::RAW_STAGES; s++) {
            mbar_init(rawfull0 + 8 * s, 1);
            mbar_init(rawempty0 + 8 * s, N_WORKERS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = lds32(tmem_slot);
    // Launched as a programmatic dependent: the next launch on the stream may begin as SMs
    // free up; here only the packed weights (written by uploads alone) are touched before
    // griddep_wait(): the activations' producer waits before its first load, the workers
    // before their first store.
    griddep_launch();

    if (warp < N_WORKERS) {
        if constexpr (TRADE) regs_inc<WORKER_REGS>();
        // ------------------------------ workers ------------------------------
        // Warp w owns TMEM lane quadrant w % 4 (weight rows 32*(w % 4) + lane)
        // and K block g = w / 4 of every unit: it decodes that block of
        // its rows into the stage's A tile, then drains column quarter g of the
        // previous unit's sums while the tensor cores work on this one.
        const int quad = warp & 3;
        const int g = warp >> 2;
        const int rl = quad * 32 + lane;                // row within the tile = TMEM lane
        static_assert(C::DRAINERS == 4 || OUT != 0, "a split tile's blocks meet in every worker");
        const bool drains = g < C::DRAINERS;
        const uint32_t drain_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + g * C::DRAIN_COLS;
        const uint32_t a_row_sw = (astage0 + rl * 128) | ((rl & 7) << 4);
        uint64_t acc2[C::DRAIN_COLS / 2];   // the row's sums, two columns per packed pair
#pragma unroll
        for (int j = 0; j < C::DRAIN_COLS / 2; j++) acc2[j] = 0ull;

        auto drain = [&](int u) {
            const int ab = u & 1;
            // the unit's sum is complete; its last MMAs waited for the minimums'
            // stage, which the row scales were written before
            mbar_wait_parked(accfull0 + 8 * ab, (u >> 1) & 1, a.status, 0x4000u);
            tc_fence_after();
            const uint32_t sc = __float_as_uint(lds32f(scale0 + ((u % SCALE_SLOTS) * TILE_M + rl) * 4));
            const uint64_t sc2 = pack2(sc, sc);
#pragma unroll
            for (int c = 0; c < C::DRAIN_COLS / 16; c++) {
                uint32_t v[16];
                tmem_ld16(drain_addr + ab * C::ACC_COLS + c * 16, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; j++) ffma2(acc2[c * 8 + j], sc2, pack2(v[2 * j], v[2 * j + 1]));
                if (C::WIDE && a.terms == 2) {      // the remainders' sums
                    tmem_ld16(drain_addr + ab * C::ACC_COLS + BN + c * 16, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; j++) ffma2(acc2[c * 8 + j], sc2, pack2(v[2 * j], v[2 * j + 1]));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(accempty0 + 8 * ab);
        };

        for (int u = 0; u < units; u++) {
            const int rs = u % C::RAW_STAGES, ms = u % C::MIN_STAGES;
            mbar_wait_parked(rawfull0 + 8 * rs, (u / C::RAW_STAGES) & 1, a.status, 0x400u);
            const uint32_t raw_row = raw0 + rs * RAW_BYTES + rl * 144;
            const uint4 hdr = lds128(raw_row);
            Q4kBlock blk;
            load_q4k_block(hdr, raw_row, g, blk);
            const int kb = KBLOCKS * u + g, stage = kb % C::A_STAGES;
            mbar_wait_parked(aempty0 + 8 * stage, ((kb / C::A_STAGES) & 1) ^ 1, a.status, 0x800u);   // the MMAs that read this stage are done
            store_q4k_block(blk, a_row_sw + stage * A_BYTES);
            fence_async_smem();          // the tensor core reads shared memory through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(afull0 + 8 * stage);
            if (g >= 2) {
                // the minimums' A operand [K group][row][16 B]: groups (hi, hi, lo, lo) of the
                // two f16 terms of -(32*dmin/s)*m_j; K block 2's warp writes m_0..m_3, K block 3's m_4..m_7
                if (u >= C::MIN_STAGES) {   // the unit that used this stage last has read its minimums
                    const int uu = u - C::MIN_STAGES;
                    mbar_wait_parked(accfull0 + 8 * (uu & 1), (uu >> 1) & 1, a.status, 0x1000u);
                }
                const Q4kFold f = q4k_fold(hdr.x);
                const float dmin32 = 32.0f * h2f_hi(hdr.x);
                const float sc = f.zero ? dmin32 : h2f_lo(hdr.x) * __uint_as_float((uint32_t)(127 + f.e) << 23);
                uint32_t b[2][2];
                mins_q4k_terms(hdr, g - 2, f.zero ? -1.0f : -(dmin32 / sc), b);
                const uint32_t am = min0 + ms * C::MIN_BYTES + rl * 16 + (g - 2) * 8;
                sts64(am, b[0][0], b[0][1]);
                sts64(am + TILE_M * 16, b[0][0], b[0][1]);
                sts64(am + 2 * TILE_M * 16, b[1][0], b[1][1]);
                sts64(am + 3 * TILE_M * 16, b[1][0], b[1][1]);
                if (g == 2) sts32f(scale0 + ((u % SCALE_SLOTS) * TILE_M + rl) * 4, sc);
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(minfull0 + 8 * ms);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(rawempty0 + 8 * rs);
            if (drains && u > 0) drain(u - 1);
        }
        if (drains) {
            const uint32_t tk = tok0 + g * C::DRAIN_COLS * 4;
            griddep_wait();   // the kernel ahead may still read or write `out` and `aux`
            // this warp's columns' token scales through shared memory (the four quadrants' warps of a
            // column group write the same values): a load from global memory ahead of every store
            // would wait for the store before it
            for (int j = lane; j < C::DRAIN_COLS; j += 32) {
                const size_t t = (size_t)col0 + g * C::DRAIN_COLS + j;
                sts32f(tok0 + (g * C::DRAIN_COLS + j) * 4, t < a.n ? a.tok_scale[t] : 1.0f);
            }
            __syncwarp();
            // nothing to multiply by for activations of the usual range: every scale is one
            bool ones = true;
            for (int j = lane; j < C::DRAIN_COLS; j += 32) ones = ones && lds32f(tk + j * 4) == 1.0f;
            const bool scaled = !__all_sync(0xffffffffu, ones);
            if (OUT == 0 && a.epi != EPI_STORE && (size_t)row0 + quad * 32 < a.rows) {
                // what the epilogue will read, on its way to L2 while the last unit multiplies
                const size_t tb = (size_t)col0 + g * C::DRAIN_COLS;
                const float *src = a.epi == EPI_ADD ? a.out.dst[0] + a.out.row0 : a.aux;
                const size_t step = a.epi == EPI_ADD ? a.out.pitch : a.rows;
                for (int j = lane; j < C::DRAIN_COLS; j += 32)
                    if (tb + j < a.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + (tb + j) * step + row0 + quad * 32));
            }
            drain(units - 1);
            float acc[C::DRAIN_COLS];
#pragma unroll
            for (int j = 0; j < C::DRAIN_COLS / 2; j++) unpack2(acc2[j], acc[2 * j], acc[2 * j + 1]);
            const size_t row = (size_t)row0 + rl;
            if (OUT == 0 && split_k > 1) {
                const int own = C::owned(split_k);
                push_shares(acc, astage0, own, g, rl, rank, split_k);
                const EmitTo to = emit_to(a.out, a.aux, a.epi, row);
#pragma unroll
                for (int q = 0; q < C::DRAIN_COLS / 8; q++) {
                    if (q % split_k != rank) continue;
                    float v[8];
                    sum_shares(acc, q, astage0, own, g, rl, rank, split_k, v);
                    if (scaled) {
#pragma unroll
                        for (int j = 0; j < 8; j++) v[j] *= lds32f(tk + (8 * q + j) * 4);
                    }
                    if (row < a.rows) gemm_emit<false>(to, a.rows, a.n, (size_t)col0 + g * C::DRAIN_COLS + 8 * q, v);
                }
            } else if (OUT == 2) {
                // The group's tile [token][row] into the rings' shared memory, which nothing reads any
                // more (the last unit's MMAs are done, its accumulator drained), then one store per
                // destination.  Rows and tokens past the end are cut off by the maps' bounds.
                const uint32_t stage = astage0 + g * (C::DRAIN_COLS * TILE_M * 4);
                if (scaled) {
#pragma unroll
                    for (int j = 0; j < C::DRAIN_COLS; j++) acc[j] *= lds32f(tk + j * 4);
                }
#pragma unroll
                for (int j = 0; j < C::DRAIN_COLS; j++) sts32f(stage + (j * TILE_M + rl) * 4, acc[j]);
                fence_async_smem();
                asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");   // the group's four warps: all 128 rows are in
                const size_t t0 = (size_t)col0 + g * C::DRAIN_COLS;
                if (quad == 0 && lane == 0 && t0 < a.n) {
#pragma unroll
                    for (int p = 0; p < DWIM_MAX_WORLD; p++)
                        if (p < a.out.world) tma_store_2d(&maps.m[p], row0, (int)t0, stage);
                    tma_store_commit_wait();
                }
            } else if (row < a.rows) {
                const size_t cbase = (size_t)col0 + g * C::DRAIN_COLS;
                const EmitTo to = emit_to(a.out, a.aux, a.epi, row);
                const size_t n = a.n, rows = a.rows;
                if (scaled) {   // the tokens' powers of two
#pragma unroll
                    for (int j = 0; j < C::DRAIN_COLS; j++) acc[j] *= lds32f(tk + j * 4);
                }
#pragma unroll
                for (int j = 0; j < C::DRAIN_COLS; j += 8) {
                    float v[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) v[i] = acc[j + i];
                    gemm_emit<SHARED>(to, rows, n, cbase + j, v);
                }
            }
        }
    } else {
        if constexpr (TRADE) regs_dec<OTHER_REGS>();      // (a warpgroup's warps at one instruction)
        if (warp == X_WARP) {
            // ------------------------------ TMA producer ------------------------------
            griddep_wait();   // the operand comes from the prologue kernel just ahead
            if (elect_one()) {
                int bs = 0, bturn = 1;
                for (int u = 0; u < units; u++) {
                    const int ms = u % C::MIN_STAGES;
                    for (int p = PASSES - 1; p >= 0; p--)      // the remainders first
                        for (int h = 0; h < KBLOCKS; h++) {
                            uint32_t full = bfull0 + 8 * bs;
                            if (JOINT) {
                                // B stage kb % B_STAGES was last read by K block kb - B_STAGES
                                const int kb = KBLOCKS * u + h, prev = kb - C::B_STAGES;
                                if (prev >= 0)
                                    mbar_wait_parked(aempty0 + 8 * (prev % C::A_STAGES), (prev / C::A_STAGES) & 1, a.status, 0x20u);
                                full = afull0 + 8 * (kb % C::A_STAGES);
                            } else {
                                mbar_wait_parked(bempty0 + 8 * bs, bturn, a.status, 0x20u);
                            }
                            mbar_expect_tx(full, C::TERM_BYTES * (C::WIDE ? a.terms : 1));
                            const uint32_t to = bstage0 + bs * C::B_BYTES;
                            const int k = (KBLOCKS * (ub + u) + h) * BK;
                            tma_load_2d(to, &tmap_x, k, p * (int)a.n + col0, full);
                            if (C::WIDE && a.terms == 2) tma_load_2d(to + C::TERM_BYTES, &tmap_x, k, (int)a.n + col0, full);
                            if (++bs == C::B_STAGES) bs = 0, bturn ^= 1;
                        }
                    // the minimums' stage was last read by unit u - MIN_STAGES
                    if (u >= C::MIN_STAGES) {
                        const int uu = u - C::MIN_STAGES;
                        mbar_wait_parked(accfull0 + 8 * (uu & 1), (uu >> 1) & 1, a.status, 0x40u);
                    }
                    mbar_expect_tx(minfull0 + 8 * ms, C::BMIN_BYTES);
                    const uint32_t bm = min0 + ms * C::MIN_BYTES + AMIN_BYTES;
                    tma_load_2d(bm, &tmap_m, (ub + u) * 16, col0, minfull0 + 8 * ms);                 // the means' hi parts
                    tma_load_2d(bm + BN * 16, &tmap_m, (ub + u) * 16 + 8, col0, minfull0 + 8 * ms);   // and lo parts
                }
            }
        } else if (warp == RAW_WARP) {
            // ------------------------------ packed weights' producer ------------------------------
            // Its own warp: the blocks come from HBM and must run as far ahead as the
            // ring allows, whatever the activations' producer is waiting for.
            if (elect_one()) {
                for (int u = 0; u < units; u++) {
                    const int rs = u % C::RAW_STAGES;
                    mbar_wait_parked(rawempty0 + 8 * rs, ((u / C::RAW_STAGES) & 1) ^ 1, a.status, 0x10u);
                    mbar_expect_tx(rawfull0 + 8 * rs, TILE_M * 144);
                    tma_load_2d(raw0 + rs * RAW_BYTES, &tmap_w, (ub + u) * 144, row0, rawfull0 + 8 * rs);
                }
            }
        } else if (warp == MMA_WARP) {
            // ------------------------------ MMA issuer ------------------------------
            // The whole warp runs the loop (uniform control flow keeps addresses
            // and descriptors on the uniform data path) and one lane issues.  Units
            // are taken two at a time so that the accumulator buffer is static.
            constexpr uint32_t idesc_min = idesc_f16(TILE_M, BN);
            const uint32_t idesc = C::WIDE && a.terms == 2 ? idesc_f16(TILE_M, C::ACC_COLS) : idesc_min;
            constexpr uint32_t desc_hi = DESC_HI_SW128;
            const uint32_t a_lo = desc_lo_sw128(astage0), b_lo = desc_lo_sw128(bstage0);
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
            int bs = 0;                                                   // the next B stage
            uint32_t bturn = 0, slot = 0, turn = 0;                       // its phase; the next A stage and its phase
            for (int u0 = 0; u0 < units; u0 += 2) {
    #pragma unroll 1
                for (int ab = 0; ab < 2; ab++) {      // (unrolled, the 256-column form spilled more and took 475 us instead of 403)
                    const int u = u0 + ab;
                    if (u >= units) break;
                    const uint32_t s1 = tm + ab * C::ACC_COLS;
                    const uint32_t upar = (u0 >> 1) & 1;
                    mbar_wait_parked(accempty0 + 8 * ab, upar ^ 1, a.status, 0x80u);   // the drain of unit u-2 is done
                    const uint32_t slot0 = slot, turn0 = turn;
                    // All of the unit's remainders, then its values: the sum grows to its size in the second pass only,
                    // whose additions alone the accumulator rounds at that size.
                    for (int p = PASSES - 1; p >= 0; p--) {
                        const bool first = p == PASSES - 1;
                        slot = slot0, turn = turn0;
    #pragma unroll
                        for (int g = 0; g < KBLOCKS; g++) {
                            if (C::A_STAGES == KBLOCKS) slot = g, turn = ab;
                            if (first) mbar_wait_parked(afull0 + 8 * slot, turn, a.status, 0x100u);
                            if (!JOINT) mbar_wait_parked(bfull0 + 8 * bs, bturn, a.status, 0x8000u);
                            tc_fence_after();
                            const uint32_t ad = a_lo + slot * (A_BYTES >> 4), bd = b_lo + bs * (C::B_BYTES >> 4);
                            if (elect_one()) {
    #pragma unroll
                                for (int k = 0; k < BK / 16; k++) {   // 32 bytes further along the swizzled row per K=16
                                    if (g == 0 && k == 0) umma_f16_lo(s1, ad, bd, desc_hi, idesc, !first);
                                    else umma_f16_lo<1>(s1, ad + 2 * k, bd + 2 * k, desc_hi, idesc);
                                }
                                // the stages may be refilled once these finish
                                if (!JOINT) umma_commit(bempty0 + 8 * bs);
                                if (p == 0) umma_commit(aempty0 + 8 * slot);
                            }
                            __syncwarp();
                            if (++bs == C::B_STAGES) bs = 0, bturn ^= 1;
                            if (C::A_STAGES != KBLOCKS && ++slot == C::A_STAGES) slot = 0, turn ^= 1;
                        }
                    }
                    const int ms = u % C::MIN_STAGES;
                    mbar_wait_parked(minfull0 + 8 * ms, (u / C::MIN_STAGES) & 1, a.status, 0x200u);
                    tc_fence_after();
                    if (elect_one()) {
                        // the minimums: terms (hi, hi | lo, lo) against the means' (hi, lo) twice
                        const uint32_t am = min0 + ms * C::MIN_BYTES;
                        const uint64_t bdm = smem_desc_plain(am + AMIN_BYTES, BN * 16);
                        umma_f16(s1, smem_desc_plain(am, TILE_M * 16), bdm, idesc_min, 1);
                        umma_f16(s1, smem_desc_plain(am + 2 * TILE_M * 16, TILE_M * 16), bdm, idesc_min, 1);
                        umma_commit(accfull0 + 8 * ab);     // the unit's sum is complete
                    }
                    __syncwarp();
                }
            }
        }
    }
    if (warp >= N_WORKERS) {
        __syncwarp();
        if (split_k > 1) {      // the workers' two meetings are the whole cluster's
            cluster_sync();
            cluster_sync();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

// ---- the dense kernel: Q8_0 and Q6_K above the small-M kernel's range --------------------------
// Those formats scale every 32 (Q8_0) or 16 (Q6_K) weights by a factor of their own, and a weight
// times its factor does not fit f16's 11 bits.  The A operand is therefore carried exactly as two f16
// terms, hi = f16(factor * q) and lo = factor * q - hi (an fma, exact: the product has 13 bits for Q6_K,
// whose factor is the integer sub-scale, and 19 for Q8_0, whose factor is the block's d times a power of
// two that brings the unit's largest to [64, 128)), two MMAs per 16 of K into one accumulator a unit;
// the unit's d (Q8_0: the power of two) is applied when it is drained, in fp32, as Q4_K's.
// The kernel is Q4_K's in outline (roles, hand-overs, drains; see there), but for: two A stages of a hi and
// a lo tile, K block kb in stage kb % 2; a ring of its own for the activations; no minimums.
// (The terms used to be written to memory by a pass of their own and loaded by every column of tiles: 64 KB
// from L2 per K block of 1024 cycles, 9.1 TB/s, was what bound it.  Products with their operand, in short bursts:
// [12288, 5120] Q6_K by 512 f32 tokens 299 us then, 209 as two columns a token, 207 now (236 with their operand);
// [5120, 5120] Q8_0 by 512 of them 127 as columns, 128 with spills in the main loop, 106 now.  Errors, 2-norm over the
// result's: 1e-6 to 1e-5 over K = 2304 to 12288 then; now, at any K from 512 to 17408, by f32 activations 4.2e-7 (Q6_K)
// and 5.9e-7 (Q8_0) up to 128 tokens and 3.2e-7 and 3.9e-7 above, by bf16 ones 2.7e-7 and 5.6e-7, the largest difference
// 2.0e-6 and 3.0e-6 of the result's root mean square.)
// Bound by the tensor pipe (68 % active by 256 tokens).  The scales are fetched where they are used: fetched a unit
// ahead they cost the 256-column forms 130 to 400 bytes of spills.
struct DenseArgs {
    size_t rows, n, units;
    int terms, epi, split_k;
    OutSpec out;
    const __half *scales;           // Q8_0: eight per unit and row; Q6_K: one
    size_t srow;
    const float *tok_scale, *aux;
    uint32_t *status;
};
// Two terms that take turns double the additions to an accumulator, so it is drained twice a unit; tiles of 64 columns
// take the place of exact sums and drain every K block.
template <int FMT, int BN, int MODE> struct DenseCfg {
    static constexpr bool WIDE = MODE == SIDE_BY_SIDE;
    static constexpr int DRAIN_KB = BN <= 64 ? 1 : MODE == TWO_PASSES ? 2 : KBLOCKS;      // K blocks between drains
    static constexpr int TERM_BYTES = BN * BK * 2, ACC_COLS = BN * (WIDE ? 2 : 1);
    static constexpr int A_STAGES = BN <= 64 ? 4 : 2, A_STAGE = 2 * A_BYTES;
    static constexpr int STEPS = KBLOCKS / DRAIN_KB;                // drains of a unit
    // Accumulator buffers: two units' where tensor memory holds them, else two steps'.
    static constexpr int ACC_BUFS = 2 * STEPS * ACC_COLS <= 512 ? 2 * STEPS : 2;
    static_assert(STEPS < 4 || (ACC_BUFS == 8 && BN == 64), "drain_unit");
    static_assert(ACC_BUFS == 2 * STEPS || STEPS == 2, "a unit of more steps than buffers would wait for itself");
    static constexpr int TMEM_COLS = ACC_BUFS * ACC_COLS > 256 ? 512 : 256;
    static constexpr int B_STAGES = ACC_COLS > 192 ? 3 : 4, B_BYTES = TERM_BYTES * (WIDE ? 2 : 1);
    // raw weights: a unit of Q6_K, half a unit of Q8_0 (128 bytes a row, swizzled)
    static constexpr int RAW_STEPS = FMT == Q8_0 ? 2 : 1;           // ring stages per unit
    static constexpr int RAW_STAGES = FMT == Q8_0 ? 3 : 2, RAW_STAGE = FMT == Q8_0 ? TILE_M * 128 : TILE_M * Q6_K_DEV;
    static constexpr int RINGS = A_STAGES * A_STAGE + B_STAGES * B_BYTES + RAW_STAGES * RAW_STAGE;
    static constexpr int SMEM = BAR_BYTES + RINGS + SCALE_SLOTS * TILE_M * 4 + BN * 4 + 1024;
    static_assert(SMEM <= MAX_SMEM, "the tile does not fit shared memory");
    static constexpr int DRAIN_COLS = BN / 4;
    static constexpr int owned(int s) { return (DRAIN_COLS / 8 + s - 1) / s * 8; }
    static constexpr bool split_fits(int s) { return s * 4 * owned(s) * TILE_M * 4 <= RINGS; }
};
// byte + 1024 as f16, minus the offset: (bytes 0, 2) and (bytes 1, 3)
__device__ __forceinline__ void bytes_to_f16(uint32_t w, uint32_t offset, uint32_t &lo, uint32_t &hi) {
    lo = hsub2(prmt(w, 0x64006400u, 0x5250u), offset);
    hi = hsub2(prmt(w, 0x64006400u, 0x5351u), offset);
}
// Eight weights (two words of bytes) times a factor as hi and lo, to 16-byte chunk `c` of the row in either tile.
__device__ __forceinline__ void store_terms(uint32_t w0, uint32_t w1, uint32_t offset, uint32_t factor, uint32_t a_row_sw, int c) {
    uint32_t q[4], h[4], l[4];
    bytes_to_f16(w0, offset, q[0], q[1]);
    bytes_to_f16(w1, offset, q[2], q[3]);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        h[i] = hmul2(q[i], factor);
        l[i] = hfma2(q[i], factor, h[i] ^ 0x80008000u);
    }
    sts128(a_row_sw ^ (c << 4), h[0], h[1], h[2], h[3]);
    sts128((a_row_sw + A_BYTES) ^ (c << 4), l[0], l[1], l[2], l[3]);
}

template <int FMT, int BN, int MODE, bool SHARED>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_dense_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ DenseArgs a) {
    using C = DenseCfg<FMT, BN, MODE>;
    constexpr int DRAIN_KB = C::DRAIN_KB, PASSES = MODE == TWO_PASSES ? 2 : 1;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    // afull, adone: one per K block of the unit, completed once a unit
    const uint32_t afull0 = base, adone0 = base + 32, bfull0 = base + 64, bempty0 = base + 96, accfull0 = base + 128, accempty0 = base + 192;
    const uint32_t rawfull0 = base + 256, rawempty0 = base + 288, tmem_slot = base + 320;
    const uint32_t astage0 = base + BAR_BYTES, bstage0 = astage0 + C::A_STAGES * C::A_STAGE, raw0 = bstage0 + C::B_STAGES * C::B_BYTES;
    const uint32_t scale0 = raw0 + C::RAW_STAGES * C::RAW_STAGE, tok0 = scale0 + SCALE_SLOTS * TILE_M * 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split_k = SHARED ? 1 : a.split_k, rank = (int)(blockIdx.x % split_k);
    const int row0 = (int)(blockIdx.x / split_k) * TILE_M, col0 = blockIdx.y * BN;
    const int ub = (int)a.units * rank / split_k, units = (int)a.units * (rank + 1) / split_k - ub;
    if (threadIdx.x == 0) {
        for (int g = 0; g < KBLOCKS; g++) {
            mbar_init(afull0 + 8 * g, 4);                // the K block's four worker warps
            mbar_init(adone0 + 8 * g, 1);
        }
        for (int s = 0; s < C::ACC_BUFS; s++) {
            mbar_init(accfull0 + 8 * s, 1);
            mbar_init(accempty0 + 8 * s, N_WORKERS);
        }
        for (int s = 0; s < C::B_STAGES; s++) {
            mbar_init(bfull0 + 8 * s, 1);
            mbar_init(bempty0 + 8 * s, 1);
        }
        for (int s = 0; s < C::RAW_STAGES; s++) {
            mbar_init(rawfull0 + 8 * s, 1);
            mbar_init(rawempty0 + 8 * s, N_WORKERS / C::RAW_STEPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = lds32(tmem_slot);
    griddep_launch();

    if (warp < N_WORKERS) {
        regs_inc<DENSE_WORKER_REGS>();
        const int quad = warp & 3, g = warp >> 2, rl = quad * 32 + lane;
        const uint32_t drain_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + g * C::DRAIN_COLS;
        const uint32_t a_row_sw = (astage0 + g % C::A_STAGES * C::A_STAGE + rl * 128) | ((rl & 7) << 4);
        const size_t row = (size_t)row0 + rl;
        uint64_t acc2[C::DRAIN_COLS / 2];
#pragma unroll
        for (int j = 0; j < C::DRAIN_COLS / 2; j++) acc2[j] = 0ull;
        int buf = 0, bufturn = 0;
        auto drain = [&](int u) {      // the next step, one of unit u's
            mbar_wait_parked(accfull0 + 8 * buf, bufturn, a.status, 0x2000000u);
            tc_fence_after();
            // written before the unit's first K block was handed over
            const uint32_t sc = __float_as_uint(lds32f(scale0 + ((u % SCALE_SLOTS) * TILE_M + rl) * 4));
            const uint64_t sc2 = pack2(sc, sc);
#pragma unroll
            for (int c = 0; c < C::DRAIN_COLS / 16; c++) {
                uint32_t v[16];
                tmem_ld16(drain_addr + buf * C::ACC_COLS + c * 16, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; j++) ffma2(acc2[c * 8 + j], sc2, pack2(v[2 * j], v[2 * j + 1]));
                if (C::WIDE && a.terms == 2) {
                    tmem_ld16(drain_addr + buf * C::ACC_COLS + BN + c * 16, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; j++) ffma2(acc2[c * 8 + j], sc2, pack2(v[2 * j], v[2 * j + 1]));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(accempty0 + 8 * buf);
            if (++buf == C::ACC_BUFS) buf = 0, bufturn ^= 1;
        };
        // All four steps of unit u: their sums meet before they reach the row's, which rounds once a unit so.
        auto drain_unit = [&](int u) {
            const uint32_t sc = __float_as_uint(lds32f(scale0 + ((u % SCALE_SLOTS) * TILE_M + rl) * 4));
            const uint64_t sc2 = pack2(sc, sc);
            uint64_t sum[C::DRAIN_COLS / 2];
#pragma unroll
            for (int half = 0; half < 2; half++) {
                uint32_t v[2][16];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    mbar_wait_parked(accfull0 + 8 * (buf + 2 * half + i), bufturn, a.status, 0x2000000u);
                    tc_fence_after();
                    tmem_ld16(drain_addr + (buf + 2 * half + i) * C::ACC_COLS, v[i]);
                }
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < C::DRAIN_COLS / 2; j++) {
                    const uint64_t two = fadd2(pack2(v[0][2 * j], v[0][2 * j + 1]), pack2(v[1][2 * j], v[1][2 * j + 1]));
                    if (half == 0) sum[j] = two;
                    else ffma2(acc2[j], sc2, fadd2(sum[j], two));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane < 4) mbar_arrive(accempty0 + 8 * (buf + lane));
            buf ^= 4;
            if (buf == 0) bufturn ^= 1;
        };
        // With two buffers for a unit's two steps the first of the unit before is drained ahead of the decode: its
        // buffer is the one that this unit's first step takes, which K blocks 2 and 3 wait for (their stages').
        constexpr int EARLY = C::ACC_BUFS == 2 * C::STEPS ? 0 : 1;
        // the row's scales (rows past the end: the last row's, their weights are zeros)
        const __half *srow = a.scales + (row < a.rows ? row : a.rows - 1) * a.srow;
        auto fetch = [&](int u) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (u < units) {
                if (FMT == Q8_0) v = *reinterpret_cast<const uint4 *>(srow + (size_t)(ub + u) * 8);
                else v.x = *reinterpret_cast<const unsigned short *>(srow + ub + u);
            }
            return v;
        };
        // (One turn more than there are units, so that the drain is in the code once or twice.)
        const uint32_t tk = tok0 + g * C::DRAIN_COLS * 4;
        for (int u = 0; u <= units; u++) {
            if (EARLY && u > 0) drain(u - 1);
            if (u < units) {
                const uint4 sc = fetch(u);
                const int r = C::RAW_STEPS == 2 ? 2 * u + (g >> 1) : u, rs = r % C::RAW_STAGES;
                mbar_wait_parked(rawfull0 + 8 * rs, (r / C::RAW_STAGES) & 1, a.status, 0x4000000u);
                // the stage's last user is done: the K block of the unit before, or with two stages (this warp has waited for
                // the use before that one) the one two K blocks back
                if (C::A_STAGES == KBLOCKS) mbar_wait_parked(adone0 + 8 * g, (u & 1) ^ 1, a.status, 0x8000000u);
                else mbar_wait_parked(adone0 + 8 * (g ^ 2), (u & 1) ^ (g < 2 ? 1 : 0), a.status, 0x8000000u);
                const uint32_t raw = raw0 + rs * C::RAW_STAGE;
                float unit_scale;
                if constexpr (FMT == Q6_K) {
                    // The block's four groups (formats.cuh): word j of lane c for them at 64 j + 16 c + 4 g.
                    const uint32_t rrow = raw + rl * Q6_K_DEV;
                    const uint32_t s4 = lds32(rrow + 192 + 4 * g) ^ 0x80808080u;      // the groups' sub-scales + 128
                    unit_scale = 0.25f * h2f_lo(sc.x);                                // the quants come four times as large
                    uint32_t f[4];                                                    // 0x6480 = 1152 = 1024 + 128
#pragma unroll
                    for (int k = 0; k < 4; k++) f[k] = hsub2(prmt(s4, 0x64006400u, 0x5050u + k * 0x0101u), 0x64806480u);
#pragma unroll
                    for (int c = 0; c < 4; c += 2) {
                        uint32_t q[2][4];
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            const uint32_t at = rrow + 16 * (c + i) + 4 * g;
                            q6k_bytes(lds32(at), lds32(at + 64), lds32(at + 128), q[i]);
                        }
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            store_terms(q[0][k] ^ 0x80808080u, q[1][k] ^ 0x80808080u, 0x64806480u, f[k], a_row_sw, 2 * k + (c >> 1));
                    }
                } else {
                    // the unit's power of two: its largest |d| to [64, 128)
                    const uint32_t m2 = __vmaxu2(__vmaxu2(sc.x & 0x7fff7fffu, sc.y & 0x7fff7fffu), __vmaxu2(sc.z & 0x7fff7fffu, sc.w & 0x7fff7fffu));
                    const int e = (int)(max(m2 & 0xffffu, m2 >> 16) >> 10);
                    const int up = 6 - (max(e, 1) - 15);
                    const float by = __uint_as_float((uint32_t)(127 + up) << 23);
                    unit_scale = __uint_as_float((uint32_t)(127 - up) << 23);
                    const uint32_t d2 = g == 0 ? sc.x : g == 1 ? sc.y : g == 2 ? sc.z : sc.w;
                    const float d0 = h2f_lo(d2) * by, d1 = h2f_hi(d2) * by;
                    const uint32_t f[2] = {f16x2_rn(d0, d0), f16x2_rn(d1, d1)};
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const uint4 q = lds128(raw + rl * 128 + ((((g & 1) * 4 + c) ^ (rl & 7)) << 4));
                        store_terms(q.x ^ 0x80808080u, q.y ^ 0x80808080u, 0x64806480u, f[c >> 1], a_row_sw, 2 * c);
                        store_terms(q.z ^ 0x80808080u, q.w ^ 0x80808080u, 0x64806480u, f[c >> 1], a_row_sw, 2 * c + 1);
                    }
                }
                if (g == 0) sts32f(scale0 + ((u % SCALE_SLOTS) * TILE_M + rl) * 4, unit_scale);
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(afull0 + 8 * g);
                    mbar_arrive(rawempty0 + 8 * rs);
                }
            } else {
                griddep_wait();   // the kernel ahead may still read or write `out` and `aux`
                for (int j = lane; j < C::DRAIN_COLS; j += 32) {
                    const size_t t = (size_t)col0 + g * C::DRAIN_COLS + j;
                    sts32f(tok0 + (g * C::DRAIN_COLS + j) * 4, t < a.n ? a.tok_scale[t] : 1.0f);
                }
                __syncwarp();
            }
            if (u > 0) {
                if constexpr (C::STEPS == 4) {
                    drain_unit(u - 1);
                } else {
#pragma unroll 1
                    for (int i = EARLY; i < C::STEPS; i++) drain(u - 1);
                }
            }
        }
        float acc[C::DRAIN_COLS];
#pragma unroll
        for (int j = 0; j < C::DRAIN_COLS / 2; j++) unpack2(acc2[j], acc[2 * j], acc[2 * j + 1]);
        const int own = C::owned(split_k);
        if (split_k > 1) push_shares(acc, astage0, own, g, rl, rank, split_k);
        const EmitTo to = emit_to(a.out, a.aux, a.epi, row);
#pragma unroll
        for (int q = 0; q < C::DRAIN_COLS / 8; q++) {
            if (q % split_k != rank) continue;
            float v[8];
            if (split_k > 1) {
                sum_shares(acc, q, astage0, own, g, rl, rank, split_k, v);
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++) v[j] = acc[8 * q + j];
            }
            if (row >= a.rows) continue;
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] *= lds32f(tk + (8 * q + j) * 4);
            gemm_emit<SHARED>(to, a.rows, a.n, (size_t)col0 + g * C::DRAIN_COLS + 8 * q, v);
        }
    } else {
        regs_dec<DENSE_OTHER_REGS>();      // (a warpgroup's warps at one instruction)
        if (warp == X_WARP) {
            griddep_wait();   // the operand comes from the prologue kernel just ahead
            if (elect_one()) {
                int s = 0, turn = 1;
                for (int kb = 0; kb < KBLOCKS * units; kb++)
                    for (int p = PASSES - 1; p >= 0; p--) {      // the remainders first
                        mbar_wait_parked(bempty0 + 8 * s, turn, a.status, 0x100000u);
                        mbar_expect_tx(bfull0 + 8 * s, C::TERM_BYTES * (C::WIDE ? a.terms : 1));
                        const uint32_t to = bstage0 + s * C::B_BYTES;
                        tma_load_2d(to, &tmap_x, (KBLOCKS * ub + kb) * BK, p * (int)a.n + col0, bfull0 + 8 * s);
                        if (C::WIDE && a.terms == 2) tma_load_2d(to + C::TERM_BYTES, &tmap_x, (KBLOCKS * ub + kb) * BK, (int)a.n + col0, bfull0 + 8 * s);
                        if (++s == C::B_STAGES) s = 0, turn ^= 1;
                    }
            }
        } else if (warp == RAW_WARP) {
            if (elect_one()) {
                for (int r = 0; r < C::RAW_STEPS * units; r++) {
                    const int s = r % C::RAW_STAGES;
                    mbar_wait_parked(rawempty0 + 8 * s, ((r / C::RAW_STAGES) & 1) ^ 1, a.status, 0x200000u);
                    mbar_expect_tx(rawfull0 + 8 * s, C::RAW_STAGE);
                    tma_load_2d(raw0 + s * C::RAW_STAGE, &tmap_w, FMT == Q8_0 ? (2 * ub + r) * 128 : (ub + r) * Q6_K_DEV, row0, rawfull0 + 8 * s);
                }
            }
        } else if (warp == MMA_WARP) {
            const uint32_t idesc = idesc_f16(TILE_M, C::WIDE && a.terms == 2 ? C::ACC_COLS : BN);
            const uint32_t a_lo = desc_lo_sw128(astage0), b_lo = desc_lo_sw128(bstage0);
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
            int bs = 0, bturn = 0, buf = 0, bufturn = 1;
            for (int u = 0; u < units; u++) {
    #pragma unroll
                for (int g = 0; g < KBLOCKS; g++) {
                    const uint32_t acc = tm + buf * C::ACC_COLS;
                    // What a K block needs: asked by lanes of the warp at once where its MMAs are so short that the 85 cycles
                    // of a test count ([5120, 5120] Q8_0 by 48 tokens 24.6 us one by one, 23.1 like this; wider tiles spill).
                    constexpr bool AT_ONCE = C::STEPS == 4;
                    if (!AT_ONCE) {
                        if (g % DRAIN_KB == 0) mbar_wait_parked(accempty0 + 8 * buf, bufturn, a.status, 0x400000u);
                        mbar_wait_parked(afull0 + 8 * g, u & 1, a.status, 0x1000000u);
                    }
    #pragma unroll AT_ONCE ? 2 : 1
                    for (int p = PASSES - 1; p >= 0; p--) {
                        if (AT_ONCE) {
                            uint32_t bar = bfull0 + 8 * bs, phase = bturn;
                            if (p == PASSES - 1 && (lane & 1)) bar = afull0 + 8 * g, phase = u & 1;
                            if (p == PASSES - 1 && (lane & 2)) bar = accempty0 + 8 * buf, phase = bufturn;
                            mbar_wait_all(bar, phase, a.status, 0x800000u);
                        } else {
                            mbar_wait_parked(bfull0 + 8 * bs, bturn, a.status, 0x800000u);
                        }
                        tc_fence_after();
                        if (elect_one()) {
                            // the weights' remainders first: they are too small for the accumulator's rounding to matter
                            const uint32_t hi = a_lo + g % C::A_STAGES * (C::A_STAGE >> 4), lo = hi + (A_BYTES >> 4), bd = b_lo + bs * (C::B_BYTES >> 4);
    #pragma unroll
                            for (int k = 0; k < BK / 16; k++) {
                                if (g % DRAIN_KB == 0 && k == 0) umma_f16_lo(acc, lo, bd, DESC_HI_SW128, idesc, p != PASSES - 1);
                                else umma_f16_lo<1>(acc, lo + 2 * k, bd + 2 * k, DESC_HI_SW128, idesc);
                            }
    #pragma unroll
                            for (int k = 0; k < BK / 16; k++) umma_f16_lo<1>(acc, hi + 2 * k, bd + 2 * k, DESC_HI_SW128, idesc);
                            umma_commit(bempty0 + 8 * bs);
                            if (p == 0) {
                                umma_commit(adone0 + 8 * g);
                                if (g % DRAIN_KB == DRAIN_KB - 1) umma_commit(accfull0 + 8 * buf);
                            }
                        }
                        __syncwarp();
                        if (++bs == C::B_STAGES) bs = 0, bturn ^= 1;
                    }
                    if (g % DRAIN_KB == DRAIN_KB - 1 && ++buf == C::ACC_BUFS) buf = 0, bufturn ^= 1;
                }
            }
        }
    }
    if (warp >= N_WORKERS) {
        __syncwarp();
        if (split_k > 1) {      // the workers' two meetings are the whole cluster's
            cluster_sync();
            cluster_sync();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

// ---- host side ---------------------------------------------------------------------
typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
    static const EncodeTiled fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (EncodeTiled)p;
    }();
    return fn;
}

}  // namespace

int encode_nd(dwim_b200_ctx *ctx, CUtensorMap *map, CUtensorMapDataType type, const void *ptr, int rank, const uint64_t *dims,
              const uint64_t *pitches, const uint32_t *box, CUtensorMapSwizzle swizzle, const char *what) {
    EncodeTiled enc = encode_fn();
    if (!enc) return fail(ctx, DWIM_B200_ECUDA, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t d[5], s[4];
    cuuint32_t b[5], es[5];
    for (int i = 0; i < rank; i++) d[i] = dims[i], b[i] = box[i], es[i] = 1;
    for (int i = 0; i + 1 < rank; i++) s[i] = pitches[i];
    CUresult r = enc(map, type, (cuuint32_t)rank, const_cast<void *>(ptr), d, s, b, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ctx, DWIM_B200_ECUDA, "encoding the %s tensor map failed (%d)", what, (int)r);
    return 0;
}

int encode_2d(dwim_b200_ctx *ctx, CUtensorMap *map, CUtensorMapDataType type, const void *ptr, uint64_t inner, uint64_t outer,
              uint64_t pitch_bytes, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swizzle, const char *what) {
    const uint64_t dims[2] = {inner, outer};
    const uint32_t box[2] = {box_inner, box_outer};
    return encode_nd(ctx, map, type, ptr, 2, dims, &pitch_bytes, box, swizzle, what);
}

namespace {

// What a unit costs by two terms an activation, in units by one: the tensor work doubles, the decode does not.
double q4k_unit(int bn, int terms) { return terms == 1 ? 1.0 : bn >= 128 ? 1.8 : 1.1; }

// How many blocks share a tile of the Q4_K kernel at this width, and how long the product then takes
// (in units of one term on the busiest block).
template <int BN, int MODE>
int gemm_split(dwim_b200_ctx *ctx, const WeightView &w, size_t n, int terms, double *time = nullptr) {
    static std::atomic<int> known[64][MAX_SPLIT + 1] = {};
    const long tiles = (long)((w.rows + TILE_M - 1) / TILE_M) * (long)((n + BN - 1) / BN);
    return pick_split(ctx, gemm_q4k_kernel<BN, 0, MODE>, GEMM_THREADS, (size_t)Cfg<BN, MODE>::SMEM, Cfg<BN, MODE>::split_fits,
                      SplitCost{3.0, 6.5}, known, tiles, (int)(w.cols / 256), q4k_unit(BN, terms), time);
}
template <int BN, int MODE> double gemm_time(dwim_b200_ctx *ctx, const WeightView &w, size_t n, int terms) {
    double t = 0;
    gemm_split<BN, MODE>(ctx, w, n, terms, &t);
    return t;
}

template <int BN, int MODE>
int launch_gemm(dwim_b200_ctx *ctx, const WeightView &w, const __half *operand, size_t n, int terms, const OutSpec &out,
                const float *aux, int epi) {
    using C = Cfg<BN, MODE>;
    const size_t units = w.cols / 256;
    CUtensorMap tw, tx, tm;
    int rc;
    // packed weights as bytes: [rows][qpitch], box [128 rows][144 bytes]; rows past the end read as zero blocks
    if ((rc = encode_2d(ctx, &tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, w.quants, w.qpitch, w.rows, w.qpitch, 144, TILE_M,
                        CU_TENSOR_MAP_SWIZZLE_NONE, "weight")))
        return rc;
    // activations: [terms][n][K] f16, box [BN][64], 128-byte swizzle; columns past the last token read as another
    // term's tokens or as zeros
    if ((rc = encode_2d(ctx, &tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, operand, w.cols, terms * n, w.cols * 2, BK, BN,
                        CU_TENSOR_MAP_SWIZZLE_128B, "activation")))
        return rc;
    // sub-block means: [n][units*16] f16, box [BN][8]
    if ((rc = encode_2d(ctx, &tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, operand + terms * n * w.cols, units * 16, n, units * 32, 8,
                        BN, CU_TENSOR_MAP_SWIZZLE_NONE, "means")))
        return rc;
    const float *tok_scale = reinterpret_cast<const float *>(operand + (terms * w.cols + units * 16) * n);
    GemmArgs a{w.rows, n, units, terms, out, tok_scale, aux, epi, 1, ctx->status};
    // A result shared by several ranks' copies takes an instantiation that stores to all of them: with
    // TMA from shared memory when every copy's slice starts on a 16-byte boundary, else from registers.
    int shared = out.world > 1 && !out.scatter_per ? 1 : 0;
    OutMaps maps;          // only the TMA form reads it
    if (shared && epi == EPI_STORE && out.pitch % 4 == 0) {
        shared = 2;
        for (int p = 0; p < out.world; p++)
            if (reinterpret_cast<uintptr_t>(out.dst[p] + out.row0) % 16) shared = 1;
        for (int p = 0; p < out.world && shared == 2; p++)
            if ((rc = encode_2d(ctx, &maps.m[p], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, out.dst[p] + out.row0, w.rows, n,
                                out.pitch * sizeof(float), TILE_M, (uint32_t)C::DRAIN_COLS,
                                CU_TENSOR_MAP_SWIZZLE_NONE, "output")))
                return rc;
    }
    // gemm_large takes tiles of 192 columns for one destination alone, and of 32 for several
    constexpr bool ONE = BN != 32, SEVERAL = BN != 192;
    if (shared ? !SEVERAL : !ONE) return fail(ctx, DWIM_B200_EINVAL, "tiles of %d columns by %d destinations", BN, out.world);
    auto kern = gemm_q4k_kernel<BN, ONE ? 0 : 1, MODE>;
    if constexpr (SEVERAL) {
        if (shared == 2) kern = gemm_q4k_kernel<BN, 2, MODE>;
        if (shared == 1) kern = gemm_q4k_kernel<BN, 1, MODE>;
    }
    static std::atomic<bool> configured[64][3] = {};
    constexpr int SHARES = C::TRADE ? 512 * WORKER_REGS + 128 * OTHER_REGS : 0;
    if ((rc = configure_gemm(ctx, kern, C::SMEM, GEMM_THREADS, SHARES, configured[ctx->device & 63][shared]))) return rc;
    dim3 grid((unsigned)((w.rows + TILE_M - 1) / TILE_M), (unsigned)((n + BN - 1) / BN));
    if constexpr (ONE) {
        if (!shared) {
            a.split_k = gemm_split<BN, MODE>(ctx, w, n, terms);
            grid.x *= a.split_k;
        }
    }
    const bool dependent = !ctx->weights_written;   // see dwim_b200_ctx::weights_written
    DWIM_CUDA(ctx, launch_clustered(dependent, (unsigned)a.split_k, kern, grid, dim3(GEMM_THREADS), (size_t)C::SMEM, ctx->stream, tw, tx, tm, a,
                                    maps));
    ctx->weights_written = false;
    DWIM_LAUNCHED(ctx);
    return 0;
}

template <int FMT, int BN, int MODE>
int dense_split(dwim_b200_ctx *ctx, const WeightView &w, size_t n, int terms, double *time = nullptr) {
    using C = DenseCfg<FMT, BN, MODE>;
    static std::atomic<int> known[64][MAX_SPLIT + 1] = {};
    const long tiles = (long)((w.rows + TILE_M - 1) / TILE_M) * (long)((n + BN - 1) / BN);
    return pick_split(ctx, gemm_dense_kernel<FMT, BN, MODE, false>, GEMM_THREADS, (size_t)C::SMEM, C::split_fits, SplitCost{2.0, 4.5}, known, tiles,
                      (int)(w.cols / 256), terms == 1 ? 1.0 : 1.9, time);
}
template <int FMT, int BN, int MODE> double dense_time(dwim_b200_ctx *ctx, const WeightView &w, size_t n, int terms) {
    double t = 0;
    dense_split<FMT, BN, MODE>(ctx, w, n, terms, &t);
    return t;
}

template <int FMT, int BN, int MODE>
int launch_dense(dwim_b200_ctx *ctx, const WeightView &w, const __half *operand, size_t n, int terms, const OutSpec &out, const float *aux,
                 int epi, size_t whole) {
    using C = DenseCfg<FMT, BN, MODE>;
    const size_t units = w.cols / 256;
    CUtensorMap tw, tx;
    int rc;
    // packed weights as bytes; rows past the end read as zeros
    if ((rc = encode_2d(ctx, &tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, w.quants, w.qpitch, w.rows, w.qpitch, FMT == Q8_0 ? 128 : Q6_K_DEV, TILE_M,
                        FMT == Q8_0 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, "weight")))
        return rc;
    if ((rc = encode_2d(ctx, &tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, operand, w.cols, terms * n, w.cols * 2, BK, BN, CU_TENSOR_MAP_SWIZZLE_128B,
                        "activation")))
        return rc;
    const float *tok_scale = reinterpret_cast<const float *>(operand + (terms * w.cols + units * 16) * n);
    DenseArgs a{w.rows, n, units, terms, epi, 1, out, w.scales, w.srow, tok_scale, aux, ctx->status};
    const bool shared = out.world > 1 && !out.scatter_per;
    auto kern = shared ? gemm_dense_kernel<FMT, BN, MODE, true> : gemm_dense_kernel<FMT, BN, MODE, false>;
    static std::atomic<bool> configured[64][2] = {};
    constexpr int SHARES = 512 * DENSE_WORKER_REGS + 128 * DENSE_OTHER_REGS;
    if ((rc = configure_gemm(ctx, kern, C::SMEM, GEMM_THREADS, SHARES, configured[ctx->device & 63][shared]))) return rc;
    dim3 grid((unsigned)((w.rows + TILE_M - 1) / TILE_M), (unsigned)((n + BN - 1) / BN));
    if (!shared) {
        a.split_k = dense_split<FMT, BN, MODE>(ctx, w, whole, terms);
        grid.x *= a.split_k;
    }
    const bool dependent = !ctx->weights_written;   // see dwim_b200_ctx::weights_written
    DWIM_CUDA(ctx, launch_clustered(dependent, (unsigned)a.split_k, kern, grid, dim3(GEMM_THREADS), (size_t)C::SMEM, ctx->stream, tw, tx, a));
    ctx->weights_written = false;
    DWIM_LAUNCHED(ctx);
    return 0;
}

}  // namespace

// Whether the tensor-core kernels take a product of n tokens by so many f16 terms: Q4_K from nine tokens on (25 us at
// nine to sixteen in the kernel of many columns, [17408, 5120], against 57 for sixteen through two small-M launches).
// Q6_K and Q8_0, whose alternative is the small-M kernel in groups of eight tokens, by time and by error:
//   two terms (f32 activations): from 25 tokens on.  Drained every K block (up to 64 tokens, and rows above 12288) the
//     dense kernel's error is 1.3e-7 to 1.5e-7 of the result in 2-norm, the groups' 2.9e-7 to 3.1e-7 (23-bit planes).
//     Products with their operand, us, at 16, 24, 32 and 48 tokens: Q8_0 [5120, 5120] 21 31 32 51 in groups, 27 28 28 29
//     dense; [12288, 5120] 37 53 64 96 and 58 58 58 58; [1024, 5120] 11 16 18 26 and 17; [20000, 1024] 20 29 38 54 and 30;
//     [5120, 17408] by 32 88 and 73, by 512 1293 and 512; Q6_K within a tenth of these.
//   one term (bf16 activations): from 65 tokens on, up to 12288 columns.  It would be faster from 17 on ([5120, 5120] by
//     48 22 us, 51 in groups), but its error is 0.9e-7 to 1.3e-7 where the groups' is 0.6e-7 to 1.2e-7.
constexpr size_t DENSE_FROM[2] = {65, 25};      // tokens, by one and two terms
bool gemm_takes(const WeightView &w, size_t n, int terms) {
    if (w.cols % 256) return false;
    if (w.fmt == Q4_K) return n > (size_t)I8_MAX_TOKENS;
    return (w.fmt == Q6_K || w.fmt == Q8_0) && n >= DENSE_FROM[terms - 1] && w.cols <= (terms == 2 ? 51200 : DENSE_ROWS);
}

// `whole`: the tokens of the product that these are a piece of (the forms drained every K block may be taken in pieces).
int gemm_large(dwim_b200_ctx *ctx, const WeightView &w, const __half *operand, size_t n, int terms, const OutSpec &out,
               const float *aux, int epilogue, size_t whole) {
    if (!gemm_takes(w, whole, terms)) return fail(ctx, DWIM_B200_EFORMAT, "the tensor-core GEMM does not take format %d, %zu tokens", w.fmt, whole);
    if (w.fmt == Q4_K) {
        // (at 33 tokens and more a tile of 64 columns: tensor memory holds four groups' sums of 32)
        if (n <= 32 && (out.world == 1 || out.scatter_per)) return gemm_few(ctx, w, operand, n, terms, out, aux, epilogue);
        if (n <= 32) return launch_gemm<32, SIDE_BY_SIDE>(ctx, w, operand, n, terms, out, aux, epilogue);
        if (n <= 64) return launch_gemm<64, SIDE_BY_SIDE>(ctx, w, operand, n, terms, out, aux, epilogue);
        if (n <= 128) return (terms == 1 ? launch_gemm<128, ONE_TERM> : launch_gemm<128, SIDE_BY_SIDE>)(ctx, w, operand, n, terms, out, aux, epilogue);
        // Above that, tiles of 192 or 256 columns: a wave of the narrower ones lasts 0.77 of one of the wider
        // when it is the only one ([18944, 5120], 148 tiles: 36.5 us and 47.4; K = 17408: 116 and 150), 0.82 in a
        // row of them (three quarters of the columns, an activations' ring of four stages instead of three), so
        // the waves decide: [17408, 5120] by 131 bf16 tokens 51.9 us in tiles of 256 and 41.5 of 192, by 384 94.0 and
        // 76.9; [5120, 17408] by 131 64.4 and 54.6; by 2048 tokens 256 takes eight waves, 192 eleven.
        auto wide = [&](auto mode) {
            constexpr int M = decltype(mode)::value;
            if (out.world == 1 && 0.82 * gemm_time<192, M>(ctx, w, n, terms) < gemm_time<256, M>(ctx, w, n, terms))
                return launch_gemm<192, M>(ctx, w, operand, n, terms, out, aux, epilogue);
            return launch_gemm<256, M>(ctx, w, operand, n, terms, out, aux, epilogue);
        };
        return terms == 1 ? wide(std::integral_constant<int, ONE_TERM>()) : wide(std::integral_constant<int, TWO_PASSES>());
    }
    // few tokens, or long rows: drained every K block, for the groups' precision (gemm_takes)
    auto dense = [&](auto fmt) {
        constexpr int F = decltype(fmt)::value;
        if (whole <= DENSE_FEW || w.cols > DENSE_ROWS)
            return launch_dense<F, 64, TWO_PASSES>(ctx, w, operand, n, terms, out, aux, epilogue, whole);
        if (n <= 128) return launch_dense<F, 128, SIDE_BY_SIDE>(ctx, w, operand, n, terms, out, aux, epilogue, whole);
        // Tiles of 192 or 256 columns by their waves, as Q4_K's: [12288, 5120] Q6_K by 192 f32 tokens 128 us in tiles of 256,
        // 100 of 192, by 384 206 and 165, by 256 129 and 166; [5120, 5120] Q8_0 by 130 52 and 40, by bf16 ones 31 and 29.
        auto wide = [&](auto mode) {
            constexpr int M = decltype(mode)::value;
            if (0.82 * dense_time<F, 192, M>(ctx, w, n, terms) < dense_time<F, 256, M>(ctx, w, n, terms))
                return launch_dense<F, 192, M>(ctx, w, operand, n, terms, out, aux, epilogue, whole);
            return launch_dense<F, 256, M>(ctx, w, operand, n, terms, out, aux, epilogue, whole);
        };
        return terms == 1 ? wide(std::integral_constant<int, ONE_TERM>()) : wide(std::integral_constant<int, TWO_PASSES>());
    };
    return w.fmt == Q6_K ? dense(std::integral_constant<int, Q6_K>()) : dense(std::integral_constant<int, Q8_0>());
}

}  // namespace dwim
