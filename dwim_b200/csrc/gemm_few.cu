// The product of 9 to 32 tokens with a Q4_K matrix: the tensor cores are nearly idle at so few columns and the time
// is the weights', from HBM through their decode into the operand.  The arithmetic is gemm.cu's (exact products
// sc*q * x into the tensor cores' fp32 accumulators, the minimums as two terms, d applied in fp32 at the drain); what
// differs is where the decoded weights go and how the work is dealt:
//   - The A operand lies in tensor memory (tcgen05.st by the thread that owns the row, tcgen05.mma reads it there).
//     In shared memory a unit's 64 KB were written once and read by every MMA: 32 cycles of its bandwidth each, and
//     the stores' bank conflicts with them.
//   - A warp decodes a row's whole unit, not one K block of it: the block's header, its barriers and the loop are
//     paid once for 256 weights instead of 64.  16 worker warps are four groups (a warp per lane quadrant of tensor
//     memory) that take every fourth unit each and keep sums of their own, added at the end in group order.
//   - A group's A slots (32 columns: a K block; and the unit's minimums) are its own, so is its accumulator.
//   - The quants enter centred, sc*(q - 8), and the minimums' factors take the difference: the accumulator rounds by
//     truncation at the size of its partial sums, which are half as large so.  The two terms of an f32 activation take
//     turns on it (2-norm error over the result's 5.7e-7 by f32 and 1.6e-7 by bf16 activations; 1.0e-6 and 3.4e-7 with
//     the quants as they are; 7.0e-7 and 4.0e-7 in gemm.cu's kernel).
//   warps 16-19  MMA issuers, one a group (one lane each): a hand-over takes such a warp 400 to 500 cycles of waits,
//                MMAs and commits, five of them a unit; one warp for all groups was what bound the kernel.
//   warps 20, 21 activations' producers (one thread each, two groups'): stages of one or two K blocks, both terms in one
//                box (a copy takes such a thread 300 cycles: [17408, 5120] by 32 tokens 26.1 us with one for all, 23.0 so)
//   warp 22      the means' producer
//   warp 23      packed weights' producer
// All rings are dealt to the groups in turn (stage % 4), so that a group waits for phases of its own alone: of a
// barrier that others' phases pass it could miss two, and take an old one for the one it waits for.
// Bound by the workers' chain and issue (1053 instructions a worker and unit; issue slots 61 %, ALU 39 %, DRAM 2.8 TB/s).
// [17408, 5120] by 16 f32 tokens 24.2 us in gemm.cu's kernel, 18.4 here (31.7 with one MMA warp), by 32 25.5 and 23.0; [5120, 17408] by 16
// 28.6 and 20.7; a layer of 16 tokens 156 and 122.
// Every mbarrier wait is bounded (ptx.cuh).
#include "gemm.cuh"

namespace dwim {

namespace {

constexpr int GROUPS = 4;
constexpr int FEW_MMA_WARP = 16, FEW_X_WARP = 20, FEW_MEANS_WARP = 22, FEW_RAW_WARP = 23, FEW_THREADS = 768;
constexpr int FEW_WORKER_REGS = 104, FEW_OTHER_REGS = 32;      // of 80 at launch
static_assert(512 * FEW_WORKER_REGS + 256 * FEW_OTHER_REGS <= FEW_THREADS * 80, "a warpgroup would wait for registers that nobody gives up");

template <int N> struct FewCfg {
    static constexpr int SLOTS = 2;                                  // A slots of a group, K block g in slot g % 2
    static constexpr int SLOT_COLS = BK / 2, MIN_COLS = 16;          // and the minimums' own
    static constexpr int ACC_COLS = GROUPS * N, GROUP_COLS = SLOTS * SLOT_COLS + MIN_COLS;
    static_assert(ACC_COLS + GROUPS * GROUP_COLS <= 512, "tensor memory");
    static constexpr int STAGE_KB = N == 16 ? 2 : 1;                 // K blocks of a B stage: [term][K block][N][64]
    static constexpr int TILE_BYTES = N * BK * 2, TERM_BYTES = STAGE_KB * TILE_BYTES, B_BYTES = 2 * TERM_BYTES, MIN_BYTES = N * 32;
    static constexpr int B_STAGES = 8, MIN_STAGES = 8, RAW_STAGES = 8;
    static_assert(B_STAGES % GROUPS == 0 && MIN_STAGES % GROUPS == 0 && RAW_STAGES % GROUPS == 0, "a stage belongs to a group");
    static constexpr int RINGS = B_STAGES * B_BYTES + MIN_STAGES * MIN_BYTES + RAW_STAGES * RAW_BYTES;
    static constexpr int SMEM = BAR_BYTES + RINGS + 1024;            // + alignment slack
    static_assert(SMEM <= MAX_SMEM, "the rings do not fit shared memory");
    static constexpr int owned(int s) { return (N + s - 1) / s; }    // columns that one of s blocks finishes
    static constexpr bool split_fits(int s) { return s * GROUPS * owned(s) * TILE_M * 4 <= RINGS; }
    static_assert(split_fits(1) && split_fits(MAX_SPLIT), "the groups' sums do not fit the rings");
};

struct FewArgs {
    size_t rows, n, units;
    int terms, epi, split_k;
    OutSpec out;
    const float *tok_scale, *aux;
    uint32_t *status;
};

// D[tmem] (+)= A[tmem] * B[smem desc]
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 db;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t"
        "}\n" ::"r"(d),
        "r"(a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"((uint32_t)acc)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// A row's scales of a unit.  W = d*sc*q - dmin*m enters as s * (sc*(q - 8)*2^-e + (8*sc*2^-e - dmin/s*m)) with
// s = d*2^e (q4k_fold).
struct FewScales {
    uint32_t unit;             // s, a float's bits
    uint32_t power;            // 2^-e as two halves; zero drops the main operand
    float by;                  // -32 * dmin / s
};
__device__ __forceinline__ FewScales few_scales(const uint4 &hdr) {
    const Q4kFold f = q4k_fold<true>(hdr.x);
    const float dmin32 = 32.0f * h2f_hi(hdr.x);
    const float s = f.zero ? dmin32 : h2f_lo(hdr.x) * __uint_as_float((uint32_t)(127 + f.e) << 23);
    FewScales k;
    k.unit = __float_as_uint(s);
    const uint32_t p = f.zero ? 0u : (f.e <= 14 ? (uint32_t)(15 - f.e) << 10 : 1u << (24 - f.e));
    k.power = p | (p << 16);
    k.by = f.zero ? -1.0f : -(dmin32 / s);
    return k;
}
// The eight 6-bit scales or minimums of a header as bytes: 0..3 and 4..7.
__device__ __forceinline__ uint32_t few_sixes(const uint4 &hdr, bool min, int part) {
    const uint32_t own = min ? hdr.z : hdr.y, low = min ? hdr.w >> 4 : hdr.w;
    return part ? (low & 0x0f0f0f0fu) | ((own >> 2) & 0x30303030u) : own & 0x3f3f3f3fu;
}
// The unit's minimums operand: 256*sc_j*2^-e + by*m_j as two f16 terms, value and rounding remainder, K elements
// (hi 0..7, hi 0..7 | lo 0..7, lo 0..7).
__device__ __forceinline__ void few_mins(const uint4 &hdr, const FewScales &k, uint32_t (&r)[16]) {
    const float p = 256.0f * h2f_lo(k.power);
#pragma unroll
    for (int part = 0; part < 2; part++) {
        const uint32_t m4 = few_sixes(hdr, true, part), s4 = few_sixes(hdr, false, part);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            float v[2];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                // byte -> float through the 2^23 magic number
                const float m = __uint_as_float(prmt(m4, 0x4B000000u, 0x7650 + 2 * i + j)) - 8388608.0f;
                const float sc = __uint_as_float(prmt(s4, 0x4B000000u, 0x7650 + 2 * i + j)) - 8388608.0f;
                v[j] = fmaf(k.by, m, p * sc);
            }
            const uint32_t hi = f16x2_rn(v[0], v[1]), lo = f16x2_rn(v[0] - h2f_lo(hi), v[1] - h2f_hi(hi));
            r[2 * part + i] = r[4 + 2 * part + i] = hi;
            r[8 + 2 * part + i] = r[12 + 2 * part + i] = lo;
        }
    }
}
// K block g of the row as halves sc*(q - 8)*2^-e in the activations' order, its two sub-blocks.
__device__ __forceinline__ void few_decode(const uint4 &hdr, const FewScales &k, uint32_t raw_row, int g, uint32_t (&r)[2][16]) {
    const uint4 q0 = lds128(raw_row + 16 + 32 * g), q1 = lds128(raw_row + 32 + 32 * g);
    const uint32_t words[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    const uint32_t s4 = few_sixes(hdr, false, g >> 1);
    // byte b as 1024 + b twice; 0x6408 = 1032, 0x5480 = 72, 0x5400 | q << 4 = 64 + q
    const uint32_t sa = hmul2(hsub2(prmt(s4, 0x64006400u, g & 1 ? 0x5252u : 0x5050u), H2_1024), k.power);
    const uint32_t sb = hmul2(hsub2(prmt(s4, 0x64006400u, g & 1 ? 0x5353u : 0x5151u), H2_1024), k.power);
    const uint32_t sb72 = hmul2(sb, 0xD480D480u);
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const uint32_t w = words[c], s = w >> 8;
        r[0][2 * c] = hmul2(hsub2(lop3_and_or(w, 0x000f000fu, H2_1024), 0x64086408u), sa);
        r[0][2 * c + 1] = hmul2(hsub2(lop3_and_or(s, 0x000f000fu, H2_1024), 0x64086408u), sa);
        r[1][2 * c] = hfma2(lop3_and_or(w, 0x00f000f0u, H2_64), sb, sb72);
        r[1][2 * c + 1] = hfma2(lop3_and_or(s, 0x00f000f0u, H2_64), sb, sb72);
    }
}

template <int N>
__global__ void __launch_bounds__(FEW_THREADS, 1)
gemm_few_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                const __grid_constant__ CUtensorMap tmap_m, const __grid_constant__ FewArgs a) {
    using C = FewCfg<N>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    // barriers, 8 bytes each; a group's slots side by side
    const uint32_t afull0 = base, aempty0 = base + 64, mfull0 = base + 128, mempty0 = base + 160, accfull0 = base + 192, accempty0 = base + 224;
    const uint32_t bfull0 = base + 256, bempty0 = base + 320, minfull0 = base + 384, minempty0 = base + 448, rawfull0 = base + 512,
                   rawempty0 = base + 576, tmem_slot = base + 640;
    static_assert(GROUPS * C::SLOTS <= 8 && C::B_STAGES <= 8 && C::MIN_STAGES <= 8 && C::RAW_STAGES <= 8, "the barriers' places");
    const uint32_t bstage0 = base + BAR_BYTES, min0 = bstage0 + C::B_STAGES * C::B_BYTES, raw0 = min0 + C::MIN_STAGES * C::MIN_BYTES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split_k = a.split_k, rank = (int)(blockIdx.x % split_k);
    const int row0 = (int)(blockIdx.x / split_k) * TILE_M;
    const int ub = (int)a.units * rank / split_k, units = (int)a.units * (rank + 1) / split_k - ub;
    if (threadIdx.x == 0) {
        for (int s = 0; s < GROUPS * C::SLOTS; s++) {
            mbar_init(afull0 + 8 * s, 4);                // a group's warps
            mbar_init(aempty0 + 8 * s, 1);               // the MMA warp's commit
        }
        for (int s = 0; s < GROUPS; s++) {
            mbar_init(mfull0 + 8 * s, 4);
            mbar_init(mempty0 + 8 * s, 1);
            mbar_init(accfull0 + 8 * s, 1);
            mbar_init(accempty0 + 8 * s, 4);
        }
        for (int s = 0; s < C::B_STAGES; s++) {
            mbar_init(bfull0 + 8 * s, 1);
            mbar_init(bempty0 + 8 * s, 1);
        }
        for (int s = 0; s < C::MIN_STAGES; s++) {
            mbar_init(minfull0 + 8 * s, 1);
            mbar_init(minempty0 + 8 * s, 1);
        }
        for (int s = 0; s < C::RAW_STAGES; s++) {
            mbar_init(rawfull0 + 8 * s, 1);
            mbar_init(rawempty0 + 8 * s, 4);             // the unit's group
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == FEW_MMA_WARP) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = lds32(tmem_slot);
    griddep_launch();

    // (A warpgroup's warps trade their registers at one instruction.  The workers' branch first: behind the others' the
    // compiler made a layer of 16 tokens 125 us of 122.)
    if (warp < N_WORKERS) {
        regs_inc<FEW_WORKER_REGS>();
        const int quad = warp & 3, i = warp >> 2, rl = quad * 32 + lane;      // i: the group
        const uint32_t lanes = tmem_base + ((uint32_t)(quad * 32) << 16);
        const uint32_t slots = lanes + C::ACC_COLS + i * C::GROUP_COLS, sums = lanes + i * N;
        const uint32_t aempty = aempty0 + 8 * i * C::SLOTS, afull = afull0 + 8 * i * C::SLOTS;
        float acc[N];      // the row's sums over this group's units
#pragma unroll
        for (int j = 0; j < N; j++) acc[j] = 0.0f;
        uint32_t turn = 0;            // of the group's units
        float scale = 0.0f;           // of the unit before
        // A block is handed over once the next one is decoded: its stores are through by then.
        auto hand_over = [&](uint32_t full) {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(full);
        };
        auto drain = [&]() {      // the unit before
            mbar_wait_parked(accfull0 + 8 * i, turn ^ 1, a.status, 0x4000u);
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < N / 16; c++) {
                uint32_t v[16];
                tmem_ld16(sums + c * 16, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; j++) acc[16 * c + j] = fmaf(scale, __uint_as_float(v[j]), acc[16 * c + j]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(accempty0 + 8 * i);
        };
        for (int u = i; u < units; u += GROUPS, turn ^= 1) {
            const int rs = u % C::RAW_STAGES;
            const bool before = u >= GROUPS;
            mbar_wait_parked(rawfull0 + 8 * rs, (u / C::RAW_STAGES) & 1, a.status, 0x400u);
            const uint32_t raw = raw0 + rs * RAW_BYTES + rl * 144;
            const uint4 hdr = lds128(raw);
            const FewScales k = few_scales(hdr);
            uint32_t r[2][16];
            few_mins(hdr, k, r[0]);
            if (before) hand_over(afull + 8);      // the unit before's last K block
            mbar_wait_parked(mempty0 + 8 * i, turn ^ 1, a.status, 0x800u);
            tc_fence_after();
            tmem_st16(slots + C::SLOTS * C::SLOT_COLS, r[0]);
#pragma unroll
            for (int g = 0; g < KBLOCKS; g++) {
                few_decode(hdr, k, raw, g, r);
                if (g == KBLOCKS - 1) {      // (every lane has its words)
                    __syncwarp();
                    if (lane == 0) mbar_arrive(rawempty0 + 8 * rs);
                }
                hand_over(g == 0 ? mfull0 + 8 * i : afull + 8 * (~g & 1));
                if (g == 0 && before) drain();
                mbar_wait_parked(aempty + 8 * (g & 1), ~g >> 1 & 1, a.status, 0x800u);      // the slot's MMAs are done
                tc_fence_after();
                tmem_st16(slots + (g & 1) * C::SLOT_COLS, r[0]);
                tmem_st16(slots + (g & 1) * C::SLOT_COLS + 16, r[1]);
            }
            scale = __uint_as_float(k.unit);
        }
        if (i < units) hand_over(afull + 8);
        // what the epilogue reads, ahead of the last unit's drains
        griddep_wait();   // the kernel ahead may still read or write `out` and `aux`
        const size_t row = (size_t)row0 + rl;
        const EmitTo to = emit_to(a.out, a.aux, a.epi, row);
        // this thread finishes its row's columns rank + split_k * (i + GROUPS * j)
        float y[N / GROUPS];
#pragma unroll
        for (int j = 0; j < N / GROUPS; j++) {
            const size_t c = rank + split_k * (i + GROUPS * j);
            y[j] = 0.0f;
            if (a.epi != EPI_STORE && row < a.rows && c < a.n) y[j] = a.epi == EPI_ADD ? to.own[c * to.pitch] : to.aux_row[c * a.rows];
        }
        if (i < units) drain();
        // the groups' and the cluster's sums meet in the finishing block's rings, which nothing uses any more
        const int own = C::owned(split_k);
        const uint32_t rings = bstage0;
        if (split_k > 1) cluster_sync();
        else asm volatile("bar.sync 1, 512;" ::: "memory");
#pragma unroll
        for (int j = 0; j < N; j++) {
            const uint32_t at = rings + (((rank * GROUPS + i) * own + j / split_k) * TILE_M + rl) * 4;
            if (split_k > 1) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_addr(at, j % split_k)), "f"(acc[j]) : "memory");
            else sts32f(at, acc[j]);
        }
        if (split_k > 1) cluster_sync();
        else asm volatile("bar.sync 1, 512;" ::: "memory");
        if (row < a.rows) {
#pragma unroll
            for (int j = 0; j < N / GROUPS; j++) {
                const int k = i + GROUPS * j;
                const size_t c = rank + split_k * k;
                if (c >= a.n || c >= (size_t)N) break;
                float v = 0.0f;
                for (int r = 0; r < split_k * GROUPS; r++) v += lds32f(rings + ((r * own + k) * TILE_M + rl) * 4);
                v *= a.tok_scale[c];
                if (a.epi == EPI_ADD) v += y[j];
                else if (a.epi == EPI_SWIGLU) v = silu_mul_f(v, y[j]);
                to.own[c * to.pitch] = v;
            }
        }
    } else if (warp < FEW_X_WARP) {
        regs_dec<FEW_OTHER_REGS>();
        constexpr uint32_t idesc = idesc_f16(TILE_M, N);
        const int i = __shfl_sync(0xffffffffu, warp, 0) - FEW_MMA_WARP;
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0), b_lo = desc_lo_sw128(bstage0);
        const uint32_t d = tm + i * N, a0 = tm + C::ACC_COLS + i * C::GROUP_COLS, afull = afull0 + 8 * i * C::SLOTS, aempty = aempty0 + 8 * i * C::SLOTS;
        int bs = i;
        uint32_t bturn = 0, turn = 0;
        // the lanes wait for several barriers at once: lane % 4 chooses
        auto wait = [&](uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, uint32_t b2, uint32_t p2) {
            const int l = lane & 3;
            mbar_wait_all(l == 0 ? b0 : l == 1 ? b1 : b2, l == 0 ? p0 : l == 1 ? p1 : p2, a.status, 0x100u);
            tc_fence_after();
        };
        for (int u = i; u < units; u += GROUPS, turn ^= 1) {
            const int ms = u % C::MIN_STAGES;
            // the minimums, terms (hi, hi | lo, lo) against the means' (hi, lo) twice, open the unit's sums
            wait(accempty0 + 8 * i, turn ^ 1, minfull0 + 8 * ms, (u / C::MIN_STAGES) & 1, mfull0 + 8 * i, turn);
            if (elect_one()) {
                const uint32_t at = a0 + C::SLOTS * C::SLOT_COLS;
                const uint64_t bd = smem_desc_plain(min0 + ms * C::MIN_BYTES, N * 16);
                umma_ts(d, at, (uint32_t)bd, (uint32_t)(bd >> 32), idesc, false);
                umma_ts(d, at + 8, (uint32_t)bd, (uint32_t)(bd >> 32), idesc, true);
                umma_commit(minempty0 + 8 * ms);
                umma_commit(mempty0 + 8 * i);
            }
            __syncwarp();
#pragma unroll
            for (int g = 0; g < KBLOCKS; g++) {
                const uint32_t ab = afull + 8 * (g & 1), bb = bfull0 + 8 * bs, par = g >> 1;      // a slot is used twice a unit
                if (g % C::STAGE_KB == 0) wait(bb, bturn, bb, bturn, ab, par);
                else wait(ab, par, ab, par, ab, par);
                if (elect_one()) {
                    const uint32_t at = a0 + (g & 1) * C::SLOT_COLS;
                    const uint32_t bd = b_lo + ((bs * C::B_BYTES + g % C::STAGE_KB * C::TILE_BYTES) >> 4);
                    if (a.terms == 2) {       // the remainders first
#pragma unroll
                        for (int k = 0; k < BK / 16; k++) umma_ts(d, at + 8 * k, bd + (C::TERM_BYTES >> 4) + 2 * k, DESC_HI_SW128, idesc, true);
                    }
#pragma unroll
                    for (int k = 0; k < BK / 16; k++) umma_ts(d, at + 8 * k, bd + 2 * k, DESC_HI_SW128, idesc, true);
                    umma_commit(aempty + 8 * (g & 1));
                    if (g % C::STAGE_KB == C::STAGE_KB - 1) umma_commit(bempty0 + 8 * bs);
                    if (g == KBLOCKS - 1) umma_commit(accfull0 + 8 * i);
                }
                __syncwarp();
                if (g % C::STAGE_KB == C::STAGE_KB - 1 && (bs += GROUPS) >= C::B_STAGES) bs = i, bturn ^= 1;
            }
        }
    } else {
        regs_dec<FEW_OTHER_REGS>();
        if (warp == FEW_X_WARP || warp == FEW_X_WARP + 1) {
            griddep_wait();   // the operand comes from the prologue kernel just ahead
            if (elect_one()) {
                int turn = 1, row = 0;      // a group's stages are used in turn
                for (int u0 = 2 * (warp - FEW_X_WARP); u0 < units; u0 += GROUPS) {
                    const int last = min(u0 + 2, units);
                    for (int g = 0; g < KBLOCKS; g += C::STAGE_KB) {
                        for (int u = u0; u < last; u++) {
                            const int bs = row * GROUPS + u % GROUPS;
                            mbar_wait_parked(bempty0 + 8 * bs, turn, a.status, 0x20u);
                            mbar_expect_tx(bfull0 + 8 * bs, C::TERM_BYTES * a.terms);
                            tma_load_4d(bstage0 + bs * C::B_BYTES, &tmap_x, 0, 0, KBLOCKS * (ub + u) + g, 0, bfull0 + 8 * bs);
                        }
                        if (++row == C::B_STAGES / GROUPS) row = 0, turn ^= 1;
                    }
                }
            }
        } else if (warp == FEW_MEANS_WARP) {
            griddep_wait();
            if (elect_one()) {
                for (int u = 0; u < units; u++) {
                    const int ms = u % C::MIN_STAGES;
                    mbar_wait_parked(minempty0 + 8 * ms, ((u / C::MIN_STAGES) & 1) ^ 1, a.status, 0x40u);
                    mbar_expect_tx(minfull0 + 8 * ms, C::MIN_BYTES);
                    tma_load_3d(min0 + ms * C::MIN_BYTES, &tmap_m, 0, 0, (ub + u) * 2, minfull0 + 8 * ms);      // [hi, lo][token][8]
                }
            }
        } else if (warp == FEW_RAW_WARP) {
            if (elect_one()) {
                int rs = 0, turn = 1;
                for (int u = 0; u < units; u++) {
                    mbar_wait_parked(rawempty0 + 8 * rs, turn, a.status, 0x10u);
                    mbar_expect_tx(rawfull0 + 8 * rs, TILE_M * 144);
                    tma_load_2d(raw0 + rs * RAW_BYTES, &tmap_w, (ub + u) * 144, row0, rawfull0 + 8 * rs);
                    if (++rs == C::RAW_STAGES) rs = 0, turn ^= 1;
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
    if (warp == FEW_MMA_WARP) tmem_dealloc(tmem_base, 512);
}

template <int N>
int launch_few(dwim_b200_ctx *ctx, const WeightView &w, const __half *operand, size_t n, int terms, const OutSpec &out, const float *aux,
               int epi) {
    using C = FewCfg<N>;
    const size_t units = w.cols / 256;
    CUtensorMap tw, tx, tm;
    int rc;
    if ((rc = encode_2d(ctx, &tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, w.quants, w.qpitch, w.rows, w.qpitch, 144, TILE_M,
                        CU_TENSOR_MAP_SWIZZLE_NONE, "weight")))
        return rc;
    // [terms][K blocks][n][64], tokens past the last read as zeros
    const uint64_t xdims[4] = {BK, n, w.cols / BK, (uint64_t)terms}, xpitch[3] = {w.cols * 2, BK * 2, n * w.cols * 2};
    const uint32_t xbox[4] = {BK, N, C::STAGE_KB, (uint32_t)terms};
    if ((rc = encode_nd(ctx, &tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, operand, 4, xdims, xpitch, xbox, CU_TENSOR_MAP_SWIZZLE_128B, "activation")))
        return rc;
    // [units][hi, lo][n][8]
    const uint64_t mdims[3] = {8, n, units * 2}, mpitch[2] = {units * 32, 16};
    const uint32_t mbox[3] = {8, N, 2};
    if ((rc = encode_nd(ctx, &tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, operand + terms * n * w.cols, 3, mdims, mpitch, mbox, CU_TENSOR_MAP_SWIZZLE_NONE,
                        "means")))
        return rc;
    const float *tok_scale = reinterpret_cast<const float *>(operand + (terms * w.cols + units * 16) * n);
    FewArgs a{w.rows, n, units, terms, epi, 1, out, tok_scale, aux, ctx->status};
    auto kern = gemm_few_kernel<N>;
    static std::atomic<bool> configured[64] = {};
    constexpr int SHARES = 512 * FEW_WORKER_REGS + 256 * FEW_OTHER_REGS;
    if ((rc = configure_gemm(ctx, kern, C::SMEM, FEW_THREADS, SHARES, configured[ctx->device & 63]))) return rc;
    static std::atomic<int> known[64][MAX_SPLIT + 1] = {};
    const long tiles = (long)((w.rows + TILE_M - 1) / TILE_M);
    // The prices of gemm.cu's kernel hold for this one: of the splits from 1 to 8 of ten shapes, by 9, 16 and 32 tokens in
    // one and two terms, the choice is within 2 % of the best for eight ([10240, 5120] by 16 17.1 us alone, 23.8 by two
    // blocks; [6144, 5120] 15.8 and 12.7; [5120, 17408] 43.4, 26.4 and 20.9 by three), and a block too far where the
    // tiles are few: [1024, 5120] takes seven for 7.7 us where five and six take 7.0, [3000, 2048] four for 7.8, two 7.5.
    a.split_k = pick_split(ctx, kern, FEW_THREADS, (size_t)C::SMEM, C::split_fits, SplitCost{3.0, 6.5}, known, tiles, (int)units, 1.0);
    const bool dependent = !ctx->weights_written;   // see dwim_b200_ctx::weights_written
    DWIM_CUDA(ctx, launch_clustered(dependent, (unsigned)a.split_k, kern, dim3((unsigned)(tiles * a.split_k)), dim3(FEW_THREADS),
                                    (size_t)C::SMEM, ctx->stream, tw, tx, tm, a));
    ctx->weights_written = false;
    DWIM_LAUNCHED(ctx);
    return 0;
}

}  // namespace

int gemm_few(dwim_b200_ctx *ctx, const WeightView &w, const __half *operand, size_t n, int terms, const OutSpec &out, const float *aux,
             int epi) {
    return (n <= 16 ? launch_few<16> : launch_few<32>)(ctx, w, operand, n, terms, out, aux, epi);
}

}  // namespace dwim
