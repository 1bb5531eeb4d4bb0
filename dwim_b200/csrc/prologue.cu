// Activation prologue: f32 activations -> the operand forms the matmul
// kernels read.  The reference does the same with its f16 shadow buffers
// (`halves`, gpu/cuda/mod.rs:313-384; to_f16.cu:6-18): convert once, reuse for
// every matmul that takes the same input.  Two forms: int8 digit planes per
// 256-wide unit for the small-M kernel (up to eight tokens), and f16 rows with
// sub-block means and a scale per token for the tensor-core kernels; either
// can be written by the same launch that applies the RMS norm in front of the
// product (rmsnorm.cu:11-58).
#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"

namespace dwim {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The largest magnitude of a warp's values; as fmaxf, a NaN is passed over.
__device__ __forceinline__ float warp_absmax(float v) {
    float m;
    asm volatile("redux.sync.max.abs.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(v));
    return m;
}

// ---- int8 digit planes (the small-M kernel's int8 routines) --------------------------------
// A unit's 256 activations of a token share one exponent e (|x| < 2^e for all of
// them) and become fixed point with P signed base-256 digits, Y = rint(x * 2^(8P-2-e))
// = sum_p d_p * 256^(P-1-p), each digit in [-128, 127] (the leading one in [-64, 64]).
// P = 4 for one and two tokens (31 bits: an activation within 2^-6 of the unit's
// largest is exact, a smaller one is rounded at 2^-31 of the largest), P = 3 for
// three to eight (23 bits: rounded at 2^-23 of the unit's largest).  A unit of
// plane p's digit is worth 2^(e-6-8p).  Columns of the int8 MMA:
//   P = 4: column = 4*token + plane   (both tokens' planes share one 8-column tile)
//   P = 3: column = plane*n + token   (tile p of the MMA holds plane p of every token)
size_t panel_i8_bytes(size_t cols, size_t n) { return ((cols + 255) / 256) * (size_t)i8_unit_bytes(i8_planes((int)n) * (int)n); }

// What one thread does with its activation once the unit's largest magnitude is
// known: the digits, their per-sub-block sums, the planes' worths.  `lane` and
// `j` are the thread's place in its sub-block and the sub-block's in the unit.
template <int P>
__device__ __forceinline__ void i8_digits(float v, float m, int t, int n, int j, int lane, bool first, uint8_t *blob) {
    const int nc = P * n;
    // |x| < 2^e; floored so that the planes' worths stay normal floats
    int e = m > 0.0f ? (int)((__float_as_uint(m) >> 23) & 0xffu) - 126 : -90;
    if (e < -90) e = -90;
    if (e > 100) e = 100;
    // v * 2^(8P-2-e) in two steps: either factor is a normal float
    const int s = 8 * P - 2 - e, s1 = s >> 1;
    const float up1 = __uint_as_float((uint32_t)(127 + s1) << 23), up2 = __uint_as_float((uint32_t)(127 + s - s1) << 23);
    const float lim = (float)(1 << (8 * P - 2));
    int y = __float2int_rn(fminf(fmaxf(v * up1 * up2, -lim), lim));   // |y| <= 2^(8P-2); the clamp only matters for inf
    int d[P];
#pragma unroll
    for (int p = P - 1; p > 0; p--) {
        d[p] = ((y + 128) & 255) - 128;
        y = (y - d[p]) >> 8;
    }
    d[0] = y;
#pragma unroll
    for (int p = 0; p < P; p++) {
        const int col = P == 4 ? 4 * t + p : p * n + t;
        blob[(j * nc + col) * 32 + lane] = (uint8_t)(int8_t)d[p];
        const int sum = __reduce_add_sync(0xffffffffu, d[p]);
        if (lane == 0) {
            const int b = ((sum + 64) & 127) - 64, a = (sum - b) >> 7;   // sum = 128*a + b
            blob[256 * nc + col * 16 + j] = (uint8_t)(int8_t)a;
            blob[256 * nc + col * 16 + 8 + j] = (uint8_t)(int8_t)b;
        }
        if (first) reinterpret_cast<float *>(blob + 272 * nc)[col] = __uint_as_float((uint32_t)(127 + e - 6 - 8 * p) << 23);
    }
}

// One block per (unit, token); warp j owns sub-block j.  Tokens are taken n at a time, every group
// with panels of its own.
template <int P>
__global__ void __launch_bounds__(256) panel_i8_kernel(const float *__restrict__ x, size_t cols, int n, uint8_t *__restrict__ panels) {
    // the small-M kernel launched next may start streaming its weights now; the
    // panels may still be read, and x written, by the kernel ahead
    griddep_launch();
    griddep_wait();
    const int u = blockIdx.x, t = blockIdx.y % n, tid = threadIdx.x, j = tid >> 5, lane = tid & 31;
    uint8_t *blob = panels + ((size_t)(blockIdx.y / n) * gridDim.x + u) * i8_unit_bytes(P * n);
    const size_t k = (size_t)u * 256 + tid;
    const float v = k < cols ? x[(size_t)blockIdx.y * cols + k] : 0.0f;
    // the unit's largest magnitude
    __shared__ float wmax[8];
    const float m0 = warp_absmax(v);
    if (lane == 0) wmax[j] = m0;
    __syncthreads();
    float m = wmax[0];
#pragma unroll
    for (int i = 1; i < 8; i++) m = fmaxf(m, wmax[i]);
    i8_digits<P>(v, m, t, n, j, lane, tid == 0, blob);
}

// The same with the RMS norm in front (Cpu::rmsnorm, gpu/cpu.rs:157-166); the f32
// result goes to xout.  Bound by latency alone (20 KB a token), and every product
// of the layer waits for it: a token's row is dealt to a cluster of up to eight
// blocks, four units a block and round, whose sums of squares meet in shared
// memory.  (The row is read before the blocks meet and written after, by the
// threads that read it: xout may be x.)  A single block per token took 13 us for
// rows of 5120; a decoder layer with two norms became 16 us shorter.  The cluster's
// first meeting, which says that the peers run, has the row's loads between its halves.
constexpr int NORM_CLUSTER = 8;
template <int P>
__global__ void __launch_bounds__(1024) normalize_i8_kernel(const float *x, const float *__restrict__ weight, float eps, float *xout,
                                                            size_t cols, int n, uint8_t *__restrict__ panels) {
    const int t = blockIdx.y, rank = blockIdx.x, ranks = gridDim.x;
    if (ranks > 1) cluster_arrive();
    griddep_launch();
    griddep_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, j = warp & 7, uu = tid >> 8;
    __shared__ float part[32];
    __shared__ float sums[NORM_CLUSTER];
    __shared__ float wmax[32];
    const float *src = x + (size_t)t * cols;
    const size_t first = (size_t)rank * 1024 + tid, step = (size_t)ranks * 1024;
    const float v0 = first < cols ? src[first] : 0.0f, w0 = first < cols ? weight[first] : 0.0f;
    float ss = v0 * v0;
    for (size_t k = first + step; k < cols; k += step) ss += src[k] * src[k];
    ss = warp_sum(ss);
    if (lane == 0) part[warp] = ss;
    __syncthreads();
    float total = warp_sum(part[lane]);
    if (ranks > 1) {
        // every block's sum to every block, added in rank order
        cluster_wait();                     // all of them run
        if (warp == 0 && lane < ranks) st_cluster_f32(smem_u32(sums + rank), lane, total);
        cluster_sync();
        total = sums[0];
        for (int i = 1; i < ranks; i++) total += sums[i];
    }
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(total, (float)cols), eps)));
    const size_t units = (cols + 255) / 256;
    for (size_t u0 = (size_t)rank * 4; u0 < units; u0 += (size_t)ranks * 4) {
        const size_t u = u0 + uu, k = u * 256 + (tid & 255);
        float v = 0.0f;
        if (u < units && k < cols) {
            const bool held = k == first;
            v = __fmul_rn(held ? v0 : src[k], __fmul_rn(scale, held ? w0 : weight[k]));
            xout[(size_t)t * cols + k] = v;
        }
        const float m0 = warp_absmax(v);
        if (lane == 0) wmax[warp] = m0;
        __syncthreads();
        float m = wmax[8 * uu];
#pragma unroll
        for (int i = 1; i < 8; i++) m = fmaxf(m, wmax[8 * uu + i]);
        __syncthreads();                    // wmax is rewritten in the next round
        if (u < units) i8_digits<P>(v, m, t, n, j, lane, (tid & 255) == 0, panels + u * i8_unit_bytes(P * n));
    }
}

// weight / eps / xout: null / 0 / null for a plain conversion, or the RMS norm's
// weight [cols], its epsilon and the f32 destination [n, cols] (may be x itself).
int build_panels_i8(dwim_b200_ctx *ctx, const float *x, size_t n, size_t cols, uint8_t *panels, const float *weight, float eps,
                    float *xout, size_t groups) {
    if (n == 0 || cols == 0) return 0;
    if (n > I8_MAX_TOKENS) return fail(ctx, DWIM_B200_EINVAL, "int8 panels take at most %d tokens, not %zu", I8_MAX_TOKENS, n);
    const bool dependent = !ctx->weights_written;
    const int planes = i8_planes((int)n);
    if (weight) {
        auto kern = planes == 4 ? normalize_i8_kernel<4> : normalize_i8_kernel<3>;
        const size_t blocks = (cols + 1023) / 1024;
        const unsigned ranks = (unsigned)(blocks < (size_t)NORM_CLUSTER ? blocks : (size_t)NORM_CLUSTER);
        DWIM_CUDA(ctx, launch_clustered(dependent, ranks, kern, dim3(ranks, (unsigned)n), dim3(1024), 0, ctx->stream, x, weight, eps,
                                        xout, cols, (int)n, panels));
    } else {
        auto kern = planes == 4 ? panel_i8_kernel<4> : panel_i8_kernel<3>;
        dim3 grid((unsigned)((cols + 255) / 256), (unsigned)(n * groups));
        DWIM_CUDA(ctx, launch_dependent(dependent, kern, grid, dim3(256), 0, ctx->stream, x, cols, (int)n, panels));
    }
    DWIM_LAUNCHED(ctx);
    return 0;
}

// Bytes of the GEMM's operand for n tokens (one f16 term an activation, or two when an f32 one travels as value and
// remainder): the f16 rows, the sub-block means, and one f32 scale per token.
size_t gemm_operand_bytes(size_t cols, size_t n, int split) {
    const size_t terms = split ? 2 : 1;
    return (terms * cols + cols / 256 * 16) * n * sizeof(__half) + ((n * sizeof(float) + 15) & ~size_t(15));
}

// Reductions over a block of THREADS and its cluster (`cluster` blocks share a row), every thread the
// result: the warps' values through shared memory, the blocks' through each other's, both in a fixed order.
constexpr size_t OPERAND_MAX_COLS = 51200;
struct RowScratch {
    float warps[16];
    float blocks[8];
};
template <int THREADS>
__device__ __forceinline__ float row_sum(float v, RowScratch &s, int rank, int cluster) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) s.warps[threadIdx.x >> 5] = v;
    __syncthreads();
    v = s.warps[0];
#pragma unroll
    for (int i = 1; i < THREADS / 32; i++) v += s.warps[i];
    if (cluster > 1) {
        cluster_wait();                     // opened at the kernel's start: all the row's blocks run
        if ((int)threadIdx.x < cluster) st_cluster_f32(smem_u32(s.blocks + rank), threadIdx.x, v);
        cluster_sync();
        v = s.blocks[0];
        for (int i = 1; i < cluster; i++) v += s.blocks[i];
    }
    return v;
}
// The largest of non-negative floats' bits (a NaN's are above infinity's).
template <int THREADS>
__device__ __forceinline__ uint32_t row_max(uint32_t v, RowScratch &s, int rank, int cluster, bool met) {
    v = __reduce_max_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) s.warps[threadIdx.x >> 5] = __uint_as_float(v);
    __syncthreads();
    v = __float_as_uint(s.warps[0]);
#pragma unroll
    for (int i = 1; i < THREADS / 32; i++) v = max(v, __float_as_uint(s.warps[i]));
    if (cluster > 1) {
        if (!met) cluster_wait();
        if ((int)threadIdx.x < cluster) st_cluster_f32(smem_u32(s.blocks + rank), threadIdx.x, __uint_as_float(v));
        cluster_sync();
        v = __float_as_uint(s.blocks[0]);
        for (int i = 1; i < cluster; i++) v = max(v, __float_as_uint(s.blocks[i]));
    }
    return v;
}

// Four values as f16 (hi) and what the rounding left, as f16 (lo), in the order (0, 2, 1, 3): the order the
// weights' bytes decode in; sh and sl: the terms' sums.
struct Terms {
    uint2 hi, lo;
    float sh, sl;
};
__device__ __forceinline__ uint32_t pack_f16(float a, float b) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
template <bool SPLIT> __device__ __forceinline__ Terms terms_finite(const float (&f)[4]) {
    Terms t;
    t.hi = make_uint2(pack_f16(f[0], f[2]), pack_f16(f[1], f[3]));
    const float h0 = h2f_lo(t.hi.x), h2 = h2f_hi(t.hi.x), h1 = h2f_lo(t.hi.y), h3 = h2f_hi(t.hi.y);
    t.sh = (h0 + h1) + (h2 + h3);
    if (!SPLIT) return t;
    t.lo = make_uint2(pack_f16(f[0] - h0, f[2] - h2), pack_f16(f[1] - h1, f[3] - h3));
    t.sl = (h2f_lo(t.lo.x) + h2f_lo(t.lo.y)) + (h2f_hi(t.lo.x) + h2f_hi(t.lo.y));
    return t;
}
// The same where a value may be an infinity or a NaN: clamped to f16's largest.
__device__ __noinline__ Terms terms_clamped(float f0, float f1, float f2, float f3) {
    const float f[4] = {f0, f1, f2, f3};
    uint32_t hi[4], lo[4];
    Terms t;
    t.sh = t.sl = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        hi[i] = to_f16_bits(f[i]);
        lo[i] = to_f16_bits(f[i] - from_f16_bits(hi[i]));
        t.sh += from_f16_bits(hi[i]);
        t.sl += from_f16_bits(lo[i]);
    }
    t.hi = make_uint2(hi[0] | hi[2] << 16, hi[1] | hi[3] << 16);
    t.lo = make_uint2(lo[0] | lo[2] << 16, lo[1] | lo[3] << 16);
    return t;
}

// A block per token row, or a cluster of up to eight; the row in chunks of THREADS * 4 activations (four a
// thread), dealt to the blocks in turn, R of them a block, and held in registers until its largest magnitude is known
// (all but a few of the longer forms': R = 9, rows of 17408, spills 144 bytes a thread, 232 to 240 with the norm; R = 5,
// rows of 5120, 24 to 48).
//   NORM: the row is first normalized by its root mean square and multiplied
//   by `weight` (Cpu::rmsnorm, gpu/cpu.rs:157-166: v * (scale * w) with
//   scale = 1 / sqrt(sum(v^2) / dim + eps)); the f32 result goes to `xout`.
// Then the row is scaled by a power of two 2^-e, chosen per token so that its
// largest magnitude lands in [4, 8): whatever finite activations' range, nothing
// is clamped, an activation down to 2^-16 of the token's largest keeps its
// full f16 precision (and, for f32 inputs, the f16 remainder its share), and
// the product's epilogue multiplies the token's results by 2^e (tok_scale)
// again.  (Rows of typical normalized activations, largest magnitude 4 to 8,
// are not scaled at all.  Scaling them up instead, to just below f16's
// maximum, was measured to slow the tensor-core kernel by half: the same
// kernel on larger operand magnitudes runs into the power limit earlier.)
template <bool NORM, bool SPLIT, int THREADS, int R>
__global__ void __launch_bounds__(THREADS, THREADS == 512 ? (R > 9 ? 1 : 2) : R > 3 ? 5 : 6)
gemm_operand_kernel(const float *x, const float *__restrict__ weight, float eps, float *xout, size_t cols, size_t units, int cluster, size_t n,
                    __half *__restrict__ x16, __half *__restrict__ means, float *__restrict__ tok_scale) {
    if (cluster > 1) cluster_arrive();
    // as the small-M prologues: let the product's kernel begin (it streams weights first),
    // wait for the kernel ahead, which may still read the operand or write x
    griddep_launch();
    griddep_wait();
    __shared__ RowScratch s[3];
    const int rank = (int)(blockIdx.x % cluster), k = threadIdx.x;
    const size_t t = blockIdx.x / cluster;
    const float *src = x + t * cols;
    // this thread's place in its block's chunk r; whole warps are in or out (cols is whole units)
    auto place = [&](int r) { return ((size_t)(rank + cluster * r) * THREADS + k) * 4; };
    float4 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = place(r) < cols ? *reinterpret_cast<const float4 *>(src + place(r)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (NORM) {
        float4 w[R];      // (fetched ahead of the sum where the registers last)
        constexpr bool AHEAD = R <= 3;
#pragma unroll
        for (int r = 0; r < R && AHEAD; r++)
            w[r] = place(r) < cols ? *reinterpret_cast<const float4 *>(weight + place(r)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float ssq = 0.0f;
#pragma unroll
        for (int r = 0; r < R; r++) ssq += (v[r].x * v[r].x + v[r].y * v[r].y) + (v[r].z * v[r].z + v[r].w * v[r].w);
        const float total = row_sum<THREADS>(ssq, s[0], rank, cluster);
        const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(total, (float)cols), eps)));
        float *dst = xout + t * cols;
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (!AHEAD) w[r] = place(r) < cols ? *reinterpret_cast<const float4 *>(weight + place(r)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            v[r].x = __fmul_rn(v[r].x, __fmul_rn(scale, w[r].x));
            v[r].y = __fmul_rn(v[r].y, __fmul_rn(scale, w[r].y));
            v[r].z = __fmul_rn(v[r].z, __fmul_rn(scale, w[r].z));
            v[r].w = __fmul_rn(v[r].w, __fmul_rn(scale, w[r].w));
            if (place(r) < cols) *reinterpret_cast<float4 *>(dst + place(r)) = v[r];
        }
    }
    auto largest = [&](uint32_t limit) {     // of the magnitudes whose bits are below the limit
        uint32_t m = 0;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float f[4] = {v[r].x, v[r].y, v[r].z, v[r].w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t b = __float_as_uint(f[i]) & 0x7fffffffu;
                if (b < limit) m = max(m, b);
            }
        }
        return m;
    };
    uint32_t top = row_max<THREADS>(largest(0x80000000u), s[1], rank, cluster, NORM);
    const bool finite = top < 0x7f800000u;
    if (!finite) top = row_max<THREADS>(largest(0x7f800001u), s[2], rank, cluster, true);     // a NaN is passed over
    // the largest in [2^(b-127), 2^(b-126)) for its biased exponent b; e = b - 127 - 2, at most 125 for a finite row;
    // 2^e and 2^-e are normal floats then (a row whose largest is below 2^-123 takes the nearest end).  A row with an
    // infinity or a NaN is clamped and stops at 2^100 either way.
    const int most = finite ? 125 : 100;
    const int e = top ? max(-most, min(most, (int)(top >> 23) - 129)) : 0;
    const float down = __uint_as_float((uint32_t)(127 - e) << 23);
    if (rank == 0 && k == 0) tok_scale[t] = __uint_as_float((uint32_t)(127 + e) << 23);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const size_t at = place(r);
        if (at >= cols) break;
        const float f[4] = {v[r].x * down, v[r].y * down, v[r].z * down, v[r].w * down};
        Terms y;
        if (finite) y = terms_finite<SPLIT>(f);
        else y = terms_clamped(f[0], f[1], f[2], f[3]);
        *reinterpret_cast<uint2 *>(x16 + t * cols + at) = y.hi;
        if (SPLIT) *reinterpret_cast<uint2 *>(x16 + (n + t) * cols + at) = y.lo;
        // sub-block sums over the eight threads that share it
        float sum = SPLIT ? y.sh + y.sl : y.sh;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if ((k & 7) == 0) {
            const float mean = sum * (1.0f / 32.0f);
            __half *m = means + (t * units + (at >> 8)) * 16 + ((at & 255) >> 5);
            const __half hi = to_f16_clamped(mean);
            m[0] = hi;
            m[8] = to_f16_clamped(mean - __half2float(hi));
        }
    }
}

// x: the activations [n, cols]; weight / eps / xout: null / 0 / null for a plain conversion, or the
// RMS-norm's weight [cols], its epsilon and the f32 destination [n, cols] (xout may be x itself).
int build_gemm_operand(dwim_b200_ctx *ctx, const float *x, size_t n, size_t cols, int split, __half *out, const float *weight,
                       float eps, float *xout) {
    if (n == 0 || cols == 0) return 0;
    if (cols % 256) return fail(ctx, DWIM_B200_EINVAL, "GEMM operand: %zu columns are not whole 256-weight units", cols);
    const size_t units = cols / 256, terms = split ? 2 : 1;
    __half *means = out + terms * n * cols;
    float *tok_scale = reinterpret_cast<float *>(means + n * units * 16);
    if (cols > OPERAND_MAX_COLS) return fail(ctx, DWIM_B200_EINVAL, "GEMM operand: rows of %zu activations are too long", cols);
    // A block a row once there are rows for every SM; below that as many blocks a row as there are SMs for.
    // Bound by a row's chain of load, reduction and store at few rows, by the bytes and the conversion's
    // instructions at many (the bytes of 2048 rows of 17408 f32 are 33 to 44 us).  The kernel alone, us, by cluster:
    // 16 rows of 17408 4.2 with eight blocks (9.0 with the row in one block's shared memory, as it was), 131 rows 5.9
    // with one; 16 rows of 5120 3.4 with five, 3.8 with one; 512 rows 6.6 with one, 9.0 with two; 2048 rows
    // 13.1 with one, 24 with two (a cluster's blocks start and end together); 2048 rows of 17408 51 as one
    // block of 512 threads (64 with both terms), 69 as four of 256.
    const size_t chunks = (cols + 1023) / 1024;
    size_t cluster = (size_t)ctx->sm_count / n;
    if (cluster < 1) cluster = 1;
    if (cluster > 8) cluster = 8;
    if (cluster > chunks) cluster = chunks;
    size_t each = (chunks + cluster - 1) / cluster;     // in chunks of 1024
    const bool wide = each > 5;                         // 512 threads, chunks of 2048
    if (wide) {
        each = (chunks + 2 * cluster - 1) / (2 * cluster);
        each = each <= 5 ? 5 : each <= 9 ? 9 : 13;
        cluster = ((chunks + 1) / 2 + each - 1) / each;
    } else {
        each = each <= 3 ? each : 5;
        cluster = (chunks + each - 1) / each;
    }
    auto pick = [&](auto norm, auto terms) {
        constexpr bool N = decltype(norm)::value, S = decltype(terms)::value;
        if (wide) return each == 5 ? gemm_operand_kernel<N, S, 512, 5> : each == 9 ? gemm_operand_kernel<N, S, 512, 9> : gemm_operand_kernel<N, S, 512, 13>;
        return each == 1 ? gemm_operand_kernel<N, S, 256, 1> : each == 2 ? gemm_operand_kernel<N, S, 256, 2>
               : each == 3 ? gemm_operand_kernel<N, S, 256, 3> : gemm_operand_kernel<N, S, 256, 5>;
    };
    using T = std::true_type;
    using F = std::false_type;
    auto kern = weight ? (split ? pick(T(), T()) : pick(T(), F())) : (split ? pick(F(), T()) : pick(F(), F()));
    DWIM_CUDA(ctx, launch_clustered(!ctx->weights_written, (unsigned)cluster, kern, dim3((unsigned)(n * cluster)), dim3(wide ? 512 : 256), 0,
                                    ctx->stream, x, weight, eps, xout, cols, units, (int)cluster, n, out, means, tok_scale));
    DWIM_LAUNCHED(ctx);
    return 0;
}

}  // namespace dwim
