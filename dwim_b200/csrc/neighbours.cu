// The operators that sit either side of the quantized product in the
// engine's layer (inference/qwen35/mod.rs:547, 603-605, 652-654, 1066-1068):
//   - normalize: RMS norm of the residual stream into the product's input
//     (Cuda::normalize, gpu/cuda/mod.rs:1177-1198; rmsnorm.cu:11-58).  The
//     reference writes the f16 copy its tile kernels read; here the same
//     launch writes the f32 result and the operand form the next product
//     reads, so that no separate activation prologue runs.
//   - the product with bf16 weights (matmul_bf16.cu:19-81): the small gate
//     matrices of the linear-attention layers, 48 calls per token.
//   - argmax over the vocabulary's logits on the device, instead of reading
//     608 KB back per drafted token and scanning them on the host
//     (inference/qwen35/mod.rs:702-710, 1066-1068).
#include <atomic>
#include <new>

#include "common.cuh"
#include "ptx.cuh"

using namespace dwim;

namespace {

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Cpu::rmsnorm (gpu/cpu.rs:157-166) for any row length: one block of 256
// threads per row, v * (scale * w) with scale = 1 / sqrt(sum(v^2) / dim + eps).
__global__ void __launch_bounds__(256) rmsnorm_rows_kernel(const float *x, const float *__restrict__ weight, float eps, float *out,
                                                           size_t dim) {
    griddep_launch();
    griddep_wait();
    __shared__ float part[8];
    const float *src = x + (size_t)blockIdx.x * dim;
    float *dst = out + (size_t)blockIdx.x * dim;
    float ss = 0.0f;
    for (size_t i = threadIdx.x; i < dim; i += 256) ss += src[i] * src[i];
    ss = warp_sum_f(ss);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = part[0];
#pragma unroll
    for (int i = 1; i < 8; i++) total += part[i];
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(total, (float)dim), eps)));
    for (size_t i = threadIdx.x; i < dim; i += 256) dst[i] = __fmul_rn(src[i], __fmul_rn(scale, weight[i]));
}

// out[t][r] = w[r] . x[t] for bf16 weights, f32 activations, fp32 sums.
struct Bf16Args {
    const uint16_t *w;
    size_t rows, cols, n;
    const float *x;
    OutSpec out;
    const float *aux;
    int epi;
};

__device__ __forceinline__ float silu_mul_n(float g, float u) { return g * (1.0f / (1.0f + expf(-g))) * u; }

__device__ __forceinline__ void bf16_emit(const Bf16Args &a, size_t t, size_t r, float y) {
    const size_t i = t * a.out.pitch + a.out.row0 + r;
    if (a.epi == EPI_ADD) y += a.out.dst[0][i];
    else if (a.epi == EPI_SWIGLU) y = silu_mul_n(y, a.aux[t * a.rows + r]);
    a.out.dst[0][i] = y;
    if (a.out.world > 1) {
#pragma unroll
        for (int p = 1; p < DWIM_MAX_WORLD; p++)
            if (p < a.out.world) a.out.dst[p][i] = y;
    }
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }           // gpu/float.rs:5-8
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// Up to BF16_FEW tokens: a block per weight row and NT tokens, its eight warps
// along K, 16 bytes of weights a thread and step.  The matrices are small (1 MB)
// and the launch is bound by the chain of loads: a warp per row walked its
// 5120 weights in twenty dependent steps on twelve blocks (53 us for 96 rows and
// five tokens); here a thread takes two or three steps.
constexpr int BF16_FEW = 16;
template <int NT>
__global__ void __launch_bounds__(256) matmul_bf16_kernel(const __grid_constant__ Bf16Args a) {
    griddep_launch();
    griddep_wait();
    __shared__ float part[8][NT];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t r = blockIdx.x, t0 = (size_t)blockIdx.y * NT;
    const int nt = (int)min((size_t)NT, a.n - t0);
    float acc[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) acc[t] = 0.0f;
    const uint16_t *row = a.w + r * a.cols;
    for (size_t k = (size_t)threadIdx.x * 8; k < a.cols; k += 2048) {
        const uint4 wv = *reinterpret_cast<const uint4 *>(row + k);
        const float wf[8] = {bf16_lo(wv.x), bf16_hi(wv.x), bf16_lo(wv.y), bf16_hi(wv.y),
                             bf16_lo(wv.z), bf16_hi(wv.z), bf16_lo(wv.w), bf16_hi(wv.w)};
#pragma unroll
        for (int t = 0; t < NT; t++) {
            // columns past the last token repeat it: no branch between the loads
            const float4 *xs = reinterpret_cast<const float4 *>(a.x + (t0 + (size_t)min(t, nt - 1)) * a.cols + k);
            const float4 x0 = xs[0], x1 = xs[1];
            acc[t] = fmaf(wf[0], x0.x, acc[t]);
            acc[t] = fmaf(wf[1], x0.y, acc[t]);
            acc[t] = fmaf(wf[2], x0.z, acc[t]);
            acc[t] = fmaf(wf[3], x0.w, acc[t]);
            acc[t] = fmaf(wf[4], x1.x, acc[t]);
            acc[t] = fmaf(wf[5], x1.y, acc[t]);
            acc[t] = fmaf(wf[6], x1.z, acc[t]);
            acc[t] = fmaf(wf[7], x1.w, acc[t]);
        }
    }
#pragma unroll
    for (int t = 0; t < NT; t++) {
        const float v = warp_sum_f(acc[t]);
        if (lane == 0) part[warp][t] = v;
    }
    __syncthreads();
    if ((int)threadIdx.x < nt) {
        float v = part[0][threadIdx.x];
#pragma unroll
        for (int i = 1; i < 8; i++) v += part[i][threadIdx.x];
        bf16_emit(a, t0 + threadIdx.x, r, v);
    }
}

// More tokens: tiles of 32 rows by 32 tokens, K dealt to the eight blocks of a
// cluster (the gate matrices have three row tiles: 512 tokens would otherwise
// be 48 blocks) and each chunk of it to a block's two groups of 128 threads, whose partial
// tiles are summed in a fixed order, the blocks' out of each other's shared memory.  A thread
// keeps 4 x 2 sums as packed pairs over even and odd k (fma.rn.f32x2), four k a load.  Bound
// by the blocks' arithmetic and loads with few warps on an SM to hide either: chunks of 64 k
// come by cp.async into a ring of four, weights as bf16.  [96, 5120] by 32, 64, 128, 256 and 512
// tokens 10.6, 10.6, 16, 22 and 24 us; 14, 14, 18, 33 and 41 with one chunk ahead in registers, one
// group and two barriers a chunk; 10.7, 16, 18, 18 and 33 with four groups; 15, 15, 23, 26 and 27 in
// tiles of 64 tokens.  (A warp per row and eight tokens took 306 us by 512.)
constexpr int BT_ROWS = 32, BT_TOK = 32, BT_K = 64, BT_PITCH = BT_K + 4, BT_WPITCH = BT_K + 8, BT_SPLIT = 8;
constexpr int BT_STAGES = 4, BT_GROUPS = 2, BT_THREADS = 128 * BT_GROUPS;
constexpr int BT_X = BT_TOK * BT_PITCH * 4, BT_W = BT_ROWS * BT_WPITCH * 2, BT_SMEM = BT_STAGES * (BT_X + BT_W);      // a stage's bytes; all
static_assert(BT_GROUPS * BT_ROWS * BT_TOK * 4 <= BT_STAGES * BT_X, "the partial tiles take the activations' place");
__device__ __forceinline__ void ffma2_n(uint64_t &d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
// 16 bytes into shared memory, zeros where `there` is false (the address is not read then)
__device__ __forceinline__ void copy16(uint32_t dst, const void *src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint64_t bf16_pair(uint32_t w) { return (uint64_t)(w << 16) | (uint64_t)(w & 0xffff0000u) << 32; }
__global__ void __cluster_dims__(BT_SPLIT, 1, 1) __launch_bounds__(BT_THREADS) matmul_bf16_tile_kernel(const __grid_constant__ Bf16Args a) {
    griddep_launch();
    griddep_wait();
    extern __shared__ __align__(16) uint8_t bt_smem[];
    float *const xs0 = reinterpret_cast<float *>(bt_smem);
    const uint8_t *const ws0 = bt_smem + BT_STAGES * BT_X;
    const uint32_t xa = smem_u32(bt_smem), wa = xa + BT_STAGES * BT_X;
    const int tid = threadIdx.x, rank = blockIdx.x % BT_SPLIT;
    const size_t r0 = (size_t)(blockIdx.x / BT_SPLIT) * BT_ROWS, t0 = (size_t)blockIdx.y * BT_TOK;
    const size_t chunks = (a.cols + BT_K - 1) / BT_K;
    const size_t c0 = chunks * rank / BT_SPLIT;
    const int n_chunks = (int)(chunks * (rank + 1) / BT_SPLIT - c0);
    const int rg = tid & 7, tg = (tid >> 3) & 15, kg = tid >> 7;      // rows rg + 8 i, tokens tg + 16 j, half kg of a chunk
    constexpr int TJ = BT_TOK / 16;
    uint64_t acc[4][TJ];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < TJ; j++) acc[i][j] = 0ull;
    // a chunk's activations: rows of sixteen float4; its weights: 32 rows of eight 16-byte groups
    auto fetch = [&](int c) {
        const int s = c % BT_STAGES;
        const size_t k0 = (c0 + c) * BT_K;
#pragma unroll
        for (int i = 0; i < BT_TOK * 16 / BT_THREADS; i++) {
            const int row = (tid >> 4) + BT_THREADS / 16 * i;
            const size_t t = t0 + row, k = k0 + (size_t)(tid & 15) * 4;
            const bool there = t < a.n && k < a.cols;
            copy16(xa + s * BT_X + (row * BT_PITCH + (tid & 15) * 4) * 4, there ? a.x + t * a.cols + k : a.x, there);
        }
        if (tid < BT_ROWS * 8) {
            const int row = tid >> 3;
            const size_t r = r0 + row, k = k0 + (size_t)(tid & 7) * 8;
            const bool there = r < a.rows && k < a.cols;
            copy16(wa + s * BT_W + (row * BT_WPITCH + (tid & 7) * 8) * 2, there ? a.w + r * a.cols + k : a.w, there);
        }
    };
#pragma unroll
    for (int c = 0; c < BT_STAGES - 1; c++) {
        if (c < n_chunks) fetch(c);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int c = 0; c < n_chunks; c++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(BT_STAGES - 2) : "memory");      // this thread's part of chunk c is there
        __syncthreads();                                                             // everyone's is, and chunk c - 1 has been read
        if (c + BT_STAGES - 1 < n_chunks) fetch(c + BT_STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *xs = xs0 + c % BT_STAGES * (BT_X / 4);
        const uint8_t *ws = ws0 + c % BT_STAGES * BT_W;
#pragma unroll
        for (int i4 = 0; i4 < BT_K / BT_GROUPS / 4; i4++) {
            const int k = kg * (BT_K / BT_GROUPS) + 4 * i4;
            uint2 wq[4];
            ulonglong2 xq[TJ];
#pragma unroll
            for (int i = 0; i < 4; i++) wq[i] = *reinterpret_cast<const uint2 *>(ws + ((rg + 8 * i) * BT_WPITCH + k) * 2);
#pragma unroll
            for (int j = 0; j < TJ; j++) xq[j] = *reinterpret_cast<const ulonglong2 *>(xs + (tg + 16 * j) * BT_PITCH + k);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint64_t w01 = bf16_pair(wq[i].x), w23 = bf16_pair(wq[i].y);
#pragma unroll
                for (int j = 0; j < TJ; j++) {
                    ffma2_n(acc[i][j], w01, xq[j].x);
                    ffma2_n(acc[i][j], w23, xq[j].y);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // the groups' partial tiles [token][row] in the activations' place, their sum in the first's
    float *const part = xs0;
    constexpr int TILE = BT_TOK * BT_ROWS;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < TJ; j++)
            part[kg * TILE + (tg + 16 * j) * BT_ROWS + rg + 8 * i] = __uint_as_float((uint32_t)acc[i][j]) + __uint_as_float((uint32_t)(acc[i][j] >> 32));
    __syncthreads();
#pragma unroll
    for (int i = tid; i < TILE; i += BT_THREADS) {
        float v = part[i];
#pragma unroll
        for (int g = 1; g < BT_GROUPS; g++) v += part[g * TILE + i];
        part[i] = v;
    }
    cluster_sync();
    // this rank's share of the tile: a warp a token, a lane a row
    static_assert(BT_TOK / BT_SPLIT <= BT_THREADS / 32, "a warp a token");
    const int t = rank * (BT_TOK / BT_SPLIT) + (tid >> 5), r = tid & 31;
    if (tid >> 5 < BT_TOK / BT_SPLIT) {
        float v = 0.0f;
#pragma unroll
        for (int p = 0; p < BT_SPLIT; p++) v += ld_cluster_f32(xa + (t * BT_ROWS + r) * 4, p);
        if (t0 + t < a.n && r0 + r < a.rows) bf16_emit(a, t0 + t, r0 + r, v);
    }
    cluster_sync();      // a block's shared memory is read until here
}

// argmax: per token (row of `len` logits) the largest value's first index.  A
// value and its index travel as one 64-bit key that orders like the pair
// (value ascending, index descending): the float's bits made monotone in the
// high word, the index's complement in the low word; a block's maximum, taken by
// warp shuffles, goes straight to pinned host memory, where the call looks through
// the blocks' after the stream (clearing a device slot first and copying it back
// after were two more operations in a chain the caller waits for: the head of one
// token 148 us then, 141 like this).
// A NaN never wins (the host's `>` never lets one in either); a row of NaNs gives
// index 0.
__device__ __forceinline__ unsigned long long argmax_key(float v, uint32_t i) {
    uint32_t b = __float_as_uint(v);
    b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    if (v != v) b = 0;
    return ((unsigned long long)b << 32) | (0xffffffffu - i);
}

__global__ void __launch_bounds__(256) argmax_kernel(const float *__restrict__ logits, size_t len, unsigned long long *keys) {
    griddep_launch();
    griddep_wait();
    const float *row = logits + (size_t)blockIdx.y * len;
    unsigned long long k = 0;
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < len; i += (size_t)gridDim.x * 256) {
        const unsigned long long c = argmax_key(row[i], (uint32_t)i);
        k = c > k ? c : k;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long c = __shfl_xor_sync(0xffffffffu, k, o);
        k = c > k ? c : k;
    }
    __shared__ unsigned long long part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = k;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 1; i < 8; i++) k = part[i] > k ? part[i] : k;
        keys[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = k;
    }
}

}  // namespace

namespace dwim {

int matmul_bf16(dwim_b200_ctx *ctx, const WeightView &w, const float *x, size_t n, const OutSpec &out, const float *aux, int epi) {
    if (n == 0 || w.rows == 0) return 0;
    Bf16Args a{reinterpret_cast<const uint16_t *>(w.quants), w.rows, w.cols, n, x, out, aux, epi};
    if ((n + 7) / 8 > 65535) return fail(ctx, DWIM_B200_EINVAL, "bf16 product: %zu tokens in one call", n);
    // Each row of blocks of the one kernel reads all the activations again, so it is for the token
    // counts whose activations are small beside a launch; the other wants whole tiles of tokens.
    const bool dependent = !ctx->weights_written;
    if (n > (size_t)BF16_FEW) {
        static std::atomic<bool> configured[64] = {};
        if (!configured[ctx->device & 63]) {
            DWIM_CUDA(ctx, cudaFuncSetAttribute(matmul_bf16_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BT_SMEM));
            configured[ctx->device & 63] = true;
        }
        const dim3 grid((unsigned)((w.rows + BT_ROWS - 1) / BT_ROWS * BT_SPLIT), (unsigned)((n + BT_TOK - 1) / BT_TOK));
        DWIM_CUDA(ctx, launch_dependent(dependent, matmul_bf16_tile_kernel, grid, dim3(BT_THREADS), (size_t)BT_SMEM, ctx->stream, a));
    } else {
        auto kern = n == 1 ? matmul_bf16_kernel<1> : n == 2 ? matmul_bf16_kernel<2> : n <= 4 ? matmul_bf16_kernel<4> : matmul_bf16_kernel<8>;
        const dim3 grid((unsigned)w.rows, (unsigned)((n + 7) / 8));
        DWIM_CUDA(ctx, launch_dependent(dependent, kern, grid, dim3(256), 0, ctx->stream, a));
    }
    ctx->weights_written = false;
    DWIM_LAUNCHED(ctx);
    return 0;
}

}  // namespace dwim

extern "C" int dwim_b200_normalize(dwim_b200_ctx *ctx, dwim_b200_buffer *out, const dwim_b200_buffer *x,
                                   const dwim_b200_buffer *weight, size_t len, float eps) {
    DWIM_DEVICE(ctx);
    if (!ctx || !out || !x || !weight) return DWIM_B200_EINVAL;
    const size_t dim = weight->len;
    // gpu/cuda/mod.rs:1184-1185
    if (dim == 0 || out->len != len || len > x->len || len % dim != 0)
        return fail(ctx, DWIM_B200_EINVAL, "normalize: out of %zu, %zu of x's %zu, rows of %zu", out->len, len, x->len, dim);
    out->shadow_kind = SHADOW_NONE;
    out->bf16_exact = false;
    if (len == 0) return 0;
    const size_t n = len / dim;
    if (dim % 256 == 0 && n > DWIM_SMALL_M_MAX && n <= 65535) {
        // more tokens than the small-M kernel takes: the next product is the tensor-core GEMM, whose
        // operand (f16 value and remainder terms, sub-block means, the token's scale) this launch writes
        const int split = ctx->act_f16 ? 0 : 1;
        int rc = reserve_shadow(ctx, out, gemm_operand_bytes(dim, n, split));
        if (rc) return rc;
        rc = build_gemm_operand(ctx, x->data, n, dim, split, (__half *)out->shadow, weight->data, eps, out->data);
        if (rc) return rc;
        shadow_made(ctx, out, SHADOW_GEMM, dim, split);
        return 0;
    }
    if (dim % 256 == 0 && n <= (size_t)I8_MAX_TOKENS) {
        // a few tokens: the int8 digit planes of the small-M kernel, from the same launch
        int rc = reserve_shadow(ctx, out, panel_i8_bytes(dim, n));
        if (rc) return rc;
        rc = build_panels_i8(ctx, x->data, n, dim, (uint8_t *)out->shadow, weight->data, eps, out->data);
        if (rc) return rc;
        shadow_made(ctx, out, SHADOW_PANEL_I8, dim, 0);
        return 0;
    }
    DWIM_CUDA(ctx, launch_dependent(!ctx->weights_written, rmsnorm_rows_kernel, dim3((unsigned)n), dim3(256), 0, ctx->stream,
                                    (const float *)x->data, (const float *)weight->data, eps, out->data, dim));
    DWIM_LAUNCHED(ctx);
    return 0;
}

extern "C" int dwim_b200_argmax(dwim_b200_ctx *ctx, const dwim_b200_buffer *logits, size_t len, uint32_t *out, size_t n) {
    DWIM_DEVICE(ctx);
    if (!ctx || !logits || (!out && n)) return DWIM_B200_EINVAL;
    if (len == 0 || n * len != logits->len || len > 0xffffffffull || n > 65535)
        return fail(ctx, DWIM_B200_EINVAL, "argmax: %zu rows of %zu logits in a buffer of %zu", n, len, logits->len);
    if (n == 0) return 0;
    size_t blocks = (len + 2047) / 2048;
    if (blocks > (size_t)ctx->sm_count * 2) blocks = (size_t)ctx->sm_count * 2;
    if (n * blocks > 65536) blocks = n < 65536 ? 65536 / n : 1;      // keys that the call looks through
    if (n * blocks > ctx->argmax_cap) {
        if (ctx->argmax_host) {
            DWIM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            cudaFreeHost(ctx->argmax_host);
            ctx->argmax_host = nullptr;
            ctx->argmax_cap = 0;
        }
        DWIM_CUDA(ctx, cudaMallocHost((void **)&ctx->argmax_host, n * blocks * sizeof(unsigned long long)));
        ctx->argmax_cap = n * blocks;
    }
    DWIM_CUDA(ctx, launch_dependent(!ctx->weights_written, argmax_kernel, dim3((unsigned)blocks, (unsigned)n), dim3(256), 0, ctx->stream,
                                    (const float *)logits->data, len, ctx->argmax_host));
    DWIM_LAUNCHED(ctx);
    DWIM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (size_t t = 0; t < n; t++) {
        unsigned long long k = 0;
        for (size_t b = 0; b < blocks; b++) k = ctx->argmax_host[t * blocks + b] > k ? ctx->argmax_host[t * blocks + b] : k;
        // a row of NaNs leaves the key at its index alone, an empty word above: index 0, as the host's scan gives
        out[t] = k >> 32 ? 0xffffffffu - (uint32_t)(k & 0xffffffffull) : 0;
    }
    return 0;
}
