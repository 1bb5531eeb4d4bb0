// tcgen05 wrappers and descriptors of the tensor-core kernels (gemm.cu).
#pragma once
#include "ptx.cuh"

namespace dwim {

// True for one lane of the (converged) warp, the same one every time.  Tensor-core and TMA
// instructions take their addresses and descriptors from uniform registers; behind elect.sync the
// compiler knows that one thread is left and moves them there directly, behind `lane == 0` it
// emits a loop over the active threads for each of them: 53 cycles to issue a
// tcgen05.mma against 9 (measured at N = 16, whose execution is shorter than either).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// Arrive on an mbarrier once every MMA this thread issued so far has finished.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// d = a * b + d on two packed floats.
__device__ __forceinline__ void ffma2(uint64_t &d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t fadd2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
    uint32_t a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v));
    lo = __uint_as_float(a);
    hi = __uint_as_float(b);
}

// Shared-memory matrix descriptors (K-major operands).
//   [0,14) address >> 4   [16,30) leading byte offset >> 4   [32,46) stride
//   byte offset >> 4   [46,48) version 1   [61,64) layout
// 128-byte swizzle: rows are 128 bytes (64 f16), eight-row groups 1024 bytes
// apart (stride offset); the leading offset is not used: (addr & 0x3ffff) >> 4 | 1 << 16 |
// 64 << 32 | 1 << 46 | 2 << 61.  The kernels keep it as a low word per stage and the high word
// all stages share, so that the MMA warp adds to 32-bit values only.
constexpr uint32_t DESC_HI_SW128 = 64u | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo_sw128(uint32_t addr) { return ((addr & 0x3ffffu) >> 4) | (1u << 16); }
// No swizzle: 8 rows x 16 bytes are contiguous (128 bytes); eight-row groups
// 128 bytes apart (stride offset); the second 8 of K `lbo` bytes further on.
__device__ __forceinline__ uint64_t smem_desc_plain(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | (8ull << 32) | (1ull << 46);
}
// Instruction descriptor: f32 accumulate (bits 4-5 = 1), f16 A and B (0),
// both K-major (0), N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_f16(int m, int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

}  // namespace dwim
