// Fifth-generation tensor core products with FP32 accumulators in tensor memory (sm_103a): one
// 128 x N x 16 bf16 product per instruction, operands in shared memory.
//
// FP32 operands enter as three bf16 terms, x = h + m + l (8 mantissa bits each, so all 24 bits of a
// normal x), and a product as h h plus the five terms h m, m h, m m, h l, l h; what is left out, m l and l m, is
// at most 2^-24 of the product (for 97 % of random pairs below 2^-26), where an FP32 product rounds by as much.
// h h and the small terms accumulate in separate accumulators, so the small ones are not rounded away against the large
// sum.  An accumulator cuts towards zero what it adds, so that the error of a long sum of one sign grows with its length.
//
// Operand layout of one term: rows contiguous, blocks of 64 rows x 8 k (1024 bytes, aligned to 1024) with 128-byte
// swizzle: element (row, k) of a block at 128 k + ((row / 8) ^ k) 16 + (row % 8) 2 (block_offset), a group of 8 k's row
// blocks 1024 bytes apart.  A 128 x 112 x 16 product takes 62 cycles, about its reads of both operands (7.7 KB).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cfloat>
#include <cstdint>

namespace spn {
namespace dev {
namespace umma {

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return uint32_t(__cvta_generic_to_shared(p)); }

// Tensor memory: `cols` columns (a power of two >= 32) of 128 lanes; a whole warp calls these.
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols));
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// generic-proxy accesses of this thread, to shared and global memory, come before later bulk copies
__device__ __forceinline__ void fence_copies() { asm volatile("fence.proxy.async;" ::: "memory"); }

__device__ __forceinline__ void bar_init(uint64_t *bar, uint32_t arrivals = 1) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(arrivals) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// Bulk copy from global memory (addresses and size multiples of 16 bytes).
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
                 "r"(smem_addr(bar))
                 : "memory");
}
// Waits for phase `parity` of the barrier; false after kWaitPolls polls.
constexpr int kWaitPolls = 1 << 20;
__device__ __forceinline__ bool bar_wait(uint64_t *bar, uint32_t parity) {
    for (int i = 0; i < kWaitPolls; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n}"
                     : "=r"(done)
                     : "r"(smem_addr(bar)), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}
// The barrier completes a phase when this thread's products so far are done.
__device__ __forceinline__ void commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// Byte of rows 4 r .. 4 r + 3 (r < 16) of k (< 8) in a block.
__device__ __forceinline__ int block_offset(int r, int k) { return 128 * k + ((((r >> 1) ^ k) << 4) | ((r & 1) << 3)); }

// Shared-memory descriptor of a term's operand from the 8-k group at addr on; groups are `group` bytes apart.  Fields: start >> 4,
// distance of row blocks >> 4, distance of 8-k groups >> 4, version 1, 128-byte swizzle.
__device__ __forceinline__ uint64_t operand(uint32_t addr, uint32_t group) {
    return uint64_t((addr >> 4) & 0x3fff) | (uint64_t(1024 >> 4) << 16) | (uint64_t(group >> 4) << 32) | (uint64_t(1) << 46) |
           (uint64_t(2) << 61);
}
// bf16 operands, rows contiguous, FP32 accumulator, M = 128.
__device__ __forceinline__ uint32_t instruction(uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (3u << 15) | ((n >> 3) << 17) | (8u << 24);
}

// D[128 x N] (+)= A B^T over 16 k; one thread issues it.
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t inst, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
                 "l"(a), "l"(b), "r"(inst), "r"(uint32_t(accumulate))
                 : "memory");
}

// D_hi, D_lo (+)= the product of `steps` x 16 k of A (128 rows) and B (n rows): the terms' operands follow each other, a_term and
// b_term bytes apart, their 8-k groups a_group and b_group bytes.
__device__ __forceinline__ void product(uint32_t d_hi, uint32_t d_lo, uint32_t a, uint32_t a_group, uint32_t a_term, uint32_t b,
                                        uint32_t b_group, uint32_t b_term, uint32_t n, int steps, bool accumulate) {
    const uint32_t inst = instruction(n);
    // the terms' descriptors differ in the start address alone
    uint64_t da[3], db[3];
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        da[t] = operand(a + t * a_term, a_group);
        db[t] = operand(b + t * b_term, b_group);
    }
    constexpr int ta[5] = {0, 1, 1, 0, 2}, tb[5] = {1, 0, 1, 2, 0};
    for (int s = 0; s < steps; ++s) {
        mma(d_hi, da[0], db[0], inst, accumulate || s > 0);
#pragma unroll
        for (int t = 0; t < 5; ++t) mma(d_lo, da[ta[t]], db[tb[t]], inst, accumulate || t > 0 || s > 0);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            da[t] += 2 * (a_group >> 4);
            db[t] += 2 * (b_group >> 4);
        }
    }
}

// 16 columns of this thread's lane (lane 32 (warp % 4) + lane id of the addressed rows).
__device__ __forceinline__ void load16(uint32_t addr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// The three bf16 terms of two values of magnitudes up to kSplitMax, above which rounding to bf16 may give infinity.
constexpr float kSplitMax = 3.3e38f;
__device__ __forceinline__ void split2(float u, float v, uint32_t &h, uint32_t &m, uint32_t &l) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(u, v);
    const float ru = u - __low2float(p), rv = v - __high2float(p);
    const __nv_bfloat162 q = __floats2bfloat162_rn(ru, rv);
    const __nv_bfloat162 s = __floats2bfloat162_rn(ru - __low2float(q), rv - __high2float(q));
    h = *reinterpret_cast<const uint32_t *>(&p);
    m = *reinterpret_cast<const uint32_t *>(&q);
    l = *reinterpret_cast<const uint32_t *>(&s);
}
// The terms of any two values: the leading one is cut instead of rounded above kSplitMax, so that every finite value keeps all three.  An
// infinite value is its leading term alone: what the small terms' accumulator then holds is no part of the product (add_terms).
__device__ __forceinline__ void split2_any(float u, float v, uint32_t &h, uint32_t &m, uint32_t &l) {
    const float cu = __uint_as_float(__float_as_uint(u) & 0xffff0000u), cv = __uint_as_float(__float_as_uint(v) & 0xffff0000u);
    const bool bu = fabsf(u) > kSplitMax, bv = fabsf(v) > kSplitMax;
    split2(bu ? (isinf(u) ? 0.0f : u - cu) : u, bv ? (isinf(v) ? 0.0f : v - cv) : v, h, m, l);
    if (bu) l = (l & 0xffff0000u) | (m & 0xffffu), m = (m & 0xffff0000u) | (h & 0xffffu), h = (h & 0xffff0000u) | (__float_as_uint(cu) >> 16);
    if (bv) l = (l & 0xffffu) | (m & 0xffff0000u), m = (m & 0xffffu) | (h & 0xffff0000u), h = (h & 0xffffu) | __float_as_uint(cv);
}
// An element of a product from its two accumulators.  An infinite operand makes the large one infinite (or NaN, as the FP32 sum is)
// and the small one NaN, from infinity times a term that is zero or of the other sign.
__device__ __forceinline__ float add_terms(float hi, float lo) { return fabsf(hi) <= FLT_MAX ? hi + lo : hi; }

}  // namespace umma
}  // namespace dev
}  // namespace spn
