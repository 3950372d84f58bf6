// tc.cuh -- thin wrappers over the sm_100-family tensor-core (tcgen05), TMEM
// and mbarrier instructions used by the learned warm start (cnn.cu).
//
// Operands are BF16 in shared memory in the no-swizzle K-major canonical
// layout: 8-row x 16-byte core matrices; the descriptor's leading byte offset
// (LBO) steps between core matrices along K, the stride byte offset (SBO)
// along M/N.  Accumulators are FP32 in TMEM (lane = output row, column =
// output channel).  Every wait is bounded: on expiry it reports failure and
// the caller sets its error flag, drains and frees its TMEM.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace nr {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor (no swizzle).
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version of the sm_100 family
    return d;
}

// Instruction descriptor of kind::f16: FP32 accumulate, A = B = BF16, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

// Waits for phase `parity` of the barrier; gives up after `limit` polls.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int limit) {
    uint32_t done = 0;
    for (int it = 0; it < limit && !done; it++) {
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.b32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
    }
    return done != 0;
}

// One warp allocates ncols TMEM columns (power of two >= 32); the address is
// written to *dst (shared memory).
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(dst)),
                 "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}

__device__ __forceinline__ void fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Makes this thread's generic-proxy shared-memory stores visible to the tensor core.
__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// D[tmem] (+)= A(desc) * B(desc); issued by one thread.
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                         uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// The same issued by a whole (converged) warp, of which one elected lane -- the
// same one each time -- performs it.  With warp-uniform operands the
// descriptors stay in uniform registers: issued from inside a one-lane branch
// they are moved there one word at a time, about 96 cycles per MMA in a
// sequence with compile-time offsets.  Descriptors as two words: an offset in
// bytes / 16 adds to the low one.
__device__ __forceinline__ void mma_bf16_warp(uint32_t tmem_d, uint32_t alo, uint32_t ahi,
                                              uint32_t blo, uint32_t bhi, uint32_t idesc,
                                              uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p, q;\n .reg .b64 a, b;\n elect.sync _|q, 0xffffffff;\n"
        " setp.ne.b32 p, %6, 0;\n mov.b64 a, {%1, %2};\n mov.b64 b, {%3, %4};\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n}\n" ::"r"(tmem_d),
        "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(accumulate));
}

// commit() by the elected lane of a whole warp.
__device__ __forceinline__ void commit_warp(uint64_t* bar) {
    asm volatile(
        "{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(
            smem_u32(bar))
        : "memory");
}

// Arrives on the barrier once every tensor-core operation issued so far by
// this thread has completed.
__device__ __forceinline__ void commit(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

// Warp w reads TMEM lanes 32(w%4) .. +31, 32 consecutive columns from col:
// thread `lane` gets row 32(w%4)+lane, r[c] = column col + c.  The wait is in
// the same statement, so the outputs are defined only once it has completed.
__device__ __forceinline__ void ld32(uint32_t tmem, uint32_t lane0, uint32_t col, uint32_t* r) {
    const uint32_t a = tmem + (lane0 << 16) + col;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(a)
        : "memory");
}

}  // namespace tc
}  // namespace nr
