// Thin wrappers over the sm_100a instructions of the tensor-core kernels:
// tcgen05 8-bit integer MMA (32-bit accumulators in TMEM, exact), mbarriers
// and bulk copies.  Every wait is bounded.
#pragma once
#include "gl.cuh"

namespace tc {

__device__ __forceinline__ u32 smem_u32(const void *p) { return (u32)__cvta_generic_to_shared(p); }

// ---------------------------------------------------------------- mbarriers

__device__ __forceinline__ void mbar_init(u64 *m, u32 count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(u64 *m)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(m)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(u64 *m, u32 bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(m)), "r"(bytes) : "memory");
}
// has the phase of the given parity completed?
__device__ __forceinline__ bool mbar_test(u64 *m, u32 parity)
{
    u32 done;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done)
                 : "r"(smem_u32(m)), "r"(parity)
                 : "memory");
    return done != 0;
}
// Bounded wait for the phase of the given parity; false after `polls` polls.
__device__ __forceinline__ bool mbar_wait(u64 *m, u32 parity, unsigned long long polls)
{
    const u32 a = smem_u32(m);
    for (unsigned long long it = 0; it < polls; it++) {
        u32 done;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(a), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// generic-proxy accesses before it are ordered before async-proxy accesses
// (bulk copies, MMA operand reads) after it
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// global -> shared bulk copy (16-byte aligned addresses and size)
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, u32 bytes, u64 *m)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(m))
                 : "memory");
}

// tiled tensor load (4 dimensions) at (0, 0, c2, c3): the first coordinate is
// 0, so 16-byte aligned
__device__ __forceinline__ void tensor_g2s(void *dst, const void *map, u32 c2, u32 c3, u64 *m)
{
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                 "[%0], [%1, {%2, %2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
                 "l"(map), "r"(0), "r"(c2), "r"(c3), "r"(smem_u32(m))
                 : "memory");
}

// ------------------------------------------------------------------ tcgen05

// Shared-memory operand descriptors, K-major.  No swizzle: core matrices of 8
// rows x 16 bytes (128 contiguous bytes); `lbo` is the byte distance of
// neighbouring core matrices along K, `sbo` along M/N.
__device__ __forceinline__ u64 desc_plain(u32 addr, u32 lbo, u32 sbo)
{
    return (u64)((addr & 0x3FFFF) >> 4) | ((u64)(lbo >> 4) << 16) | ((u64)(sbo >> 4) << 32) | (1ull << 46);
}
// 128-byte swizzle: rows of 128 bytes, groups of 8 rows of 1024 bytes (1024-byte
// aligned), the 16-byte chunk index XORed with the row index mod 8.
__device__ __forceinline__ u64 desc_sw128(u32 addr)
{
    return (u64)((addr & 0x3FFFF) >> 4) | (1ull << 16) | ((u64)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// the same operand `bytes` further (no carry out of the 14-bit address field
// as long as the end lies in shared memory)
__device__ __forceinline__ u64 desc_at(u64 desc, u32 bytes)
{
    return (desc & 0xFFFFFFFF00000000ull) | ((u32)desc + (bytes >> 4));
}
// Instruction descriptor of kind::i8: 32-bit integer accumulators, M = 128,
// N columns; operands of unsigned or signed bytes.
__host__ __device__ constexpr u32 idesc_i8(u32 n, bool a_signed, bool b_signed)
{
    return (2u << 4) | ((a_signed ? 1u : 0u) << 7) | ((b_signed ? 1u : 0u) << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
// D[128 x N] (+)= A[128 x 32] B[N x 32]^T, issued by one thread
__device__ __forceinline__ void mma_i8(u32 d, u64 a, u64 b, u32 idesc, bool accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                 "l"(a), "l"(b), "r"(idesc), "r"((u32)accumulate)
                 : "memory");
}
// arrive on `m` once every MMA issued by this thread so far is complete
__device__ __forceinline__ void commit(u64 *m)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(m))
                 : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// called by one whole warp each
__device__ __forceinline__ void tmem_alloc_512(u32 *slot)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free_512(u32 tmem)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}
// 16 accumulator columns of this thread's TMEM lane (lane quadrant = warp mod 4);
// the values are ready after tmem_wait16 on the same array
__device__ __forceinline__ void tmem_ld16(u32 addr, u32 (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_wait16(u32 (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

// ------------------------------------------------- byte accumulators to mod p

__device__ __forceinline__ u64 mad_wide(u32 a, u32 b, u64 c)
{
    u64 r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
// Two residues lo + hi 2^32 mod p (lazy), lo, hi < 2^51.  With hi = h1:h0 and
// 2^64 = 2^32 - 1 each is t + h0 2^32, t = lo + h1 (2^32 - 1); the sum leaves
// 64 bits only when h0 is within t_hi < 2^21 of 2^32, so that case is a branch
// rarely taken instead of a carry chain (27 clocks per output and scheduler
// with its recombination against 40 and more with the chain).
__device__ __forceinline__ void fold2(u64 lo0, u64 hi0, u64 lo1, u64 hi1, u64 &r0, u64 &r1)
{
    const u64 t0 = mad_wide((u32)(hi0 >> 32), 0xFFFFFFFFu, lo0), t1 = mad_wide((u32)(hi1 >> 32), 0xFFFFFFFFu, lo1);
    const u32 w0 = (u32)(t0 >> 32) + (u32)hi0, w1 = (u32)(t1 >> 32) + (u32)hi1;
    r0 = ((u64)w0 << 32) | (u32)t0;
    r1 = ((u64)w1 << 32) | (u32)t1;
    const bool c0 = w0 < (u32)hi0, c1 = w1 < (u32)hi1;
    if (__builtin_expect(c0 | c1, 0)) {
        if (c0) r0 += gl::EPS;  // w < 2^21: no second carry
        if (c1) r1 += gl::EPS;
    }
}
// Eight byte accumulators each of two outputs, sum_s a[s] 2^(8s) mod p.
// wide: unsigned accumulators below 2^27 (43 clocks per output and scheduler)
__device__ __forceinline__ void recombine2_wide(const u32 (&a)[16], u64 &r0, u64 &r1)
{
    u64 w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        w[i] = mad_wide(a[4 * i + 1], 1u << 8, (u64)a[4 * i]);
        w[i] = mad_wide(a[4 * i + 2], 1u << 16, w[i]);
        w[i] = mad_wide(a[4 * i + 3], 1u << 24, w[i]);
    }
    fold2(w[0], w[1], w[2], w[3], r0, r1);
}
// Signed accumulators with |a[s] + 2^8 a[s+1]| below 2^30: neighbours meet in
// 32 bits first (t[i], weight 2^(16i)), which halves the wide multiply-adds.
// Each t is lifted by a constant near 1.5 2^30 to make it unsigned; the four
// constants, weighted 2^(16i), add up to 24576 p.
constexpr u64 LIFT_M = 24576;
__host__ __device__ constexpr u32 lift(int i)
{
    return (u32)(i == 0 ? LIFT_M + (LIFT_M << 16) : (LIFT_M << 16) - (i == 2 ? 2 : 1) * LIFT_M);
}
__device__ __forceinline__ void fold2_lifted(const u32 (&t)[4], const u32 (&s)[4], u64 &r0, u64 &r1)
{
    fold2(mad_wide(t[1], 1u << 16, (u64)t[0]), mad_wide(t[3], 1u << 16, (u64)t[2]), mad_wide(s[1], 1u << 16, (u64)s[0]),
          mad_wide(s[3], 1u << 16, (u64)s[2]), r0, r1);
}
__device__ __forceinline__ void recombine2_signed(const u32 (&a)[16], u64 &r0, u64 &r1)
{
    u32 t[4], s[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        t[i] = a[2 * i] + lift(i) + (a[2 * i + 1] << 8);
        s[i] = a[8 + 2 * i] + lift(i) + (a[9 + 2 * i] << 8);
    }
    fold2_lifted(t, s, r0, r1);
}

}  // namespace tc
