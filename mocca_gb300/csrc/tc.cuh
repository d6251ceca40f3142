// tc.cuh -- tcgen05 (5th-generation tensor core) building blocks for sm_103a:
// TMEM allocation, shared-memory matrix descriptors, the BF16 MMA with FP32
// accumulation in TMEM, commit to an mbarrier, TMEM loads, and a bounded
// mbarrier wait.
//
// Operand layout used throughout: K-major, no swizzle.  A tile of R rows and
// 32 columns (K) of bf16 is stored as 8x8 "core matrices" of 128 contiguous
// bytes (8 rows of 16 bytes); the core matrix of row group rg and K group kg
// sits at byte ((rg * 4) + kg) * 128.  In the descriptor, the leading byte
// offset (between K groups) is 128 and the stride byte offset (between row
// groups) is 512.  One MMA consumes K = 16, i.e. two K groups; the second
// K step starts 256 bytes further.
#pragma once

#include <stdint.h>

namespace mg {
namespace tc {

constexpr int kRowBytes = 64;        // bytes of one 32-wide bf16 row (K = 32)
constexpr uint32_t kLbo = 128;       // leading byte offset: next K group
constexpr uint32_t kSbo = 512;       // stride byte offset: next 8-row group
constexpr uint32_t kKStep = 256;     // bytes between the two K = 16 halves

__host__ __device__ inline uint32_t kmajor_off(int row, int k) {
    return (uint32_t)((((row >> 3) * 4 + (k >> 3)) * 128) + (row & 7) * 16 + (k & 7) * 2);
}

// Same layout for a tile with kg K groups (K = 8 kg): stride byte offset 128 kg.
__host__ __device__ inline uint32_t kmajor_off_g(int row, int k, int kg) {
    return (uint32_t)((((row >> 3) * kg + (k >> 3)) * 128) + (row & 7) * 16 + (k & 7) * 2);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor (no swizzle, fixed field 0b001 at bit 46).
__device__ __forceinline__ uint64_t desc(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((kLbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((kSbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

__device__ __forceinline__ uint64_t desc_sbo(uint32_t saddr, uint32_t sbo) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((kLbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Instruction descriptor of kind::f16: FP32 D, BF16 A and B, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db,
                                         uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void commit(uint64_t* mbar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(mbar))
        : "memory");
}

// Whole warp: allocate ncols (power of two >= 32) TMEM columns, address to *slot.
__device__ __forceinline__ void alloc(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(slot)),
                 "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}

__device__ __forceinline__ void fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Generic-proxy shared-memory writes become visible to the tensor core.
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* mbar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Wait for phase `parity` of the mbarrier, giving up after ~max_cycles SM
// clocks.  Returns true when the phase completed.
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, uint32_t parity, long long max_cycles) {
    const uint32_t a = smem_u32(mbar);
    const auto done = [a, parity]() {
        uint32_t d;
        // the hardware may suspend the thread for up to 20 us per try
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
            "selp.b32 %0, 1, 0, p;\n}\n"
            : "=r"(d)
            : "r"(a), "r"(parity), "r"(20000u)
            : "memory");
        return d != 0;
    };
    if (done()) return true;
    const long long t0 = clock64();
    while (!done())
        if (clock64() - t0 > max_cycles) return false;
    return true;
}

// The context's status word, in host memory: a wait ran out.
__device__ __forceinline__ void report_timeout(int* status) {
    asm volatile("st.relaxed.sys.global.s32 [%0], 1;" ::"l"(status) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// 8-byte asynchronous global -> shared copy (cp.async, L1-allocating).
__device__ __forceinline__ void cp_async8(void* sdst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(sdst)), "l"(gsrc)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// 32 TMEM lanes x 16 consecutive 32-bit columns: lane (base + laneid), columns c..c+15.
// The registers are valid only after wait_ld() on them.
__device__ __forceinline__ void ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// 32 TMEM lanes x 8 consecutive 32-bit columns.
__device__ __forceinline__ void ld4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}

__device__ __forceinline__ void wait_ld(uint32_t (&r)[4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3])
                 :
                 : "memory");
}

__device__ __forceinline__ void ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7])
        : "r"(taddr));
}

__device__ __forceinline__ void wait_ld(uint32_t (&r)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7])
                 :
                 : "memory");
}

// Wait for the TMEM loads issued so far; the registers are tied to the wait
// so that no use of them is scheduled before it.
__device__ __forceinline__ void wait_ld(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

}  // namespace tc
}  // namespace mg
