// tcgen05 / tensor-memory wrappers (inline PTX for sm_100a) and the bounded barrier wait shared by every kernel that
// issues tensor-core work.
#pragma once
#include "tma.cuh"

namespace cinn {

constexpr long long WAIT_LIMIT_CYCLES = 4000000000LL;   // about two seconds

// Bounded wait.  Returns false when the kernel is being abandoned; `status` receives `code` once.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code, int* status) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t spin = 1;; ++spin) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 255u) == 0) {
            if (*abort_flag) return false;
            if (clock64() - t0 > WAIT_LIMIT_CYCLES) {
                *abort_flag = 1;
                atomicCAS(status, 0, code);
                return false;
            }
        }
    }
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Arrival on the barrier once the MMAs issued so far have retired; called by a whole warp and issued by the lane that
// elect.sync chooses, the one that issued the MMAs.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(bar) : "memory");
}

// whole-warp allocation of `cols` tensor-memory columns (a power of two, at least 32); the base address lands in *slot
__device__ __forceinline__ void tc_alloc(uint32_t slot_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t base, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}

// The MMA warp runs as a whole and one elected lane issues: with warp-uniform control flow the descriptors live in
// uniform registers.  Issued from a branch that one lane takes, an MMA cost its issuer 70 to 130 cycles of moves, more
// than the MMA itself.
// 16-bit operands of one type: D[tmem] (+)= A[smem desc] * B[smem desc], fp32 accumulation
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// D[tmem] = A[smem desc] * B[smem desc], e4m3 x e4m3 -> fp32.  Called by a whole warp, issued by one elected lane.
// The four MMAs of a K block by one statement with one election: one by one, with 64-bit descriptors, they cost their warp 350
// cycles, like this 100.  Low words of the descriptors; STEP_B: 16-byte units from one step's B to the next.
template <int STEP_B>
__device__ __forceinline__ void tc_mma_f8_block(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
    constexpr uint32_t hi = (uint32_t)((((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61)) >> 32);
    asm volatile(
        "{\n\t.reg .pred e;\n\t.reg .b64 a, b;\n\t.reg .b32 x, y;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "mov.b64 a, {%1, %4};\n\tmov.b64 b, {%2, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %3, 0;\n\t"
        "add.u32 x, %1, 2;\n\tadd.u32 y, %2, %5;\n\tmov.b64 a, {x, %4};\n\tmov.b64 b, {y, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %3, 1;\n\t"
        "add.u32 x, %1, 4;\n\tadd.u32 y, %2, %6;\n\tmov.b64 a, {x, %4};\n\tmov.b64 b, {y, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %3, 1;\n\t"
        "add.u32 x, %1, 6;\n\tadd.u32 y, %2, %7;\n\tmov.b64 a, {x, %4};\n\tmov.b64 b, {y, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %3, 1;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(hi), "n"(STEP_B), "n"(2 * STEP_B), "n"(3 * STEP_B) : "memory");
}

// kind::f16 instruction descriptor: fp32 accumulate, A and B of the same 16-bit type; *_mn: that operand is MN-major
__host__ __device__ constexpr uint32_t make_idesc_f16(bool bf16, int m, int n, bool a_mn = false, bool b_mn = false) {
    return (1u << 4)                                   // D format: fp32
           | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10)   // A, B format: 0 = fp16, 1 = bf16
           | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16)
           | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Operands in panels: 128 rows (or as many as the other side has) of 128 bytes, 128-byte swizzle.  A panel is used K-major (its 64 columns
// are the reduction axis; a step of four takes 16 of them: 32 bytes) and MN-major (its 128 rows are; a step of eight takes 16 of them: 2048
// bytes).  Both have one descriptor, of which only the low word (the address in units of 16 bytes) varies.
constexpr uint32_t DESC_HI = (uint32_t)((((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61)) >> 32);
__device__ __forceinline__ uint32_t panel_desc(uint32_t panel) { return ((panel >> 4) & 0x3FFFu) | (1u << 16); }

// One warp issues all MMAs, so what it does between two of them is time the tensor core waits.  A panel's steps are one
// statement with one election: issued one by one, with 64-bit descriptors, a panel of four cost the warp 350 cycles where
// the MMAs take 256; like this 257.
// D (+)= A B over the 64 columns of two K-major panels; the first step overwrites D when `fresh`
__device__ __forceinline__ void mma_panels(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, bool fresh) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 a, b;\n\t.reg .b32 x, y;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 a, {%1, %4};\n\tmov.b64 b, {%2, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t"
        "add.u32 x, %1, 2;\n\tadd.u32 y, %2, 2;\n\tmov.b64 a, {x, %4};\n\tmov.b64 b, {y, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, 1;\n\t"
        "add.u32 x, %1, 4;\n\tadd.u32 y, %2, 4;\n\tmov.b64 a, {x, %4};\n\tmov.b64 b, {y, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, 1;\n\t"
        "add.u32 x, %1, 6;\n\tadd.u32 y, %2, 6;\n\tmov.b64 a, {x, %4};\n\tmov.b64 b, {y, %4};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, 1;\n\t}"
        ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(DESC_HI), "r"(fresh ? 0u : 1u) : "memory");
}

// 32 lanes x 16 consecutive fp32 columns: thread i receives TMEM lane (base lane + i)
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor, 128-byte swizzle, Blackwell descriptor version 1.
// lbo / sbo in bytes.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;     // descriptor version
    d |= (uint64_t)2 << 61;     // SWIZZLE_128B
    return d;
}

}  // namespace cinn
