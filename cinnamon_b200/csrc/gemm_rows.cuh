// Block-scaled FP8 GEMM for few rows (included by gemm.cu): a projection of a prompt or of a generated token.
//
// What has to move is the weight, once; on 128 x 256 tiles a 64 x 7168 -> 4096 product keeps 16 SMs busy, each with a chain of 56 K
// blocks of half a microsecond.  Here a CTA takes 32 columns over the whole reduction, two CTAs per SM: 128 of them pull the weight
// through rings of eight stages, and the rows' bytes, which every CTA reads, come from L2.  The K blocks of a batch of four have a
// TMEM buffer each and one barrier, so that the promotion's chain (a load and 16 FMAs per K block) is short.  Every output
// element is the sum the other kernels form, in their order: the same bits.
// 64 x 7168 -> 4096 31.5 -> 19.2 us, 64 x 2048 -> 7168 14.7 -> 9.3, 128 x 512 -> 1024 8.6 -> 5.9: half a thousand cycles per K block, of
// which the promotion's loads are the half (a ring twice as deep changes nothing).
//
// Roles (6 warps): 0-3 promotion and store, 4 TMA producer, 5 TMEM allocation and MMAs.  All waits are bounded.
#pragma once

namespace rows {

constexpr int RN = 32;                  // columns of a CTA
constexpr int BATCH = 4;                // K blocks per tensor-memory barrier
constexpr int RTHREADS = 6 * 32;
constexpr int RTMEM_COLS = 2 * BATCH * RN;
constexpr int RB_BYTES = RN * BK;

// ROWS: rows of A that a stage has room for, 64 or 128; p.box_rows of them are copied.  The MMAs take 128 rows: the rest are whatever
// lies there and bytes of other stages, whose products nobody reads.
template <int ROWS> struct Shape {
    static constexpr int STAGES = ROWS == 64 ? 8 : 5;
    static constexpr int A_BYTES = ROWS * BK;
    static constexpr int BAR_OFF = STAGES * (A_BYTES + RB_BYTES);
    static constexpr size_t BYTES = (size_t)BAR_OFF + 256 + 1024;
};

constexpr uint32_t RIDESC = (1u << 4) | ((uint32_t)(RN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);

template <int ROWS, int OUT>
__global__ void __launch_bounds__(RTHREADS, 2)
fp8_gemm_rows_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
    using S = Shape<ROWS>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t smem_a = smem_u32(smem), smem_b = smem_a + S::STAGES * S::A_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::BAR_OFF);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + S::STAGES);
    const uint32_t tfull0 = smem_u32(bars + 2 * S::STAGES), tempty0 = tfull0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S::STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int PROMOTERS = ROWS / 32;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < S::STAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(tfull0 + 8 * b, 1); mbar_init(tempty0 + 8 * b, PROMOTERS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tc_alloc(smem_u32(tmem_slot), RTMEM_COLS);
    pdl_wait();                                        // (all of the above is this block's own; from here on, memory is read)
    if (warp == 5) pdl_trigger();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int n0 = blockIdx.x * RN, m0 = blockIdx.y * 128;
    const int KB = (p.K + BK - 1) / BK, batches = (KB + BATCH - 1) / BATCH;

    if (warp == 4) {
        if (lane == 0) {
            bool alive = true;
            uint32_t s = 0, ph = 0;
            for (int kb = 0; kb < KB; ++kb) {
                if (!mbar_wait(empty0 + 8 * s, ph ^ 1, abort_flag, (6 << 8) | 1)) { alive = false; break; }
                mbar_expect_tx(full0 + 8 * s, p.box_rows * BK + RB_BYTES);
                tma_load_2d(&tmB, full0 + 8 * s, smem_b + s * RB_BYTES, kb * BK, n0);
                tma_load_2d(&tmA, full0 + 8 * s, smem_a + s * S::A_BYTES, kb * BK, m0);
                if (++s == S::STAGES) { s = 0; ph ^= 1; }
            }
            if (!alive) {                              // abandoned: let the copies in flight land
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000LL) { }
            }
        }
    } else if (warp == 5) {
        const uint32_t a0 = ((smem_a >> 4) & 0x3FFF) | (1u << 16), b0 = ((smem_b >> 4) & 0x3FFF) | (1u << 16);
        bool alive = true;
        uint32_t s = 0, ph = 0;
        for (int g = 0; g < batches && alive; ++g) {
            const uint32_t b = g & 1;
            if (!mbar_wait_warp(tempty0 + 8 * b, ((g >> 1) & 1) ^ 1, abort_flag, (6 << 8) | 2)) { alive = false; break; }
            const int last = min(BATCH, KB - g * BATCH);
            for (int i = 0; i < last; ++i) {
                if (!mbar_wait_warp(full0 + 8 * s, ph, abort_flag, (6 << 8) | 3)) { alive = false; break; }
                tc_fence_after();
                tc_mma_f8_block<2>(tmem + (b * BATCH + i) * RN, a0 + s * (S::A_BYTES >> 4), b0 + s * (RB_BYTES >> 4), RIDESC);
                tc_commit(empty0 + 8 * s);
                if (++s == S::STAGES) { s = 0; ph ^= 1; }
            }
            if (alive) tc_commit(tfull0 + 8 * b);
        }
    } else if (warp < PROMOTERS) {
        const int row = m0 + warp * 32 + lane;
        const bool valid = row < p.M;
        const float* sa = p.sA + (int64_t)(valid ? row : m0) * p.sa_stride_m;
        const float* sb = p.sB + (int64_t)(n0 / 128) * p.sb_stride_n;
        float acc[RN], a[BATCH], bs[BATCH];
#pragma unroll
        for (int i = 0; i < RN; ++i) acc[i] = 0.0f;
        auto fetch = [&](int g) {
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int kb = min(g * BATCH + i, KB - 1);
                a[i] = ld_scale(sa + (int64_t)kb * p.sa_stride_k);
                bs[i] = ld_scale(sb + (int64_t)kb * p.sb_stride_k);
            }
        };
        fetch(0);
        bool alive = true;
        for (int g = 0; g < batches; ++g) {
            const uint32_t b = g & 1;
            float s[BATCH];
#pragma unroll
            for (int i = 0; i < BATCH; ++i) s[i] = a[i] * bs[i];
            if (g + 1 < batches) fetch(g + 1);
            if (!mbar_wait_warp(tfull0 + 8 * b, (g >> 1) & 1, abort_flag, (6 << 8) | 4)) { alive = false; break; }
            tc_fence_after();
            const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + b * BATCH * RN;
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                if (g * BATCH + i < KB) {
                    uint64_t s2;
                    asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s[i]));
#pragma unroll
                    for (int c = 0; c < RN; c += 16) {
                        float v[16];
                        tc_ld16(taddr + i * RN + c, v);
#pragma unroll
                        for (int j = 0; j < 16; j += 2)
                            asm("{\n\t.reg .b64 a, x;\n\t"
                                "mov.b64 a, {%0, %1};\n\t"
                                "mov.b64 x, {%2, %3};\n\t"
                                "fma.rn.f32x2 a, x, %4, a;\n\t"
                                "mov.b64 {%0, %1}, a;\n\t}"
                                : "+f"(acc[c + j]), "+f"(acc[c + j + 1]) : "f"(v[j]), "f"(v[j + 1]), "l"(s2));
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty0 + 8 * b);
        }
        const bool vec = p.ldc % (16 / (int64_t)sizeof(typename OutT<OUT>::type)) == 0;
        if (alive && valid) {
#pragma unroll
            for (int j = 0; j < RN / 8; ++j) {
                const int col = n0 + j * 8, left = p.N - col;
                if (left > 0) store8<OUT>(p.C, (int64_t)row * p.ldc + col, &acc[j * 8], vec, left);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        tc_dealloc(tmem, RTMEM_COLS);
    }
}

}  // namespace rows
