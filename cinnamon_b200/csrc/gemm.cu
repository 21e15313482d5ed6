// Block-scaled FP8 GEMM for sm_100a: tcgen05 MMAs on e4m3 tiles that TMA stages in
// shared memory, fp32 partial sums in tensor memory (TMEM), and a CUDA-core
// "promotion" of every 128-deep K block: partial * sA[row, kb] * sB[kb, nb] is
// added to fp32 registers.  Semantics of cinnamon's fp8_gemm_kernel
// (src/kernels.py:618-664); the grouped variant follows grouped_gemm_kernel
// (src/kernels.py:466-523) with the same e4m3 operands and scales.
//
// One persistent CTA per SM, 11 warps:
//   warps 0-7   promotion + epilogue: tcgen05.ld a K block's partial tile, scale, accumulate; a finished tile leaves
//               through TMA stores (2-byte outputs, whole tiles) or staged 16-byte stores with row/column predicates
//               (fp32 outputs, ragged expert tails, rows scattered to per-row addresses)
//   warp  8     TMA producer (one lane): A 128x128 B and B 256x128 B tiles, 128-byte swizzle, 4-stage ring
//   warps 9-10  MMA issuers (one lane each) on alternate K blocks: four 128x256x32 MMAs per block into one of two
//               256-column TMEM buffers, so block i+1 runs while block i is promoted; warp 9 owns the TMEM allocation
// Every wait is bounded: when one runs out the kernel records a code in a device status
// word, every role leaves its loop, TMEM is freed and the kernel returns.
#include "common.cuh"
#include "tcgen05.cuh"
#include <cuda.h>
#include <mutex>
#include <atomic>
#include <cmath>
#include <cstdlib>

namespace cinn {

constexpr int BM = 128;            // tile rows
constexpr int BN = 256;            // tile columns (two 128-column scale blocks)
constexpr int BK = 128;            // bytes (= e4m3 elements) per K block: one scale block, one swizzle row
constexpr int STAGES = 4;             // even: each of the two MMA issuers then always meets the same stages, so it
                                      // sees every phase of their barriers (a parity wait cannot skip a phase)
constexpr int C_SLOT_BYTES = BM * 128;   // one TMA-store box: 128 rows x 64 columns of a 2-byte type
constexpr int C_STAGE_BYTES = 2 * C_SLOT_BYTES;   // one slot per column group of promotion warps
constexpr int STORE_ROWS = 32;           // rows of the FP8 kernels' TMA-store boxes: those of one promotion warp
constexpr int A_BYTES = BM * BK;   // 16 KiB
constexpr int B_BYTES = BN * BK;   // 32 KiB
constexpr int EPI_WARPS = 8;                    // four TMEM lane quarters x two column groups
constexpr int WCOLS = BN / (EPI_WARPS / 4);     // accumulator columns per epilogue warp
constexpr int THREADS = (EPI_WARPS + 3) * 32;     // + TMA producer + two MMA issuers
constexpr int TMEM_COLS = 512;
constexpr int MAX_EXPERTS = 384;      // bounded by the shared memory left for the per-expert prefix sums
constexpr int MAX_SEGMENTS = 1024;    // experts of a grouped weight gradient
constexpr int GROUP_M = 16;        // rasterisation: m-tiles per L2 group (dense)

// device status word: 0 = fine, otherwise (role << 8) | reason
__device__ int g_device_status = 0;

struct GemmParams {
    const float* sA; int64_t sa_stride_m, sa_stride_k;
    const float* sB; int64_t sb_stride_k, sb_stride_n, sb_stride_e;
    void* C; int64_t ldc;          // scatter variant: C is a table of byte addresses, one per output row (0 = drop the row)
    int M, N, K;                   // dense: A is (M, K); grouped: M = total rows T
    const int64_t* starts; const int64_t* ends; int E; int b_rows_per_expert;
    int splits;                    // SPLIT: pieces the reduction is cut into; C is then (splits, M, N) fp32 partial sums
    int tma_out;                   // 1: finished tiles leave through TMA stores (2-byte outputs, N % 8 == 0)
    int box_rows;                  // the kernel for few rows: rows of A that one copy brings
};

// ---------------------------------------------------------------------------
// bounded waits
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    return mbar_wait_bounded(bar, parity, abort_flag, code, &g_device_status);
}

// The same wait taken by a whole warp, with one verdict for all its lanes: the promotion warps execute
// warp-collective tcgen05.ld next, so no lane may leave the wait on its own.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    const bool ok = mbar_wait(bar, parity, abort_flag, code);
    return __all_sync(0xffffffffu, ok);
}

// fp32 load through the read-only path, pinned in program order
__device__ __forceinline__ float ld_scale(const float* p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// Instruction descriptor for kind::f8f6f4: fp32 accumulate, e4m3 x e4m3, A K-major.
__host__ __device__ constexpr uint32_t make_idesc(bool b_mn_major) {
    return (1u << 4)                              // D format: fp32
           | (0u << 7) | (0u << 10)               // A, B format: e4m3
           | (0u << 15)                           // A major: K
           | ((b_mn_major ? 1u : 0u) << 16)       // B major
           | ((uint32_t)(BN >> 3) << 17)          // N
           | ((uint32_t)(BM >> 4) << 24);         // M
}

// ---------------------------------------------------------------------------
// tile schedule shared by all roles
// ---------------------------------------------------------------------------
struct TileInfo {
    int m0;        // first row of A / C
    int m_end;     // one past the last valid row for this tile
    int n0;        // first output column
    int expert;
};

template <bool GROUPED>
__device__ __forceinline__ int total_tiles(const GemmParams& p, const int* cum) {
    const int n_tiles = (p.N + BN - 1) / BN;
    if constexpr (GROUPED) return cum[p.E] * n_tiles;
    else return ((p.M + BM - 1) / BM) * n_tiles;
}

template <bool GROUPED>
__device__ __forceinline__ TileInfo tile_info(const GemmParams& p, const int* cum, int t) {
    TileInfo ti;
    const int n_tiles = (p.N + BN - 1) / BN;
    if constexpr (GROUPED) {
        const int mt = t / n_tiles;
        ti.n0 = (t - mt * n_tiles) * BN;
        int lo = 0, hi = p.E;                      // largest e with cum[e] <= mt
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (cum[mid] <= mt) lo = mid; else hi = mid;
        }
        ti.expert = lo;
        const long long s = p.starts[lo], e = p.ends[lo];
        ti.m0 = (int)s + (mt - cum[lo]) * BM;
        ti.m_end = (int)(e < (long long)p.M ? e : (long long)p.M);
    } else {
        const int m_tiles = (p.M + BM - 1) / BM;
        const int per_group = GROUP_M * n_tiles;
        const int g = t / per_group;
        const int first_m = g * GROUP_M;
        const int gsize = min(GROUP_M, m_tiles - first_m);
        const int r = t - g * per_group;
        ti.m0 = (first_m + r % gsize) * BM;
        ti.n0 = (r / gsize) * BN;
        ti.m_end = p.M;
        ti.expert = 0;
    }
    return ti;
}

// grouped: cum[e] = row tiles (of `rows`) of the experts before e, cum[E] = all of them; by one warp
__device__ __forceinline__ void tile_prefix_sum(const GemmParams& p, int* cum, int rows, int lane) {
    int carry = 0;
    for (int base = 0; base < p.E; base += 32) {
        const int e = base + lane;
        int cnt = 0;
        if (e < p.E) {
            long long s = p.starts[e], t = p.ends[e];
            if (t > (long long)p.M) t = p.M;
            if (s < 0) s = 0;
            if (t > s) cnt = (int)((t - s + rows - 1) / rows);
        }
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (e < p.E) cum[e] = carry + incl - cnt;
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) cum[p.E] = carry;
}

template <int OUT> struct OutT;
template <> struct OutT<CINN_BF16> { using type = __nv_bfloat16; };
template <> struct OutT<CINN_F16> { using type = __half; };
template <> struct OutT<CINN_F32> { using type = float; };
template <> struct OutT<CINN_F32_BF16> { using type = float; };   // fp32 storage of the bf16-rounded value

template <int OUT>
__device__ __forceinline__ void store8(void* C, int64_t off, const float* a, bool vec, int ncols) {
    using T = typename OutT<OUT>::type;
    T* dst = reinterpret_cast<T*>(C) + off;
    float b[8];
    if constexpr (OUT == CINN_F32_BF16) {
#pragma unroll
        for (int i = 0; i < 8; ++i) b[i] = __bfloat162float(__float2bfloat16_rn(a[i]));
        a = b;
    }
    if (vec && ncols >= 8) {
        if constexpr (OUT == CINN_F32 || OUT == CINN_F32_BF16) {
            reinterpret_cast<float4*>(dst)[0] = make_float4(a[0], a[1], a[2], a[3]);
            reinterpret_cast<float4*>(dst)[1] = make_float4(a[4], a[5], a[6], a[7]);
        } else if constexpr (OUT == CINN_BF16) {
            uint4 v;
            __nv_bfloat162 t0 = __floats2bfloat162_rn(a[0], a[1]), t1 = __floats2bfloat162_rn(a[2], a[3]);
            __nv_bfloat162 t2 = __floats2bfloat162_rn(a[4], a[5]), t3 = __floats2bfloat162_rn(a[6], a[7]);
            v.x = *reinterpret_cast<uint32_t*>(&t0); v.y = *reinterpret_cast<uint32_t*>(&t1);
            v.z = *reinterpret_cast<uint32_t*>(&t2); v.w = *reinterpret_cast<uint32_t*>(&t3);
            *reinterpret_cast<uint4*>(dst) = v;
        } else {
            uint4 v;
            __half2 t0 = __floats2half2_rn(a[0], a[1]), t1 = __floats2half2_rn(a[2], a[3]);
            __half2 t2 = __floats2half2_rn(a[4], a[5]), t3 = __floats2half2_rn(a[6], a[7]);
            v.x = *reinterpret_cast<uint32_t*>(&t0); v.y = *reinterpret_cast<uint32_t*>(&t1);
            v.z = *reinterpret_cast<uint32_t*>(&t2); v.w = *reinterpret_cast<uint32_t*>(&t3);
            *reinterpret_cast<uint4*>(dst) = v;
        }
    } else {
        for (int i = 0; i < 8 && i < ncols; ++i) {
            if constexpr (OUT == CINN_F32 || OUT == CINN_F32_BF16) dst[i] = a[i];
            else if constexpr (OUT == CINN_BF16) dst[i] = __float2bfloat16_rn(a[i]);
            else dst[i] = __float2half_rn(a[i]);
        }
    }
}

// Tile store through shared memory.  Each promotion thread owns one output row; storing it directly would
// make every warp-wide store touch 32 different rows (32 cache lines per instruction).  Instead the warp
// stages 64 bytes of each of its 32 rows (XOR-swizzled 16-byte slots, conflict-free both ways) and writes
// them back out as 8 rows x 64 contiguous bytes per instruction.  `stage` is this warp's 2 KiB.
template <int OUT>
__device__ __forceinline__ uint4 pack16(const float* a) {
    uint4 v;
    if constexpr (OUT == CINN_F32) {
        v = make_uint4(__float_as_uint(a[0]), __float_as_uint(a[1]), __float_as_uint(a[2]), __float_as_uint(a[3]));
    } else if constexpr (OUT == CINN_F32_BF16) {
        // two packed conversions, then each half widened again by a shift / a mask
        __nv_bfloat162 t0 = __floats2bfloat162_rn(a[0], a[1]), t1 = __floats2bfloat162_rn(a[2], a[3]);
        const uint32_t p0 = *reinterpret_cast<uint32_t*>(&t0), p1 = *reinterpret_cast<uint32_t*>(&t1);
        v = make_uint4(p0 << 16, p0 & 0xffff0000u, p1 << 16, p1 & 0xffff0000u);
    } else if constexpr (OUT == CINN_BF16) {
        __nv_bfloat162 t0 = __floats2bfloat162_rn(a[0], a[1]), t1 = __floats2bfloat162_rn(a[2], a[3]);
        __nv_bfloat162 t2 = __floats2bfloat162_rn(a[4], a[5]), t3 = __floats2bfloat162_rn(a[6], a[7]);
        v = make_uint4(*reinterpret_cast<uint32_t*>(&t0), *reinterpret_cast<uint32_t*>(&t1), *reinterpret_cast<uint32_t*>(&t2), *reinterpret_cast<uint32_t*>(&t3));
    } else {
        __half2 t0 = __floats2half2_rn(a[0], a[1]), t1 = __floats2half2_rn(a[2], a[3]);
        __half2 t2 = __floats2half2_rn(a[4], a[5]), t3 = __floats2half2_rn(a[6], a[7]);
        v = make_uint4(*reinterpret_cast<uint32_t*>(&t0), *reinterpret_cast<uint32_t*>(&t1), *reinterpret_cast<uint32_t*>(&t2), *reinterpret_cast<uint32_t*>(&t3));
    }
    return v;
}

template <int OUT, int NCOLS, bool SCATTER = false>
__device__ __forceinline__ void store_rows_staged(const float* acc, uint8_t* stage, void* C, int64_t ldc, int row0, int m_end,
                                                  int col0, int N, int lane) {
    using T = typename OutT<OUT>::type;
    constexpr int PER16 = 16 / (int)sizeof(T);      // elements per 16-byte slot
    constexpr int PER64 = 4 * PER16;                // elements per staged row piece
#pragma unroll
    for (int ps = 0; ps < NCOLS / PER64; ++ps) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            *reinterpret_cast<uint4*>(stage + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = pack16<OUT>(&acc[ps * PER64 + c * PER16]);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = i * 8 + (lane >> 2), c = lane & 3;
            const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 64 + ((c ^ ((r >> 1) & 3)) << 4));
            const int grow = row0 + r, gcol = col0 + ps * PER64 + c * PER16;
            if constexpr (SCATTER) {
                // C is a table of byte addresses, one per row; the rows may live in another GPU's memory
                if (grow < m_end && gcol < N) {
                    T* dst = reinterpret_cast<T*>(reinterpret_cast<const long long*>(C)[grow]);
                    if (dst) *reinterpret_cast<uint4*>(dst + gcol) = v;
                }
            } else {
                if (grow < m_end && gcol < N) *reinterpret_cast<uint4*>(reinterpret_cast<T*>(C) + (int64_t)grow * ldc + gcol) = v;
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------
// SPLIT: a few tiles with a long reduction leave most SMs idle, so every tile is computed p.splits times over different
// K blocks (tile t of n_total belongs to piece t / tiles) and the partial sums are added by split_sum_kernel.
template <bool B_MN, bool GROUPED, int OUT, bool SCATTER = false, bool SPLIT = false>
__global__ void __launch_bounds__(THREADS, 1)
fp8_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmC, const GemmParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    // layout: operand stages | output staging (32 KiB, 1024-aligned) | barriers and flags (256 B) | expert prefix sums
    uint8_t* smem_a = smem;
    uint8_t* smem_b = smem + STAGES * A_BYTES;
    uint8_t* c_stage = smem + STAGES * (A_BYTES + B_BYTES);
    uint64_t* bars = reinterpret_cast<uint64_t*>(c_stage + C_STAGE_BYTES);
    // bars[0..S) full, [S..2S) empty, [2S..2S+2) tmem full, [2S+2..2S+4) tmem empty
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint8_t* store_stage = c_stage;                                        // 2 KiB per promotion warp (non-TMA path)
    int* cum = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(bars) + 256);   // grouped: E + 1 prefix counts of m-tiles

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);
    const uint32_t tfull0 = smem_u32(bars + 2 * STAGES), tempty0 = smem_u32(bars + 2 * STAGES + 2);

    if (threadIdx.x == 0) *abort_flag = 0;
    if (warp == EPI_WARPS && lane == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(tfull0 + 8 * b, 1); mbar_init(tempty0 + 8 * b, EPI_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == EPI_WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();                                    // (all of the above is this block's own; from here on, memory is read)
    if (warp == EPI_WARPS + 1) pdl_trigger();
    if constexpr (GROUPED) {
        if (warp == 0) tile_prefix_sum(p, cum, BM, lane);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int KB_all = (p.K + BK - 1) / BK;
    const int n_tiles_all = total_tiles<GROUPED>(p, cum);
    const int n_total = SPLIT ? n_tiles_all * p.splits : n_tiles_all;
    // tile t -> its K blocks [kb0, kb0 + KB) and its place in the output
    auto blocks_of = [&](int t, int& kb0, int& KB) {
        if constexpr (SPLIT) {
            const int piece = t / n_tiles_all;
            kb0 = (int)((int64_t)KB_all * piece / p.splits);
            KB = (int)((int64_t)KB_all * (piece + 1) / p.splits) - kb0;
        } else {
            kb0 = 0; KB = KB_all;
        }
    };
    auto tile_of = [&](int t) { return tile_info<GROUPED>(p, cum, SPLIT ? t % n_tiles_all : t); };

    if (warp >= EPI_WARPS) {
      if (warp == EPI_WARPS) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            uint32_t it = 0;
            bool alive = true;
            for (int t = blockIdx.x; t < n_total && alive; t += gridDim.x) {
                const TileInfo ti = tile_of(t);
                int kb0, KB;
                blocks_of(t, kb0, KB);
                const int b_row0 = GROUPED ? ti.expert * p.b_rows_per_expert : 0;
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    if (!mbar_wait(empty0 + 8 * s, ph ^ 1, abort_flag, (1 << 8) | 1)) { alive = false; break; }
                    const uint32_t fb = full0 + 8 * s;
                    mbar_expect_tx(fb, A_BYTES + B_BYTES);
                    const int k = (kb0 + kb) * BK;
                    tma_load_2d(&tmA, fb, smem_u32(smem_a + s * A_BYTES), k, ti.m0);
                    if constexpr (!B_MN) {
                        tma_load_2d(&tmB, fb, smem_u32(smem_b + s * B_BYTES), k, b_row0 + ti.n0);
                    } else {
                        tma_load_2d(&tmB, fb, smem_u32(smem_b + s * B_BYTES), ti.n0, b_row0 + k);
                        tma_load_2d(&tmB, fb, smem_u32(smem_b + s * B_BYTES + B_BYTES / 2), ti.n0 + 128, b_row0 + k);
                    }
                }
            }
            if (!alive) {
                // abandoned: let the copies already issued land before shared memory is given up
                const uint32_t issued = it;
                for (uint32_t j = (issued > STAGES ? issued - STAGES : 0); j < issued; ++j) {
                    const long long t0 = clock64();
                    while (!mbar_try_wait(full0 + 8 * (j % STAGES), (j / STAGES) & 1)) {
                        if (clock64() - t0 > WAIT_LIMIT_CYCLES) break;
                    }
                }
            }
        }
    } else {
        // ------------------------------ MMA issuers ------------------------------
        // Two warps take alternate K blocks (one TMEM buffer each), each as a whole with one elected lane issuing: with
        // warp-uniform control flow the descriptors live in uniform registers.  Issued from a branch of one lane, a K block's
        // four MMAs and its commits took their issuer 600 cycles, more than the 512 of the arithmetic, and with the probes
        // around them that (and not the promotion) set the pace.
        {
            constexpr uint32_t idesc = make_idesc(B_MN);
            const uint32_t mine = (uint32_t)(warp - (EPI_WARPS + 1));
            const uint32_t a0 = ((smem_u32(smem_a) >> 4) & 0x3FFF) | (1u << 16);
            const uint32_t b0 = ((smem_u32(smem_b) >> 4) & 0x3FFF) | ((B_MN ? (uint32_t)B_BYTES / 2 >> 4 : 1u) << 16);
            uint32_t it = 0, last = 0xffffffffu;
            bool alive = true;
            for (int t = blockIdx.x; t < n_total && alive; t += gridDim.x) {
                int kb0, KB;
                blocks_of(t, kb0, KB);
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    if ((it & 1u) != mine) continue;
                    last = it;
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    const uint32_t b = it & 1, bph = (it >> 1) & 1;
                    // operands first (they landed long ago: this costs one barrier probe, taken while
                    // the epilogue still works on the buffer), then the TMEM buffer
                    if (!mbar_wait_warp(full0 + 8 * s, ph, abort_flag, (2 << 8) | 1)) { alive = false; break; }
                    if (!mbar_wait_warp(tempty0 + 8 * b, bph ^ 1, abort_flag, (2 << 8) | 2)) { alive = false; break; }
                    tc_fence_after();
                    tc_mma_f8_block<B_MN ? 256 : 2>(tmem_base + b * BN, a0 + s * (A_BYTES >> 4), b0 + s * (B_BYTES >> 4), idesc);
                    tc_commit(tfull0 + 8 * b);      // the partial tile is ready for promotion once these MMAs retire
                    tc_commit(empty0 + 8 * s);      // and the stage may be refilled
                }
            }
            // every MMA issued above must have retired before tensor memory is freed
            if (alive && last != 0xffffffffu) mbar_wait(tfull0 + 8 * (last & 1), (last >> 1) & 1, abort_flag, (2 << 8) | 3);
        }
      }
    } else {
        // ------------------------------ epilogue ------------------------------
        const int q = warp & 3, h = warp >> 2;
        uint32_t it = 0;
        bool alive = true;
        const bool vec_ok = (OUT == CINN_F32 || OUT == CINN_F32_BF16) ? (p.ldc % 4 == 0) : (p.ldc % 8 == 0);
        // The first three scale pairs of a tile are fetched while the previous tile is being stored, so that
        // a tile does not start with an exposed round trip to L2 (it matters when K is only a few blocks).
        float sa0 = 0.f, sb0 = 0.f, sa1 = 0.f, sb1 = 0.f, sa2 = 0.f, sb2 = 0.f;
        auto scale_ptrs = [&](const TileInfo& ti, int kb0, const float*& sa_ptr, const float*& sb_ptr) {
            const int row = ti.m0 + q * 32 + lane;
            const int col0 = ti.n0 + h * WCOLS;
            sa_ptr = p.sA + (int64_t)(row < ti.m_end ? row : ti.m0) * p.sa_stride_m;
            sb_ptr = p.sB + (int64_t)ti.expert * p.sb_stride_e + (int64_t)(col0 < p.N ? col0 / 128 : 0) * p.sb_stride_n;
            if constexpr (SPLIT) {
                sa_ptr += (int64_t)kb0 * p.sa_stride_k;
                sb_ptr += (int64_t)kb0 * p.sb_stride_k;
            }
        };
        auto prefetch_scales = [&](int t) {
            const TileInfo ti = tile_of(t);
            const float *sa_ptr, *sb_ptr;
            int kb0, KB;
            blocks_of(t, kb0, KB);
            scale_ptrs(ti, kb0, sa_ptr, sb_ptr);
            sa0 = ld_scale(sa_ptr); sb0 = ld_scale(sb_ptr);
            if (KB > 1) { sa1 = ld_scale(sa_ptr + p.sa_stride_k); sb1 = ld_scale(sb_ptr + p.sb_stride_k); }
            if (KB > 2) { sa2 = ld_scale(sa_ptr + 2 * p.sa_stride_k); sb2 = ld_scale(sb_ptr + 2 * p.sb_stride_k); }
        };
        if ((int)blockIdx.x < n_total) prefetch_scales(blockIdx.x);
        for (int t = blockIdx.x; t < n_total && alive; t += gridDim.x) {
            const TileInfo ti = tile_of(t);
            int kb0, KB;
            blocks_of(t, kb0, KB);
            void* C = SPLIT ? (void*)(reinterpret_cast<float*>(p.C) + (int64_t)(t / n_tiles_all) * p.M * p.N) : p.C;
            const int row = ti.m0 + q * 32 + lane;
            const bool rvalid = row < ti.m_end;
            const int col0 = ti.n0 + h * WCOLS;
            const bool cvalid = col0 < p.N;
            const float *sa_ptr, *sb_ptr;
            scale_ptrs(ti, kb0, sa_ptr, sb_ptr);
            float acc[WCOLS];
#pragma unroll
            for (int i = 0; i < WCOLS; ++i) acc[i] = 0.0f;
            // within a tile scales are fetched three K blocks ahead with loads the compiler may not move
            // (a load sunk to its use would expose a full L2 round trip in every K block)
            for (int kb = 0; kb < KB; ++kb, ++it) {
                const float s = sa0 * sb0;
                sa0 = sa1; sb0 = sb1; sa1 = sa2; sb1 = sb2;
                if (kb + 3 < KB) {
                    sa2 = ld_scale(sa_ptr + (int64_t)(kb + 3) * p.sa_stride_k);
                    sb2 = ld_scale(sb_ptr + (int64_t)(kb + 3) * p.sb_stride_k);
                }
                const uint32_t b = it & 1, bph = (it >> 1) & 1;
                if (!mbar_wait_warp(tfull0 + 8 * b, bph, abort_flag, (3 << 8) | 1)) { alive = false; break; }
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + b * BN + h * WCOLS;
                // packed fp32x2 FMAs: half the issue slots of 128 scalar ones, the same IEEE result in every lane
                uint64_t s2;
                asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s));
#pragma unroll
                for (int c = 0; c < WCOLS / 16; ++c) {
                    float v[16];
                    tc_ld16(taddr + c * 16, v);
#pragma unroll
                    for (int j = 0; j < 16; j += 2)
                        asm("{\n\t.reg .b64 a, x;\n\t"
                            "mov.b64 a, {%0, %1};\n\t"
                            "mov.b64 x, {%2, %3};\n\t"
                            "fma.rn.f32x2 a, x, %4, a;\n\t"
                            "mov.b64 {%0, %1}, a;\n\t}"
                            : "+f"(acc[c * 16 + j]), "+f"(acc[c * 16 + j + 1]) : "f"(v[j]), "f"(v[j + 1]), "l"(s2));
                }
                // (Measured alternatives, all slower on B200: wider TMEM loads with a larger register budget,
                // double-buffered loads, sixteen promotion warps.  Packed FMAs are worth 1 - 2 %.)
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty0 + 8 * b);
            }
            if (alive && t + (int)gridDim.x < n_total) prefetch_scales(t + gridDim.x);
            constexpr bool TMA_OUT = (OUT == CINN_BF16 || OUT == CINN_F16);
            // Rows that all belong to the tile leave through TMA stores.  Every promotion warp owns a 4 KiB box: its lanes
            // drop 64 columns of their rows into it (16-byte chunks, 128-byte swizzle), one lane hands the box to the TMA
            // unit, and the warp repeats for its other 64 columns once the unit has read the box.  (No warp waits for
            // another: see the two-SM kernel.)  Storing one row per thread straight from registers costs thousands of
            // cycles per tile, and so do shared-memory round trips next to a busy tensor pipe.
            const bool whole = !GROUPED || row - lane + STORE_ROWS <= ti.m_end;
            if (TMA_OUT && alive && p.tma_out && whole) {
                const uint32_t slot = smem_u32(c_stage) + warp * STORE_ROWS * 128;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    if (lane == 0) tma_store_wait_read();             // the unit has finished reading this box
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint4 v = pack16<OUT>(&acc[r * 64 + j * 8]);
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(slot + lane * 128 + ((j ^ (lane & 7)) << 4)),
                                     "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        const int col = col0 + r * 64;
                        if (col < p.N) tma_store_2d(&tmC, slot, col, row);
                        tma_store_commit();
                    }
                    __syncwarp();   // the lane rejoins its warp before the next warp-collective instruction
                }
            } else if (alive && vec_ok && !(TMA_OUT && p.tma_out)) {
                // warp-uniform: every lane takes part in the staging even if its own row is past the end
                if (cvalid) store_rows_staged<OUT, WCOLS, SCATTER>(acc, store_stage + warp * 2048, C, p.ldc, ti.m0 + q * 32, ti.m_end, col0, p.N, lane);
            } else if (alive && rvalid && cvalid) {
                const int64_t base = (int64_t)row * p.ldc + col0;
#pragma unroll
                for (int j = 0; j < WCOLS / 8; ++j) {
                    const int ncols = p.N - (col0 + j * 8);
                    if (ncols > 0) store8<OUT>(C, base + j * 8, &acc[j * 8], vec_ok, ncols);
                }
            }
        }
        if (lane == 0) tma_store_wait_all();                // this warp's boxes have reached global memory
    }

    tc_fence_before();
    __syncthreads();
    if (warp == EPI_WARPS + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

#include "gemm_pair.cuh"
#include "gemm_rows.cuh"
#include "gemm16.cuh"

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn get_encode() {
    static EncodeFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeFn>(p);
    });
    return fn;
}

int encode_map_2d(CUtensorMap* map, const void* base, uint64_t inner, uint64_t rows, uint64_t pitch_bytes,
                  uint32_t box_inner, uint32_t box_rows, CUtensorMapDataType dtype, CUtensorMapSwizzle swizzle) {
    EncodeFn enc = get_encode();
    if (!enc) { set_error("cuTensorMapEncodeTiled is not available from the CUDA driver"); return CINN_ERR_CUDA; }
    cuuint64_t dims[2] = {inner, rows};
    cuuint64_t strides[1] = {pitch_bytes};
    cuuint32_t box[2] = {box_inner, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, dtype, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_ERROR_INVALID_CONTEXT || r == CUDA_ERROR_NOT_INITIALIZED) {
        // a thread that has made no runtime call yet (an autograd worker, say) has no context bound:
        // let the runtime bind the device's primary context, then encode again
        cudaFree(nullptr);
        r = enc(map, dtype, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult %d (base %p inner %llu rows %llu pitch %llu)", (int)r, base,
                  (unsigned long long)inner, (unsigned long long)rows, (unsigned long long)pitch_bytes);
        return CINN_ERR_CUDA;
    }
    return CINN_OK;
}

int encode_map(CUtensorMap* map, const void* base, uint32_t rank, const uint64_t* dims, const uint64_t* strides, const uint32_t* box,
               CUtensorMapDataType dtype, CUtensorMapSwizzle swizzle) {
    EncodeFn enc = get_encode();
    if (!enc) { set_error("cuTensorMapEncodeTiled is not available from the CUDA driver"); return CINN_ERR_CUDA; }
    const cuuint32_t ones[5] = {1, 1, 1, 1, 1};
    cuuint64_t d[5], st[4];
    cuuint32_t bx[5];
    for (uint32_t i = 0; i < rank; ++i) { d[i] = dims[i]; bx[i] = box[i]; if (i) st[i - 1] = strides[i - 1]; }
    auto go = [&] {
        return enc(map, dtype, rank, const_cast<void*>(base), d, st, bx, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = go();
    if (r == CUDA_ERROR_INVALID_CONTEXT || r == CUDA_ERROR_NOT_INITIALIZED) { cudaFree(nullptr); r = go(); }
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult %d (base %p, %u dimensions)", (int)r, base, rank);
        return CINN_ERR_CUDA;
    }
    return CINN_OK;
}

// 3-D map: `planes` matrices of (rows, inner), boxes of box_inner columns x box_rows of one matrix; rows past a matrix's end
// read as zeros instead of its neighbour's, and are not written
int encode_map_3d(CUtensorMap* map, const void* base, uint64_t inner, uint64_t rows, uint64_t planes, uint64_t pitch_bytes,
                  uint32_t box_rows, CUtensorMapDataType dtype, uint32_t box_inner, CUtensorMapSwizzle swizzle) {
    EncodeFn enc = get_encode();
    if (!enc) { set_error("cuTensorMapEncodeTiled is not available from the CUDA driver"); return CINN_ERR_CUDA; }
    cuuint64_t dims[3] = {inner, rows, planes};
    cuuint64_t strides[2] = {pitch_bytes, pitch_bytes * rows};
    cuuint32_t box[3] = {box_inner, box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    auto go = [&] {
        return enc(map, dtype, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = go();
    if (r == CUDA_ERROR_INVALID_CONTEXT || r == CUDA_ERROR_NOT_INITIALIZED) { cudaFree(nullptr); r = go(); }
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult %d (base %p inner %llu rows %llu planes %llu)", (int)r, base,
                  (unsigned long long)inner, (unsigned long long)rows, (unsigned long long)planes);
        return CINN_ERR_CUDA;
    }
    return CINN_OK;
}

// GEMM operands and outputs: 128-byte swizzle; `pitch` in BYTES
static int make_map(CUtensorMap* map, const void* base, uint64_t inner, uint64_t rows, uint64_t pitch, uint32_t box_inner,
                    uint32_t box_rows, CUtensorMapDataType dtype = CU_TENSOR_MAP_DATA_TYPE_UINT8) {
    return encode_map_2d(map, base, inner, rows, pitch, box_inner, box_rows, dtype, CU_TENSOR_MAP_SWIZZLE_128B);
}

static size_t smem_bytes(int E) {
    size_t n = (size_t)STAGES * (A_BYTES + B_BYTES) + C_STAGE_BYTES + 1024 + 256 + 4 * (size_t)(E + 2);
    return n;
}

// Output map for the TMA-store epilogue: (rows, N) of a 2-byte type, boxes of 64 columns x 128 rows, 128-byte swizzle.
// Sets p.tma_out; when the output cannot go through TMA the (unused) operand map is passed in its place.
static int make_out_map(CUtensorMap* tc, const CUtensorMap& fallback, GemmParams& p, int out_dtype, int64_t rows,
                        int box_rows, bool fp32_boxes = false) {
    p.tma_out = 0;
    *tc = fallback;
    if (((uintptr_t)p.C & 15) != 0) return CINN_OK;               // TMA wants a 16-byte aligned base; plain stores otherwise
    if (fp32_boxes && (out_dtype == CINN_F32 || out_dtype == CINN_F32_BF16) && p.N % 4 == 0) {
        // the two-SM kernel also sends 4-byte outputs through TMA: boxes of 32 columns
        int rc = make_map(tc, p.C, (uint64_t)p.N, (uint64_t)rows, (uint64_t)p.ldc * 4, 32, box_rows, CU_TENSOR_MAP_DATA_TYPE_FLOAT32);
        if (rc) return rc;
        p.tma_out = 1;
        return CINN_OK;
    }
    if ((out_dtype == CINN_BF16 || out_dtype == CINN_F16) && p.N % 8 == 0) {
        int rc = make_map(tc, p.C, (uint64_t)p.N, (uint64_t)rows, (uint64_t)p.ldc * 2, 64, box_rows,
                          out_dtype == CINN_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
        if (rc) return rc;
        p.tma_out = 1;
    }
    return CINN_OK;
}

template <bool B_MN, bool GROUPED, int OUT, bool SCATTER = false, bool SPLIT = false>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GemmParams& p, int grid,
                  cudaStream_t st) {
    constexpr auto kern = fp8_gemm_kernel<B_MN, GROUPED, OUT, SCATTER, SPLIT>;
    const size_t smem = smem_bytes(GROUPED ? p.E : 0);
    int rc = allow_smem_once<kern>(smem_bytes(GROUPED ? MAX_EXPERTS : 0));
    if (rc) return rc;
    CINN_CHECK_CUDA(launch_dependent(kern, grid, THREADS, smem, st, ta, tb, tc, p));
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

template <bool B_MN, bool GROUPED>
static int launch_out(const CUtensorMap& ta, const CUtensorMap& tb, GemmParams& p, int out_dtype, int grid,
                      cudaStream_t st) {
    CUtensorMap tc;
    int rc = make_out_map(&tc, ta, p, out_dtype, p.M, STORE_ROWS);
    if (rc) return rc;
    switch (out_dtype) {
        case CINN_BF16: return launch<B_MN, GROUPED, CINN_BF16>(ta, tb, tc, p, grid, st);
        case CINN_F32: return launch<B_MN, GROUPED, CINN_F32>(ta, tb, tc, p, grid, st);
        case CINN_F16: return launch<B_MN, GROUPED, CINN_F16>(ta, tb, tc, p, grid, st);
        case CINN_F32_BF16: return launch<B_MN, GROUPED, CINN_F32_BF16>(ta, tb, tc, p, grid, st);
        default: set_error("GEMM: unknown output dtype tag %d", out_dtype); return CINN_ERR_INVALID;
    }
}

template <bool B_MN, int OUT, bool GK = false, bool GR = false, bool OWN = false>
static int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GemmParams& p, int clusters,
                       cudaStream_t st) {
    constexpr auto kern = pair::fp8_gemm_pair_kernel<B_MN, OUT, GK, GR, OWN>;
    constexpr int MOST = GR ? MAX_EXPERTS : GK ? MAX_SEGMENTS : -2;              // (counts in shared memory, one per expert and two)
    const size_t smem = pair::PSMEM_BYTES + (GR || GK ? 4 * (size_t)(p.E + 2) : 0);
    int rc = allow_smem_once<kern>(pair::PSMEM_BYTES + 4 * (size_t)(MOST + 2));
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * clusters, 1, 1);
    cfg.blockDim = dim3(pair::PTHREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    CINN_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, ta, tb, tc, p));
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

template <bool B_MN>
static int launch_pair_out(const CUtensorMap& ta, const CUtensorMap& tb, GemmParams& p, int out_dtype, int clusters,
                           cudaStream_t st) {
    CUtensorMap tc;
    int rc = make_out_map(&tc, ta, p, out_dtype, p.M, STORE_ROWS, true);
    if (rc) return rc;
    switch (out_dtype) {
        case CINN_BF16: return launch_pair<B_MN, CINN_BF16>(ta, tb, tc, p, clusters, st);
        case CINN_F32: return launch_pair<B_MN, CINN_F32>(ta, tb, tc, p, clusters, st);
        case CINN_F16: return launch_pair<B_MN, CINN_F16>(ta, tb, tc, p, clusters, st);
        case CINN_F32_BF16: return launch_pair<B_MN, CINN_F32_BF16>(ta, tb, tc, p, clusters, st);
        default: set_error("GEMM: unknown output dtype tag %d", out_dtype); return CINN_ERR_INVALID;
    }
}

// Two-SM pairs serve dense problems whose waves of 256 x 256 tiles cost no more than the one-SM kernel's (dense_plan), and
// grouped ones with enough rows per expert; CINN_GEMM_PAIR=0 keeps every problem on the one-SM kernel.
static int pair_mode() {
    static int mode = -1;
    if (mode < 0) {
        const char* e = getenv("CINN_GEMM_PAIR");
        mode = (e && e[0] == '0') ? 0 : (e && e[0] == '2') ? 2 : 1;     // 2 = pairs for every layout (tests)
    }
    return mode;
}

// The persistent GEMM kernels normally take every SM.  A caller that wants other kernels to run beside them
// (the send/receive kernels of an all-to-all on another stream) can cap the number of SMs they occupy.  Read once per call:
// another thread may change it meanwhile.
static std::atomic<int> g_gemm_sm_limit{0};
static inline int gemm_sms() {
    const int lim = g_gemm_sm_limit.load(std::memory_order_relaxed), all = sm_count();
    return (lim > 0 && lim < all) ? lim : all;
}
bool gemm_sms_capped() { return g_gemm_sm_limit.load(std::memory_order_relaxed) > 0 && gemm_sms() < sm_count(); }
int set_gemm_sm_limit(int n) { return g_gemm_sm_limit.exchange(n < 0 ? 0 : n); }

static inline bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// ---------------------------------------------------------------------------
// dense problems: which kernel, and into how many pieces the reduction is cut
// ---------------------------------------------------------------------------
// Sum of the `splits` partial results of every output element, in a fixed order (the result does not depend on which
// piece finished first), rounded once.  Bound by reading the pieces, which were just written and mostly sit in L2.
template <int OUT>
__global__ void __launch_bounds__(256)
split_sum_kernel(const float* __restrict__ part, void* __restrict__ out, int64_t n, int splits) {
    using T = typename OutT<OUT>::type;
    pdl_wait();
    const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 4;
    if (i >= n) return;
    float a[4] = {0.f, 0.f, 0.f, 0.f};
    const bool vec = i + 4 <= n && (n & 3) == 0;
    if (vec) {
#pragma unroll 4
        for (int s = 0; s < splits; ++s) {
            const float4 v = __ldcs(reinterpret_cast<const float4*>(part + s * n + i));
            a[0] += v.x; a[1] += v.y; a[2] += v.z; a[3] += v.w;
        }
    } else {
        for (int s = 0; s < splits; ++s)
            for (int j = 0; j < 4 && i + j < n; ++j) a[j] += part[s * n + i + j];
    }
    T* dst = reinterpret_cast<T*>(out) + i;
    if constexpr (OUT == CINN_F32 || OUT == CINN_F32_BF16) {
        if constexpr (OUT == CINN_F32_BF16)
            for (int j = 0; j < 4; ++j) a[j] = __bfloat162float(__float2bfloat16_rn(a[j]));
        if (vec) *reinterpret_cast<float4*>(dst) = make_float4(a[0], a[1], a[2], a[3]);
        else for (int j = 0; j < 4 && i + j < n; ++j) dst[j] = a[j];
    } else {
        T h[4];
        for (int j = 0; j < 4; ++j) {
            if constexpr (OUT == CINN_BF16) h[j] = __float2bfloat16_rn(a[j]);
            else h[j] = __float2half_rn(a[j]);
        }
        if (vec) *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(h);
        else for (int j = 0; j < 4 && i + j < n; ++j) dst[j] = h[j];
    }
}

static int launch_split_sum(const float* part, void* out, int64_t n, int splits, int out_dtype, cudaStream_t st) {
    const unsigned grid = (unsigned)((n + 1023) / 1024);
    switch (out_dtype) {
        case CINN_BF16: CINN_CHECK_CUDA(launch_dependent(split_sum_kernel<CINN_BF16>, grid, 256, 0, st, part, out, n, splits)); break;
        case CINN_F32: CINN_CHECK_CUDA(launch_dependent(split_sum_kernel<CINN_F32>, grid, 256, 0, st, part, out, n, splits)); break;
        case CINN_F16: CINN_CHECK_CUDA(launch_dependent(split_sum_kernel<CINN_F16>, grid, 256, 0, st, part, out, n, splits)); break;
        case CINN_F32_BF16: CINN_CHECK_CUDA(launch_dependent(split_sum_kernel<CINN_F32_BF16>, grid, 256, 0, st, part, out, n, splits)); break;
        default: set_error("GEMM: unknown output dtype tag %d", out_dtype); return CINN_ERR_INVALID;
    }
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

// us that a wave of tiles of a reduction over K takes on single SMs and on pairs, fitted to 130 calls of both kernels one after
// another (M 256 ... 16384, N 256 ... 8192, K 128 ... 16384; 4 % off on average)
static double tile_cost(int64_t K, bool pair) {
    const double KB = (double)((K + BK - 1) / BK);
    return pair ? KB * 0.44 + 1.75 : KB * 0.50 + 1.6;
}

struct DensePlan { bool pair; int splits; bool rows; };

template <int ROWS>
static int launch_rows(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int out_dtype, cudaStream_t st) {
    const dim3 grid((unsigned)((p.N + rows::RN - 1) / rows::RN), (unsigned)((p.M + 127) / 128));
    auto go = [&](auto kern, int (*allow)(size_t)) {
        int rc = allow(rows::Shape<ROWS>::BYTES);
        if (rc) return rc;
        CINN_CHECK_CUDA(launch_dependent(kern, grid, dim3(rows::RTHREADS), rows::Shape<ROWS>::BYTES, st, ta, tb, p));
        CINN_CHECK_LAUNCH();
        return (int)CINN_OK;
    };
#define CINN_ROWS(O) case O: return go(rows::fp8_gemm_rows_kernel<ROWS, O>, allow_smem_once<rows::fp8_gemm_rows_kernel<ROWS, O>>)
    switch (out_dtype) {
        CINN_ROWS(CINN_BF16);
        CINN_ROWS(CINN_F32);
        CINN_ROWS(CINN_F16);
        CINN_ROWS(CINN_F32_BF16);
        default: set_error("GEMM: unknown output dtype tag %d", out_dtype); return CINN_ERR_INVALID;
    }
#undef CINN_ROWS
}

// The kernel for few rows: where its CTAs of 32 columns fit on the SMs twice and the reduction is short; without a workspace, that is
// where the alternative is a handful of long tiles, also where it is long.  us with cold operands, launch included, other kernels ->
// this one (rows x columns x reduction): 128 x 1024 x 512 12.3 -> 8.2, 512 x 1024 x 512 13.1 -> 8.2, 128 x 512 x 2048 17.2 -> 10.2, 256 x 2560 x
// 1024 15.2 -> 11.0, 512 of them 14.5 -> 13.1, 64 x 7168 x 2048 18.4 -> 12.3, 64 x 4096 x 7168 whole 36 -> 20.5; on the other side of
// the line 256 x 7168 x 2048 18.4 -> 20.4, 64 x 18432 x 7168 43.8 and 43.0, 64 x 4096 x 7168 cut 23.6, 64 x 576 x 7168 cut 19.5
// and 19.3, 64 x 7168 x 18432 cut 46.1 and 47.1.
static bool rows_pay(int64_t M, int64_t N, int64_t K, int b_layout, int64_t workspace_bytes, int sms) {
    if (b_layout != 0 || pair_mode() != 1 || sms < sm_count()) return false;
    const int64_t KB = (K + BK - 1) / BK, blocks = (N + rows::RN - 1) / rows::RN * ((M + 127) / 128);
    if (blocks > 2 * sms) return false;
    if (M <= 128 && workspace_bytes == 0) return true;
    return KB <= 40 && (M <= 128 || blocks * KB <= 16 * sms);
}

// Whole, by waves of tiles (tile_cost).  2155 x 320 -> 4352 takes 10.6 us on single SMs (two waves) and 12.3 on pairs (three), 4498 x 128 -> 8128
// 19.1 and 23.2 (one K block), 10646 x 512 -> 1472 18.8 and 16.0.
// Cut along K, with cold operands and the launch: a K block of a tile costs about 0.45 us in either kernel, a tile about 3 us
// around its K blocks on one SM and 1.6 on a pair.  Splitting adds a pass over the partial sums: about 3 us of launch and the bytes at the
// rate L2 returns them.  The plan with the smallest sum of these wins.  Whole -> as planned (M x N x K): 300 x 576 x 7168 29.7 -> 15.4 (B
// MN-major), 512 x 1024 x 32768 117 -> 31 on single SMs and 29 on pairs, 16 x 18432 x 7168 38.9 -> 34.3.  The demands (12 us, a gain of a
// tenth) leave the problems whole where the second launch eats what is won: 1024 x 4096 x 4096 (22 us).
static DensePlan dense_plan(int64_t M, int64_t N, int64_t K, int b_layout, int64_t workspace_bytes, int sms) {
    const int64_t KB = (K + BK - 1) / BK;
    auto waves = [](int64_t tiles, int64_t slots) { return (double)((tiles + slots - 1) / slots); };
    const int64_t pair_tiles = ((M + pair::PM - 1) / pair::PM) * ((N + pair::PN - 1) / pair::PN);
    const int64_t tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
    const double block_us = 0.45, tile_us = 3.0, pair_tile_us = 1.6;
    const int pm = pair_mode();
    // the pair kernel wins with B K-major, the one-SM kernel with B MN-major
    if (rows_pay(M, N, K, b_layout, workspace_bytes, sms)) return {false, 1, true};
    DensePlan best{false, 1, false};
    double best_us = waves(tiles, sms) * (KB * block_us + tile_us);
    // (128 rows would leave a CTA idle; a pair takes two SMs)
    const bool pairs = sms >= 2 && pm == 1 && b_layout == 0 && M > BM;
    if (pairs || (sms >= 2 && pm == 2 && pair_tiles >= sm_count() / 2)) {
        if (pm == 2 || waves(pair_tiles, sms / 2) * tile_cost(K, true) <= waves(tiles, sms) * tile_cost(K, false)) {
            best = {true, 1, false};
            best_us = waves(pair_tiles, sms / 2) * (KB * block_us + pair_tile_us);
        }
    }
    if (best_us < 12.0 || tiles >= sms) return best;
    for (int s = 2; s <= 32 && s * 2 <= KB; ++s) {
        const int64_t bytes = s * M * N * 4;
        if (bytes > workspace_bytes) break;
        const double blocks_us = (double)((KB + s - 1) / s) * block_us, sum_us = 3.0 + bytes / 4e6;
        const double us = waves(tiles * s, sms) * (blocks_us + tile_us) + sum_us;
        if (us < 0.9 * best_us) { best = {false, s, false}; best_us = us; }
        // (partial sums leave through TMA in rows of 16-byte multiples)
        const double pair_us = waves(pair_tiles * s, sms / 2) * (blocks_us + pair_tile_us) + sum_us;
        if (pairs && N % 4 == 0 && s * M < (1LL << 31) && pair_us < 0.9 * best_us) { best = {true, s, false}; best_us = pair_us; }
    }
    return best;
}

constexpr int64_t MAX_SPLIT_BYTES = 64LL << 20;

int64_t fp8_gemm_workspace_bytes(int64_t M, int64_t N, int64_t K, int b_layout) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const DensePlan plan = dense_plan(M, N, K, b_layout, MAX_SPLIT_BYTES, gemm_sms());
    return plan.splits > 1 ? plan.splits * M * N * 4 : 0;
}

// lda, ldb: bytes from one stored row of A and B to the next (a column range of a wider matrix is read in place)
int fp8_gemm(const void* A, int64_t lda, const float* sA, int64_t ld_sa, const void* B, int64_t ldb, const float* sB, int64_t sbk,
             int64_t sbn, void* C, int64_t M, int64_t N, int64_t K, int b_layout, int out_dtype, cudaStream_t st, void* workspace,
             int64_t workspace_bytes) {
    CINN_CHECK_ARG(M >= 0 && N >= 0 && K >= 0, "fp8_gemm: negative shape");
    if (M == 0 || N == 0) return CINN_OK;
    CINN_CHECK_ARG(A && sA && B && sB && C, "fp8_gemm: null pointer");
    CINN_CHECK_ARG(K > 0, "fp8_gemm: K must be positive");
    CINN_CHECK_ARG(M < (1LL << 31) && N < (1LL << 31) && K < (1LL << 31), "fp8_gemm: dimension too large");
    CINN_CHECK_ARG(K % 16 == 0, "fp8_gemm: K (%lld) must be a multiple of 16", (long long)K);
    CINN_CHECK_ARG(al16(A) && al16(B) && al16(C) && al16(workspace), "fp8_gemm: A, B, C and the workspace must be 16-byte aligned");
    CINN_CHECK_ARG(b_layout == 0 || b_layout == 1, "fp8_gemm: unknown B layout %d", b_layout);
    CINN_CHECK_ARG(b_layout == 0 || N % 16 == 0, "fp8_gemm: B stored (K, N) needs N %% 16 == 0");
    CINN_CHECK_ARG(lda >= K && ldb >= (b_layout == 0 ? K : N) && lda % 16 == 0 && ldb % 16 == 0,
                   "fp8_gemm: row pitches (%lld, %lld) must be multiples of 16 and no shorter than a row", (long long)lda, (long long)ldb);
    const int sms = gemm_sms();
    const DensePlan plan = dense_plan(M, N, K, b_layout, workspace ? workspace_bytes : 0, sms);
    CUtensorMap ta, tb;
    // (rows past the end are not free: a box of 64 with one row inside took the kernel 17.7 us at 1 x 4096 -> 7168, one of 8 takes it 12.0)
    const int box_rows = plan.rows && M <= 128 ? (int)((M + 7) / 8 * 8) : BM;
    int rc = make_map(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BK, box_rows);
    if (rc) return rc;
    if (b_layout == 0) rc = make_map(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, BK, plan.rows ? rows::RN : plan.pair ? 128 : BN);
    else rc = make_map(&tb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 128, BK);
    if (rc) return rc;
    GemmParams p{};
    p.sA = sA; p.sa_stride_m = ld_sa; p.sa_stride_k = 1;
    p.sB = sB; p.sb_stride_k = sbk; p.sb_stride_n = sbn; p.sb_stride_e = 0;
    p.C = C; p.ldc = N; p.M = (int)M; p.N = (int)N; p.K = (int)K;
    p.starts = nullptr; p.ends = nullptr; p.E = 1; p.b_rows_per_expert = 0; p.splits = 1;
    p.box_rows = box_rows;
    if (plan.rows) return M <= 64 ? launch_rows<64>(ta, tb, p, out_dtype, st) : launch_rows<128>(ta, tb, p, out_dtype, st);
    if (plan.pair) {
        const int64_t pair_tiles = ((M + pair::PM - 1) / pair::PM) * ((N + pair::PN - 1) / pair::PN) * plan.splits;
        const int clusters = (int)(pair_tiles < sms / 2 ? pair_tiles : sms / 2);
        if (plan.splits > 1) {
            p.C = workspace; p.E = plan.splits;
            CUtensorMap tc;
            rc = make_out_map(&tc, ta, p, CINN_F32, plan.splits * M, STORE_ROWS, true);
            if (rc) return rc;
            rc = launch_pair<false, CINN_F32, true>(ta, tb, tc, p, clusters, st);
            if (rc) return rc;
            return launch_split_sum(static_cast<const float*>(workspace), C, M * N, plan.splits, out_dtype, st);
        }
        return b_layout == 0 ? launch_pair_out<false>(ta, tb, p, out_dtype, clusters, st)
                             : launch_pair_out<true>(ta, tb, p, out_dtype, clusters, st);
    }
    const int64_t tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN) * plan.splits;
    const int grid = (int)(tiles < sms ? tiles : sms);
    if (plan.splits > 1) {
        p.C = workspace; p.splits = plan.splits;
        rc = b_layout == 0 ? launch<false, false, CINN_F32, false, true>(ta, tb, ta, p, grid, st)
                           : launch<true, false, CINN_F32, false, true>(ta, tb, ta, p, grid, st);
        if (rc) return rc;
        return launch_split_sum(static_cast<const float*>(workspace), C, M * N, plan.splits, out_dtype, st);
    }
    return b_layout == 0 ? launch_out<false, false>(ta, tb, p, out_dtype, grid, st)
                         : launch_out<true, false>(ta, tb, p, out_dtype, grid, st);
}

// Grouped problems run on pairs of SMs and 256-row tiles from 256 rows per expert on average (how the rows are really spread only
// the device knows): below that the half-empty tiles cost more than the pair saves.  Both directions; for the input gradient, whose
// weight is read MN-major, 7168 x 4096 of 32 experts, 32768 rows, 1045 -> 920 us, and 512 x 512
// of 16 experts, 65536 rows, 67 -> 59.  Not where the pairs' last wave is nearly empty and the single SMs' is not, with half a tile
// too many per expert: 8 experts, 3045 rows, 3328 -> 2560 53 us on pairs (three waves) and 43 (two), 32 of 9123, 1024 -> 768 25.6 and 21.5.
static bool grouped_on_pairs(int64_t E, int64_t T, int64_t N, int64_t K, int sms) {
    if (pair_mode() == 0 || sms < 2 || T < pair::PM * E) return false;
    const int64_t n_tiles = (N + pair::PN - 1) / pair::PN;
    if ((T + pair::PM - 1) / pair::PM * n_tiles < sms / 2) return false;
    auto waves = [&](int64_t rows, int slots) { return std::ceil((double)(2 * T + rows * E) / (double)(2 * rows) * (double)n_tiles / slots); };
    return waves(pair::PM, sms / 2) * tile_cost(K, true) <= 1.25 * waves(BM, sms) * tile_cost(K, false);
}

template <bool B_MN>
static int launch_grouped_pair(const CUtensorMap& ta, const CUtensorMap& tb, GemmParams& p, int out_dtype, int clusters, cudaStream_t st) {
    CUtensorMap tc;
    int rc = make_out_map(&tc, ta, p, out_dtype, p.M, STORE_ROWS, true);
    if (rc) return rc;
    switch (out_dtype) {
        case CINN_BF16: return launch_pair<B_MN, CINN_BF16, false, true>(ta, tb, tc, p, clusters, st);
        case CINN_F16: return launch_pair<B_MN, CINN_F16, false, true>(ta, tb, tc, p, clusters, st);
        case CINN_F32: return launch_pair<B_MN, CINN_F32, false, true>(ta, tb, tc, p, clusters, st);
        case CINN_F32_BF16: return launch_pair<B_MN, CINN_F32_BF16, false, true>(ta, tb, tc, p, clusters, st);
        default: set_error("GEMM: unknown output dtype tag %d", out_dtype); return CINN_ERR_INVALID;
    }
}

int fp8_grouped_gemm(const void* A, const float* sA, const void* W, const float* sW, const int64_t* starts,
                     const int64_t* ends, int64_t E, int64_t T, int64_t d_in, int64_t d_out, void* C, int out_dtype,
                     cudaStream_t st, const long long* row_dst) {
    CINN_CHECK_ARG(E >= 0 && T >= 0 && d_in >= 0 && d_out >= 0, "grouped_gemm: negative shape");
    if (E == 0 || T == 0 || d_out == 0) return CINN_OK;
    CINN_CHECK_ARG(A && sA && W && sW && starts && ends && (C || row_dst), "grouped_gemm: null pointer");
    CINN_CHECK_ARG(row_dst == nullptr || (d_out % 8 == 0 && (out_dtype == CINN_BF16 || out_dtype == CINN_F16)),
                   "grouped_gemm: scattered output rows need a 2-byte output type and d_out %% 8 == 0");
    CINN_CHECK_ARG(E <= MAX_EXPERTS, "grouped_gemm: at most %d experts are supported (got %lld)", MAX_EXPERTS, (long long)E);
    CINN_CHECK_ARG(d_in > 0 && d_in % 16 == 0, "grouped_gemm: d_in (%lld) must be a positive multiple of 16", (long long)d_in);
    CINN_CHECK_ARG(T < (1LL << 31) && d_out < (1LL << 31) && d_in < (1LL << 31) && E * d_out < (1LL << 31),
                   "grouped_gemm: dimension too large");
    CINN_CHECK_ARG(al16(A) && al16(W) && al16(C), "grouped_gemm: A, W and C must be 16-byte aligned");
    CUtensorMap ta, tb;
    int rc = make_map(&ta, A, (uint64_t)d_in, (uint64_t)T, (uint64_t)d_in, BK, BM);
    if (rc) return rc;
    const int sms = gemm_sms();
    const bool use_pair = row_dst == nullptr && grouped_on_pairs(E, T, d_out, d_in, sms);
    rc = make_map(&tb, W, (uint64_t)d_in, (uint64_t)(E * d_out), (uint64_t)d_in, BK, use_pair ? 128 : BN);
    if (rc) return rc;
    const int64_t nkb = (d_in + 127) / 128, nnb = (d_out + 127) / 128;
    GemmParams p{};
    p.sA = sA; p.sa_stride_m = nkb; p.sa_stride_k = 1;
    p.sB = sW; p.sb_stride_k = 1; p.sb_stride_n = nkb; p.sb_stride_e = nnb * nkb;
    p.C = C; p.ldc = d_out; p.M = (int)T; p.N = (int)d_out; p.K = (int)d_in;
    p.starts = starts; p.ends = ends; p.E = (int)E; p.b_rows_per_expert = (int)d_out;
    if (row_dst != nullptr) {
        // scattered rows: the table travels in the C slot of the parameters, tiles leave through staged 16-byte stores
        p.C = const_cast<long long*>(row_dst);
        p.tma_out = 0;
        return out_dtype == CINN_BF16 ? launch<false, true, CINN_BF16, true>(ta, tb, ta, p, sms, st)
                                      : launch<false, true, CINN_F16, true>(ta, tb, ta, p, sms, st);
    }
    if (use_pair) return launch_grouped_pair<false>(ta, tb, p, out_dtype, sms / 2, st);
    return launch_out<false, true>(ta, tb, p, out_dtype, sms, st);
}

// Input gradient of the grouped GEMM: dX[starts[e]:ends[e], :] = dY[starts[e]:ends[e], :] @ W[e]
// (W[e] is (d_out, d_in); its bytes are read MN-major, exactly as the dense dgrad reads a weight).
int fp8_grouped_gemm_dgrad(const void* dY, const float* sdY, const void* W, const float* sW, const int64_t* starts,
                           const int64_t* ends, int64_t E, int64_t T, int64_t d_in, int64_t d_out, void* dX, int out_dtype,
                           cudaStream_t st) {
    CINN_CHECK_ARG(E >= 0 && T >= 0 && d_in >= 0 && d_out >= 0, "grouped_gemm_dgrad: negative shape");
    if (E == 0 || T == 0 || d_in == 0) return CINN_OK;
    CINN_CHECK_ARG(dY && sdY && W && sW && starts && ends && dX, "grouped_gemm_dgrad: null pointer");
    CINN_CHECK_ARG(E <= MAX_EXPERTS, "grouped_gemm_dgrad: at most %d experts are supported (got %lld)", MAX_EXPERTS, (long long)E);
    CINN_CHECK_ARG(d_out > 0 && d_out % 16 == 0 && d_in % 16 == 0,
                   "grouped_gemm_dgrad: d_out (%lld) and d_in (%lld) must be multiples of 16", (long long)d_out, (long long)d_in);
    CINN_CHECK_ARG(T < (1LL << 31) && d_out < (1LL << 31) && d_in < (1LL << 31) && E * d_out < (1LL << 31),
                   "grouped_gemm_dgrad: dimension too large");
    CINN_CHECK_ARG(al16(dY) && al16(W) && al16(dX), "grouped_gemm_dgrad: dY, W and dX must be 16-byte aligned");
    CUtensorMap ta, tb;
    int rc = make_map(&ta, dY, (uint64_t)d_out, (uint64_t)T, (uint64_t)d_out, BK, BM);
    if (rc) return rc;
    // W viewed as (E * d_out) reduction rows of d_in output bytes: boxes of 128 output columns x 128 reduction rows.
    // A K block that runs past an expert's d_out rows meets zero-filled columns of dY, so the neighbour's bytes it
    // reads contribute nothing (quantised weights hold no NaN codes).
    rc = make_map(&tb, W, (uint64_t)d_in, (uint64_t)(E * d_out), (uint64_t)d_in, 128, BK);
    if (rc) return rc;
    const int64_t nkb_in = (d_in + 127) / 128, nob = (d_out + 127) / 128;
    GemmParams p{};
    p.sA = sdY; p.sa_stride_m = nob; p.sa_stride_k = 1;
    p.sB = sW; p.sb_stride_k = nkb_in; p.sb_stride_n = 1; p.sb_stride_e = nob * nkb_in;
    p.C = dX; p.ldc = d_in; p.M = (int)T; p.N = (int)d_in; p.K = (int)d_out;
    p.starts = starts; p.ends = ends; p.E = (int)E; p.b_rows_per_expert = (int)d_out;
    const int sms = gemm_sms();
    if (grouped_on_pairs(E, T, d_in, d_out, sms)) return launch_grouped_pair<true>(ta, tb, p, out_dtype, sms / 2, st);
    return launch_out<true, true>(ta, tb, p, out_dtype, sms, st);
}

// Weight gradients of all experts in one launch (the GK instantiation of the pair kernel): dW (E, d_out, d_in) with
// A = dY^T quantised per expert segment, (d_out, max_tiles * 128), and B = x block-quantised per segment and
// transposed, (d_in, max_tiles * 128); kb_start (E + 1 ints, device) gives every expert's K blocks.
int fp8_gemm_grouped_k(const void* A, const float* sA, const void* B, const float* sB, const int* kb_start, int64_t E,
                       int64_t M, int64_t N, int64_t max_tiles, void* C, int out_dtype, cudaStream_t st) {
    CINN_CHECK_ARG(E >= 1 && E <= MAX_SEGMENTS && M > 0 && N > 0 && max_tiles >= 1, "grouped-K GEMM: bad shape");
    CINN_CHECK_ARG(M % pair::PM == 0 && N % pair::PN == 0, "grouped-K GEMM: M (%lld) and N (%lld) must be multiples of 256",
                   (long long)M, (long long)N);
    CINN_CHECK_ARG(A && sA && B && sB && kb_start && C && al16(A) && al16(B) && al16(C), "grouped-K GEMM: null or unaligned pointer");
    CINN_CHECK_ARG(E * M < (1LL << 31) && N < (1LL << 31) && max_tiles * 128 < (1LL << 31), "grouped-K GEMM: dimension too large");
    const int64_t Kp = max_tiles * 128;
    CUtensorMap ta, tb;
    int rc = make_map(&ta, A, (uint64_t)Kp, (uint64_t)M, (uint64_t)Kp, BK, BM);
    if (rc) return rc;
    rc = make_map(&tb, B, (uint64_t)Kp, (uint64_t)N, (uint64_t)Kp, BK, 128);
    if (rc) return rc;
    const int64_t nnb = (N + 127) / 128;
    GemmParams p{};
    p.sA = sA; p.sa_stride_m = max_tiles; p.sa_stride_k = 1;
    p.sB = sB; p.sb_stride_k = nnb; p.sb_stride_n = 1; p.sb_stride_e = 0;
    p.C = C; p.ldc = N; p.M = (int)M; p.N = (int)N; p.K = 0;
    p.starts = reinterpret_cast<const int64_t*>(kb_start); p.ends = nullptr; p.E = (int)E; p.b_rows_per_expert = 0;
    CUtensorMap tc;
    rc = make_out_map(&tc, ta, p, out_dtype, E * M, STORE_ROWS, true);
    if (rc) return rc;
    const int64_t tiles = E * (M / pair::PM) * (N / pair::PN);
    const int sms = gemm_sms(), pairs = sms >= 2 ? sms / 2 : 1;              // (only the two-SM kernel does this: a cap of one SM counts as two)
    const int clusters = (int)(tiles < pairs ? tiles : pairs);
    // Below two K blocks per expert on average, 4-byte gradients are bound by their stores and by how early a tile's scales are there.  In us with the
    // quantisers, through the scale warp and OWN: 32 experts of 64 rows, 2048 x 2048 in fp32 142 -> 131, of 192 156 -> 141, of 256 158 and 163,
    // of 512 207 and 225; 32 of 128 rows, 7168 x 4096 854 -> 777; in bf16, of 128 rows 93 and 101.
    const bool own = max_tiles - E < 2 * E;
    switch (out_dtype) {
        case CINN_BF16: return launch_pair<false, CINN_BF16, true>(ta, tb, tc, p, clusters, st);
        case CINN_F32: return own ? launch_pair<false, CINN_F32, true, false, true>(ta, tb, tc, p, clusters, st)
                                  : launch_pair<false, CINN_F32, true>(ta, tb, tc, p, clusters, st);
        case CINN_F32_BF16: return own ? launch_pair<false, CINN_F32_BF16, true, false, true>(ta, tb, tc, p, clusters, st)
                                       : launch_pair<false, CINN_F32_BF16, true>(ta, tb, tc, p, clusters, st);
        default: set_error("grouped-K GEMM: the gradient is fp32 (optionally holding bf16-rounded values) or bf16"); return CINN_ERR_INVALID;
    }
}

// Grouped GEMM on 16-bit operands: C[starts[e]:ends[e]] = A[starts[e]:ends[e]] @ W[e]^T with A (T, d_in) and
// W (E, d_out, d_in) both bf16 or both fp16, fp32 accumulation (the reference's grouped_gemm_kernel arithmetic).
template <bool BF16_IN, int OUT>
static int launch16(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GemmParams& p, int grid,
                    cudaStream_t st) {
    constexpr auto kern = g16::grouped_gemm16_kernel<BF16_IN, OUT>;
    const size_t smem = smem_bytes(p.E);
    int rc = allow_smem_once<kern>(smem_bytes(MAX_EXPERTS));
    if (rc) return rc;
    kern<<<grid, g16::GTHREADS, smem, st>>>(ta, tb, tc, p);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

int grouped_gemm_16bit(const void* A, const void* W, int in_dtype, const int64_t* starts, const int64_t* ends, int64_t E,
                       int64_t T, int64_t d_in, int64_t d_out, void* C, int out_dtype, cudaStream_t st) {
    CINN_CHECK_ARG(E >= 0 && T >= 0 && d_in >= 0 && d_out >= 0, "grouped_gemm_16bit: negative shape");
    if (E == 0 || T == 0 || d_out == 0) return CINN_OK;
    CINN_CHECK_ARG(A && W && starts && ends && C, "grouped_gemm_16bit: null pointer");
    CINN_CHECK_ARG(in_dtype == CINN_BF16 || in_dtype == CINN_F16, "grouped_gemm_16bit: operands must be bf16 or fp16 (tag %d)", in_dtype);
    CINN_CHECK_ARG(E <= MAX_EXPERTS, "grouped_gemm_16bit: at most %d experts are supported (got %lld)", MAX_EXPERTS, (long long)E);
    CINN_CHECK_ARG(d_in > 0 && d_in % 8 == 0, "grouped_gemm_16bit: d_in (%lld) must be a positive multiple of 8", (long long)d_in);
    CINN_CHECK_ARG(T < (1LL << 31) && d_out < (1LL << 31) && d_in < (1LL << 30) && E * d_out < (1LL << 31),
                   "grouped_gemm_16bit: dimension too large");
    CINN_CHECK_ARG(al16(A) && al16(W) && al16(C), "grouped_gemm_16bit: A, W and C must be 16-byte aligned");
    const CUtensorMapDataType dt = in_dtype == CINN_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUtensorMap ta, tb;
    int rc = make_map(&ta, A, (uint64_t)d_in, (uint64_t)T, (uint64_t)d_in * 2, BK / 2, BM, dt);
    if (rc) return rc;
    rc = make_map(&tb, W, (uint64_t)d_in, (uint64_t)(E * d_out), (uint64_t)d_in * 2, BK / 2, BN, dt);
    if (rc) return rc;
    GemmParams p{};
    p.sA = nullptr; p.sB = nullptr;
    p.C = C; p.ldc = d_out; p.M = (int)T; p.N = (int)d_out; p.K = (int)d_in;
    p.starts = starts; p.ends = ends; p.E = (int)E; p.b_rows_per_expert = (int)d_out;
    CUtensorMap tc;
    rc = make_out_map(&tc, ta, p, out_dtype, p.M, BM);
    if (rc) return rc;
    const int grid = gemm_sms();
#define CINN_G16(BF, O) return launch16<BF, O>(ta, tb, tc, p, grid, st)
    if (in_dtype == CINN_BF16) {
        switch (out_dtype) {
            case CINN_BF16: CINN_G16(true, CINN_BF16);
            case CINN_F16: CINN_G16(true, CINN_F16);
            case CINN_F32: CINN_G16(true, CINN_F32);
        }
    } else {
        switch (out_dtype) {
            case CINN_BF16: CINN_G16(false, CINN_BF16);
            case CINN_F16: CINN_G16(false, CINN_F16);
            case CINN_F32: CINN_G16(false, CINN_F32);
        }
    }
#undef CINN_G16
    set_error("grouped_gemm_16bit: unknown output dtype tag %d", out_dtype);
    return CINN_ERR_INVALID;
}

int read_quant_status(int* out, int reset);
int read_moe_status(int* out, int reset);
int read_indexer_status(int* out, int reset);
int read_attn_status(int* out, int reset);
int read_linear_few_status(int* out, int reset);

// One word for the caller: the GEMM's code if it has one, else the quantisers', the exchange kernels', the indexer's,
// the attention's, the few-row linear's.
int read_device_status(int* out, int reset) {
    int v = 0, q = 0, m = 0, x = 0, a = 0, f = 0;
    CINN_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_device_status, sizeof(int)));
    if (reset && v != 0) {
        int z = 0;
        CINN_CHECK_CUDA(cudaMemcpyToSymbol(g_device_status, &z, sizeof(int)));
    }
    int rc = read_quant_status(&q, reset);
    if (rc) return rc;
    rc = read_moe_status(&m, reset);
    if (rc) return rc;
    rc = read_indexer_status(&x, reset);
    if (rc) return rc;
    rc = read_attn_status(&a, reset);
    if (rc) return rc;
    rc = read_linear_few_status(&f, reset);
    if (rc) return rc;
    *out = v != 0 ? v : (q != 0 ? q : (m != 0 ? m : (x != 0 ? x : (a != 0 ? a : f))));
    return CINN_OK;
}

}  // namespace cinn

