// Lightning indexer logits: I[b, t, s] = sum_h relu(q[b, t, h, :] . k[b, s, :]) * w[b, t, h], fp16 result.
//
// Semantics of cinnamon's lightning_indexer_kernel / lightning_indexer_fused (src/kernels.py:321-433): the
// operands of the dot product are rounded to fp16 (:374), products are accumulated in fp32, ReLU and the head
// weights are applied in fp32 (:377), the logits are stored as fp16 (:381).
//
// Tensor-core kernels (rows up to 128 wide, the widths indexers have): 128 queries x 128 keys at a time, tcgen05.mma (kind::f16, 128 x 128
// x d per head) into 128-column tensor-memory buffers, and warps that fold the dot products, relu * w, into fp32 registers.  Bound: two
// CUDA-core instructions per (query, key, head), the MMAs (64 cycles per 16 features of a tile) and the write of the logits.
//
// Persistent form (2-byte inputs that TMA can read, heads that fit in shared memory): one CTA per SM with a run of tiles, one query
// tile after the other.  A warp brings keys and heads by TMA, four warps turn bf16 into fp16 in place (the swizzled panels are what
// the MMA reads), one issues the MMAs into a ring of four tensor-memory buffers, sixteen fold and store.  A query tile's heads stay for
// all its key tiles.  The loads are what the other form waits for: a CTA's 80 KiB in four rounds of registers.
// The general form and this one, us a call: 8 x 1024, 4 heads of 64 in bf16 20.5 and 16.1; 8 x 2544 109 and 67; 16 x 1725 126 and 82; 32 x 1621, 2 of
// 128 194 and 112; 1 x 601, 2 of 128 18.5 and 6.8 (with the host's part, a native call now).  Issue slots 65 %, ALU 54 %, tensor pipe 25 % at 8 heads:
// a head of a tile takes its sixteen warps 760 cycles of 120 instructions each.
//
// General form (fp32, any strides, many heads): one CTA per tile.  All threads read the inputs (16 bytes at a time where the layout allows),
// round to fp16 and write the swizzled tiles; one warp issues the MMAs into one of two buffers while eight warps fold the previous
// head's (64 registers per thread).  Queries of up to 64 KiB of heads are resident at a time, so two CTAs share an SM and one loads
// while the other computes.  Its weights stay a load per head and its odd rows are stored element by element: brought into shared
// memory ahead the weights cost 183 us for 171 (8 x 2753, 4 heads of 64 in fp32), stores of words from the odd rows' first boundary 180 for 171.  One
// statement per panel of MMAs gives 167, an early start 168, both 164; 8 x 1024 24.4 -> 20.9.
//
// Scalar kernel (wider rows): 16 queries x 64 keys per CTA.  The key tile is kept transposed in shared memory as fp16
// ([d][key], so the 16 lanes that share a query read 16 consecutive keys), the queries of all heads as fp16
// ([query][head][d], broadcast reads).  A thread owns one query and four keys: per head a d-long dot product for each
// of the four, then relu * w into the running sum.
#include "tcgen05.cuh"
#include <type_traits>

namespace cinn {

namespace {
template <typename T> __device__ __forceinline__ __half to_half_rn(T v);
template <> __device__ __forceinline__ __half to_half_rn<float>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __half to_half_rn<__half>(__half v) { return v; }
template <> __device__ __forceinline__ __half to_half_rn<__nv_bfloat16>(__nv_bfloat16 v) { return __float2half_rn(__bfloat162float(v)); }
template <typename T> __device__ __forceinline__ float w_to_float(T v);
template <> __device__ __forceinline__ float w_to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float w_to_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float w_to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
}  // namespace

constexpr int IDX_TQ = 16, IDX_TK = 64;

template <typename T>
__global__ void __launch_bounds__(256)
indexer_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ w, __half* __restrict__ out,
               int Lq, int Lk, int H, int d, int64_t sqb, int64_t sqq, int64_t sqh, int64_t sqd, int64_t skb, int64_t skk,
               int64_t skd, int64_t swb, int64_t swq, int64_t swh) {
    extern __shared__ __align__(16) unsigned char idx_smem[];
    __half* sK = reinterpret_cast<__half*>(idx_smem);                 // [d][IDX_TK + 2]
    __half* sQ = sK + (size_t)d * (IDX_TK + 2);                       // [IDX_TQ][H][d]
    const int b = blockIdx.z, q0 = blockIdx.y * IDX_TQ, k0 = blockIdx.x * IDX_TK;
    const int tid = threadIdx.x;
    for (int e = tid; e < IDX_TK * d; e += 256) {
        const int kk = e / d, dd = e - kk * d;
        const int s = k0 + kk;
        sK[dd * (IDX_TK + 2) + kk] = s < Lk ? to_half_rn<T>(k[b * skb + s * skk + dd * skd]) : __float2half_rn(0.0f);
    }
    for (int e = tid; e < IDX_TQ * H * d; e += 256) {
        const int dd = e % d, h = (e / d) % H, qq = e / (d * H);
        const int t = q0 + qq;
        sQ[e] = t < Lq ? to_half_rn<T>(q[b * sqb + t * sqq + h * sqh + dd * sqd]) : __float2half_rn(0.0f);
    }
    __syncthreads();
    const int tq = tid >> 4, tk = tid & 15;
    const int t = q0 + tq;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int h = 0; h < H; ++h) {
        float dot[4] = {0.f, 0.f, 0.f, 0.f};
        const __half* qh = sQ + ((size_t)tq * H + h) * d;
        for (int dd = 0; dd < d; ++dd) {
            const float qv = __half2float(qh[dd]);
            const __half* kr = sK + dd * (IDX_TK + 2) + tk;
#pragma unroll
            for (int i = 0; i < 4; ++i) dot[i] = fmaf(qv, __half2float(kr[16 * i]), dot[i]);
        }
        const float wh = t < Lq ? w_to_float<T>(w[b * swb + t * swq + h * swh]) : 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = fmaf(fmaxf(dot[i], 0.0f), wh, acc[i]);
    }
    if (t < Lq) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int s = k0 + tk + 16 * i;
            if (s < Lk) out[((int64_t)b * Lq + t) * Lk + s] = __float2half_rn(acc[i]);
        }
    }
}

// ---------------------------------------------------------------------------
// tensor-core kernel
// ---------------------------------------------------------------------------
__device__ int g_indexer_status = 0;       // 0, or (role << 8) | reason of a bounded wait that ran out

constexpr int ITC_T = 128;                 // queries and keys per tile
constexpr int ITC_THREADS = 256;           // eight warps load, then fold; warp 0 issues the MMAs as well
constexpr int ITC_PANEL = ITC_T * 128;     // bytes of 128 rows x 64 fp16 columns: one swizzle panel
constexpr int ITC_MAX_D = 128;
constexpr int ITC_Q_BYTES = 64 * 1024;     // resident queries

struct IndexerArgs {
    int Lq, Lk, H, d, dpad, heads_per_chunk;
    int64_t sqb, sqq, sqh, sqd, skb, skk, skd, swb, swq, swh;
    bool vec_q, vec_k;                     // 16-byte loads allowed
};

// eight features as they are stored, and rounded to fp16
template <typename T> struct Raw8i { uint4 a; };
template <> struct Raw8i<float> { float4 a, b; };
__device__ __forceinline__ uint32_t half2_bits(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint4 to_half8(const Raw8i<float>& r) {
    return make_uint4(half2_bits(r.a.x, r.a.y), half2_bits(r.a.z, r.a.w), half2_bits(r.b.x, r.b.y), half2_bits(r.b.z, r.b.w));
}
__device__ __forceinline__ uint4 to_half8(const Raw8i<__half>& r) { return r.a; }
__device__ __forceinline__ uint4 to_half8(const Raw8i<__nv_bfloat16>& r) {
    auto two = [](uint32_t w) { return half2_bits(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); };
    return make_uint4(two(r.a.x), two(r.a.y), two(r.a.z), two(r.a.w));
}
template <typename T>
__device__ __forceinline__ Raw8i<T> load_raw8i(const T* p, bool live) {
    Raw8i<T> r;
    if constexpr (sizeof(T) == 4) {
        r.a = make_float4(0.f, 0.f, 0.f, 0.f); r.b = r.a;
        if (live) { r.a = __ldg(reinterpret_cast<const float4*>(p)); r.b = __ldg(reinterpret_cast<const float4*>(p) + 1); }
    } else {
        r.a = make_uint4(0u, 0u, 0u, 0u);
        if (live) r.a = __ldg(reinterpret_cast<const uint4*>(p));
    }
    return r;
}
// any strides, one element at a time; features beyond d and rows that do not exist are zero
template <typename T>
__device__ __forceinline__ uint4 gather8_half(const T* row, bool live, int d0, int d, int64_t sd) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half z = __float2half_rn(0.0f);
        const __half lo = live && d0 + 2 * i < d ? to_half_rn<T>(row[(d0 + 2 * i) * sd]) : z;
        const __half hi = live && d0 + 2 * i + 1 < d ? to_half_rn<T>(row[(d0 + 2 * i + 1) * sd]) : z;
        w[i] = (uint32_t)__half_as_ushort(lo) | ((uint32_t)__half_as_ushort(hi) << 16);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// byte offset of 16-byte chunk c (of dpad / 8) of row r in a tile of 128 rows stored as 64-column swizzle panels
__device__ __forceinline__ uint32_t panel_off(int r, int c) {
    return (uint32_t)((c >> 3) * ITC_PANEL + r * 128 + (((c & 7) ^ (r & 7)) << 4));
}

// one 128-row tile into its panels; `rows` of its rows exist.  With 16-byte loads four pieces of a thread are in flight.
template <typename T>
__device__ __forceinline__ void load_tile(uint8_t* dst, const T* src, int rows, int64_t ld, int64_t sd, int d, int dpad, bool vec) {
    const int sh = dpad == 64 ? 3 : 4;                              // 16-byte pieces per row: 8 or 16
    if (!vec) {
        for (int e = threadIdx.x; e < ITC_T << sh; e += ITC_THREADS) {
            const int r = e >> sh, c = e - (r << sh);
            *reinterpret_cast<uint4*>(dst + panel_off(r, c)) = gather8_half<T>(src + r * ld, r < rows, c * 8, d, sd);
        }
        return;
    }
    for (int e0 = threadIdx.x; e0 < ITC_T << sh; e0 += 4 * ITC_THREADS) {
        Raw8i<T> v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = e0 + u * ITC_THREADS, r = e >> sh, c = e - (r << sh);
            v[u] = load_raw8i<T>(src + r * ld + c * 8, r < rows && c * 8 < d);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = e0 + u * ITC_THREADS, r = e >> sh, c = e - (r << sh);
            *reinterpret_cast<uint4*>(dst + panel_off(r, c)) = to_half8(v[u]);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(ITC_THREADS, 2)
indexer_tc_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ w, __half* __restrict__ out,
                  const IndexerArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int head_bytes = (a.dpad / 64) * ITC_PANEL;
    uint8_t* sQ = smem;                                            // [head of the chunk][panel][row][128 B]
    uint8_t* sK = smem + (size_t)a.heads_per_chunk * head_bytes;   // [panel][row][128 B]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sK + head_bytes); // two "dot products ready", two "buffer free"
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.z, q0 = blockIdx.y * ITC_T, k0 = blockIdx.x * ITC_T;
    const uint32_t full0 = smem_u32(bars), free0 = smem_u32(bars + 2);
    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < 2; ++i) { mbar_init(full0 + 8 * i, 1); mbar_init(free0 + 8 * i, 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc_alloc(smem_u32(tmem_slot), 2 * ITC_T);
    pdl_wait();
    if (warp == 0) pdl_trigger();
    const T* kb = k + b * a.skb;
    const T* qb = q + b * a.sqb;
    load_tile<T>(sK, kb + k0 * a.skk, a.Lk - k0, a.skk, a.skd, a.d, a.dpad, a.vec_k);
    const int quarter = warp & 3, group = warp >> 2;                // TMEM lane quarter, column group of 64 keys
    const int t = q0 + quarter * 32 + lane;
    float acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.0f;
    uint32_t it0 = 0;                                               // heads of earlier chunks; head n uses buffer n & 1
    bool alive = true;
    uint32_t tmem = 0;
    for (int h0 = 0; h0 < a.H; h0 += a.heads_per_chunk) {
        const int nh = min(a.heads_per_chunk, a.H - h0);
        for (int h = 0; h < nh; ++h)
            load_tile<T>(sQ + h * head_bytes, qb + q0 * a.sqq + (h0 + h) * a.sqh, a.Lq - q0, a.sqq, a.sqd, a.d, a.dpad, a.vec_q);
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        tmem = *tmem_slot;
        // head h of the chunk: issued by warp 0 once the buffer's previous dot products have been read
        auto issue = [&](int h) {
            const uint32_t n = it0 + h, buf = n & 1;
            const bool ok = mbar_wait_bounded(free0 + 8 * buf, ((n >> 1) & 1) ^ 1, abort_flag, (7 << 8) | 1, &g_indexer_status);
            if (!__all_sync(0xffffffffu, ok)) return;
            tc_fence_after();
            for (int c = 0; c < a.dpad / 64; ++c)
                mma_panels(tmem + buf * ITC_T, panel_desc(smem_u32(sQ) + h * head_bytes + c * ITC_PANEL), panel_desc(smem_u32(sK) + c * ITC_PANEL),
                           make_idesc_f16(false, ITC_T, ITC_T), c == 0);
            tc_commit(full0 + 8 * buf);
        };
        if (warp == 0) {
            issue(0);
            if (nh > 1) issue(1);
        }
        for (int h = 0; h < nh && alive; ++h) {
            const uint32_t n = it0 + h, buf = n & 1;
            const float wh = t < a.Lq ? w_to_float<T>(w[b * a.swb + t * a.swq + (h0 + h) * a.swh]) : 0.0f;
            const bool ok = mbar_wait_bounded(full0 + 8 * buf, (n >> 1) & 1, abort_flag, (7 << 8) | 2, &g_indexer_status);
            if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
            tc_fence_after();
            const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + buf * ITC_T + group * 64;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float v[16];
                tc_ld16(taddr + c * 16, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[c * 16 + i] = fmaf(fmaxf(v[i], 0.0f), wh, acc[c * 16 + i]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(free0 + 8 * buf);
            __syncwarp();
            if (warp == 0 && h + 2 < nh) issue(h + 2);
        }
        it0 += nh;
        __syncthreads();              // every MMA of these heads has been read, hence has finished: the queries may go
    }
    if (alive) {
        // through this warp's 4 KiB of the (now unused) operand tiles, so that rows leave as contiguous pieces
        uint8_t* stage = smem + warp * 4096;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            *reinterpret_cast<uint4*>(stage + lane * 128 + ((c ^ (lane & 7)) << 4)) =
                make_uint4(half2_bits(acc[c * 8], acc[c * 8 + 1]), half2_bits(acc[c * 8 + 2], acc[c * 8 + 3]),
                           half2_bits(acc[c * 8 + 4], acc[c * 8 + 5]), half2_bits(acc[c * 8 + 6], acc[c * 8 + 7]));
        }
        __syncwarp();
        const int s0 = k0 + group * 64, t0 = q0 + quarter * 32;
        __half* ob = out + ((int64_t)b * a.Lq + t0) * a.Lk + s0;
        if ((a.Lk & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = i * 4 + (lane >> 3), c = lane & 7;
                if (t0 + r < a.Lq && s0 + c * 8 < a.Lk)
                    *reinterpret_cast<uint4*>(ob + (int64_t)r * a.Lk + c * 8) =
                        *reinterpret_cast<const uint4*>(stage + r * 128 + ((c ^ (r & 7)) << 4));
            }
        } else {
            for (int r = 0; r < 32 && t0 + r < a.Lq; ++r) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int s = lane + 32 * i;
                    if (s0 + s < a.Lk)
                        ob[(int64_t)r * a.Lk + s] = *reinterpret_cast<const __half*>(stage + r * 128 + (((s >> 3) ^ (r & 7)) << 4) + (s & 7) * 2);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tc_dealloc(*tmem_slot, 2 * ITC_T);
    }
}

// 32 lanes x 32 consecutive fp32 columns, waited for
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
        "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---------------------------------------------------------------------------
// persistent form
// ---------------------------------------------------------------------------
constexpr int IRUN_FOLD_WARPS = 16, IRUN_CONVERT_WARPS = 4;
constexpr int IRUN_MMA = IRUN_FOLD_WARPS, IRUN_TMA = IRUN_MMA + 1;
constexpr int IRUN_THREADS = (IRUN_FOLD_WARPS + 2 + IRUN_CONVERT_WARPS) * 32;
constexpr int IRUN_COLS = ITC_T / (IRUN_FOLD_WARPS / 4);          // keys of a fold warp
constexpr int IRUN_BUFS = 4;                                       // tensor-memory buffers of ITC_T columns
constexpr int IRUN_STAGE_BYTES = ITC_T * ITC_T * 2;               // a tile's logits
constexpr int IRUN_MAX_SLOTS = 12;                                 // key tiles and query heads in shared memory
constexpr int IRUN_SLOT_BYTES = IRUN_MAX_SLOTS * ITC_PANEL;
constexpr int IRUN_BAR_BYTES = 512;
constexpr int IRUN_MAX_HEADS = IRUN_MAX_SLOTS - 3;                // of 64 columns; 4 of 128
constexpr int IRUN_SMEM_BYTES = IRUN_STAGE_BYTES + IRUN_SLOT_BYTES + IRUN_BAR_BYTES + IRUN_MAX_HEADS * ITC_T * 2;

struct IndexerRun {
    int Lq, Lk, H, panels, k_slots, q_slots, q_tiles, k_tiles, tiles;
    int64_t swb, swq, swh;
};

__device__ __forceinline__ void tma_load_4d(const CUtensorMap* map, uint32_t bar, uint32_t dst, int x, int y, int z, int w) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void tma_load_keys(const CUtensorMap* map, uint32_t bar, uint32_t dst, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}

// A place in one of the two rings; every role that follows a ring counts its own.
struct RingPlace {
    uint32_t slot = 0, lap = 0;
    __device__ __forceinline__ void next(int slots) { if (++slot == (uint32_t)slots) { slot = 0; ++lap; } }
};

template <typename T>
__global__ void __launch_bounds__(IRUN_THREADS, 1)
indexer_run_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const T* __restrict__ w,
                   __half* __restrict__ out, const IndexerRun a) {
    static_assert(sizeof(T) == 2, "2-byte inputs");
    constexpr bool CONVERT = std::is_same<T, __nv_bfloat16>::value;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tile_bytes = a.panels * ITC_PANEL;
    // layout: output staging | key tiles | query heads | barriers | head weights
    uint8_t* sK = smem + IRUN_STAGE_BYTES;
    uint8_t* sQ = sK + a.k_slots * tile_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + IRUN_STAGE_BYTES + IRUN_SLOT_BYTES);
    T* sW = reinterpret_cast<T*>(reinterpret_cast<uint8_t*>(bars) + IRUN_BAR_BYTES);        // [head][query]
    // "landed", "converted", "free" of every slot (keys first), "ready" and "free" of the tensor-memory buffers, "wrote" and "read" of the
    // quarters of the staging, "there" of their rows' weights
    const uint32_t landed0 = smem_u32(bars), converted0 = landed0 + 8 * IRUN_MAX_SLOTS, free0 = converted0 + 8 * IRUN_MAX_SLOTS;
    const uint32_t tfull0 = free0 + 8 * IRUN_MAX_SLOTS, tempty0 = tfull0 + 8 * IRUN_BUFS;
    const uint32_t wrote0 = tempty0 + 8 * IRUN_BUFS, read0 = wrote0 + 32, weights0 = read0 + 32;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * IRUN_MAX_SLOTS + 2 * IRUN_BUFS + 12);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < a.k_slots + a.q_slots; ++i) {
            mbar_init(landed0 + 8 * i, 1);
            mbar_init(converted0 + 8 * i, IRUN_CONVERT_WARPS);
            mbar_init(free0 + 8 * i, 1);
        }
        for (int i = 0; i < IRUN_BUFS; ++i) { mbar_init(tfull0 + 8 * i, 1); mbar_init(tempty0 + 8 * i, IRUN_FOLD_WARPS); }
        for (int i = 0; i < 12; ++i) mbar_init(wrote0 + 8 * i, IRUN_FOLD_WARPS / 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == IRUN_MMA) tc_alloc(smem_u32(tmem_slot), IRUN_BUFS * ITC_T);
    pdl_wait();
    if (warp == IRUN_MMA) pdl_trigger();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // tile t = (query tile over all batches, key tile)
    const int t_begin = (int)((int64_t)a.tiles * blockIdx.x / gridDim.x), t_end = (int)((int64_t)a.tiles * (blockIdx.x + 1) / gridDim.x);
    auto wait = [&](uint32_t bar, uint32_t parity, int code) {
        const bool ok = mbar_wait_bounded(bar, parity, abort_flag, (7 << 8) | code, &g_indexer_status);
        return (bool)__all_sync(0xffffffffu, ok);
    };
    const uint32_t q_first = 8 * a.k_slots;                        // of the queries' barriers behind the keys'
    if (warp == IRUN_TMA) {
        if (lane == 0) {
            RingPlace kp, qp;
            int have = -1;
            bool alive = true;
            auto room = [&](uint32_t bar, const RingPlace& r) {
                return mbar_wait_bounded(bar, (r.lap & 1) ^ 1, abort_flag, (7 << 8) | 1, &g_indexer_status);
            };
            for (int t = t_begin; t < t_end && alive; ++t) {
                const int qt = t / a.k_tiles, b = qt / a.q_tiles, q0 = (qt - b * a.q_tiles) * ITC_T, k0 = (t - qt * a.k_tiles) * ITC_T;
                const uint32_t at = 8 * kp.slot;
                if (!(alive = room(free0 + at, kp))) break;
                mbar_expect_tx(landed0 + at, tile_bytes);
                for (int p = 0; p < a.panels; ++p)
                    tma_load_keys(&tmK, landed0 + at, smem_u32(sK) + kp.slot * tile_bytes + p * ITC_PANEL, p * 64, k0, b);
                kp.next(a.k_slots);
                if (qt == have) continue;
                have = qt;
                for (int h = 0; h < a.H; ++h) {
                    const uint32_t qat = q_first + 8 * qp.slot;
                    if (!(alive = room(free0 + qat, qp))) break;
                    mbar_expect_tx(landed0 + qat, tile_bytes);
                    for (int p = 0; p < a.panels; ++p)
                        tma_load_4d(&tmQ, landed0 + qat, smem_u32(sQ) + qp.slot * tile_bytes + p * ITC_PANEL, p * 64, h, q0, b);
                    qp.next(a.q_slots);
                }
            }
            if (!alive) {                                          // abandoned: let the copies in flight land
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000LL) { }
            }
        }
    } else if (warp > IRUN_TMA) {
        if constexpr (CONVERT) {
            const int ctid = tid - (IRUN_TMA + 1) * 32;
            RingPlace kp, qp;
            int have = -1;
            auto convert = [&](uint32_t at, const RingPlace& r, uint8_t* tile) {
                if (!wait(landed0 + at, r.lap & 1, 2)) return false;
                for (int e0 = ctid; e0 < a.panels * (ITC_PANEL / 16); e0 += 8 * IRUN_CONVERT_WARPS * 32) {
                    Raw8i<T> v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[u].a = *reinterpret_cast<const uint4*>(tile + (e0 + u * IRUN_CONVERT_WARPS * 32) * 16);
#pragma unroll
                    for (int u = 0; u < 8; ++u) *reinterpret_cast<uint4*>(tile + (e0 + u * IRUN_CONVERT_WARPS * 32) * 16) = to_half8(v[u]);
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(converted0 + at);
                return true;
            };
            bool alive = true;
            for (int t = t_begin; t < t_end && alive; ++t) {
                const int qt = t / a.k_tiles;
                alive = convert(8 * kp.slot, kp, sK + kp.slot * tile_bytes);
                kp.next(a.k_slots);
                if (qt == have) continue;
                have = qt;
                for (int h = 0; h < a.H && alive; ++h) {
                    alive = convert(q_first + 8 * qp.slot, qp, sQ + qp.slot * tile_bytes);
                    qp.next(a.q_slots);
                }
            }
        }
    } else if (warp == IRUN_MMA) {
        const uint32_t ready0 = CONVERT ? converted0 : landed0, k_desc = panel_desc(smem_u32(sK)), q_desc = panel_desc(smem_u32(sQ));
        constexpr uint32_t idesc = make_idesc_f16(false, ITC_T, ITC_T);
        RingPlace kp, q0p;                                         // the key tile; the first head of the query tile
        uint32_t n = 0;
        bool fresh = true, alive = true;
        for (int t = t_begin; t < t_end && alive; ++t) {
            const bool last = t + 1 == t_end || (t + 1) / a.k_tiles != t / a.k_tiles;       // the queries' last use
            RingPlace qp = q0p;
            alive = wait(ready0 + 8 * kp.slot, kp.lap & 1, 3);
            for (int h = 0; h < a.H && alive; ++h, ++n) {
                const uint32_t buf = n % IRUN_BUFS, qat = q_first + 8 * qp.slot;
                if (fresh) alive = wait(ready0 + qat, qp.lap & 1, 4);
                alive = alive && wait(tempty0 + 8 * buf, ((n / IRUN_BUFS) & 1) ^ 1, 5);
                if (!alive) break;
                tc_fence_after();
                const uint32_t qd = q_desc + qp.slot * (uint32_t)(tile_bytes >> 4), kd = k_desc + kp.slot * (uint32_t)(tile_bytes >> 4);
                mma_panels(tmem + buf * ITC_T, qd, kd, idesc, true);
                if (a.panels > 1) mma_panels(tmem + buf * ITC_T, qd + (ITC_PANEL >> 4), kd + (ITC_PANEL >> 4), idesc, false);
                tc_commit(tfull0 + 8 * buf);
                if (last) tc_commit(free0 + qat);
                qp.next(a.q_slots);
            }
            if (!alive) break;
            tc_commit(free0 + 8 * kp.slot);
            kp.next(a.k_slots);
            fresh = last;
            if (last) q0p = qp;
        }
    } else {
        const int quarter = warp & 3, group = warp >> 2;            // TMEM lane quarter, columns
        uint8_t* stage = smem + quarter * (32 * 2 * ITC_T);        // this quarter's 32 rows of logits, 16-byte chunks XOR-ed with the row
        const uint32_t wrote = wrote0 + 8 * quarter, read = read0 + 8 * quarter, there = weights0 + 8 * quarter;
        const T* my_w = sW + quarter * 32 + lane;
        int have = -1;
        uint32_t loaded = 0;
        const bool aligned = (a.Lk & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
        uint32_t n = 0, round = 0;
        bool alive = true;
        for (int t = t_begin; t < t_end && alive; ++t, ++round) {
            const int qt = t / a.k_tiles, b = qt / a.q_tiles, q0 = (qt - b * a.q_tiles) * ITC_T, k0 = (t - qt * a.k_tiles) * ITC_T;
            const int row = q0 + quarter * 32 + lane;
            if (qt != have) {
                // the rows' weights, once per query tile (a load per head was a round trip per head: 950 cycles where the arithmetic takes
                // 400); nobody reads the last ones any more once the tile before has been stored
                have = qt;
                if (round > 0 && !(alive = wait(read, (round - 1) & 1, 7))) break;
                for (int h = group; h < a.H; h += IRUN_FOLD_WARPS / 4)
                    sW[h * ITC_T + quarter * 32 + lane] = row < a.Lq ? w[b * a.swb + row * a.swq + h * a.swh] : T(0.0f);
                __syncwarp();
                if (lane == 0) mbar_arrive(there);
                if (!(alive = wait(there, loaded++ & 1, 9))) break;
            }
            uint64_t acc[IRUN_COLS / 2];
#pragma unroll
            for (int i = 0; i < IRUN_COLS / 2; ++i) acc[i] = 0u;
            for (int h = 0; h < a.H; ++h, ++n) {
                const uint32_t buf = n % IRUN_BUFS;
                uint64_t w2;
                asm("mov.b64 %0, {%1, %1};" : "=l"(w2) : "f"(w_to_float<T>(my_w[h * ITC_T])));
                alive = wait(tfull0 + 8 * buf, (n / IRUN_BUFS) & 1, 6);
                if (!alive) break;
                tc_fence_after();
                uint32_t v[IRUN_COLS];
                tc_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + buf * ITC_T + group * IRUN_COLS, v);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty0 + 8 * buf);
#pragma unroll
                for (int i = 0; i < IRUN_COLS / 2; ++i) {
                    uint64_t x;
                    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(fmaxf(__uint_as_float(v[2 * i]), 0.0f)), "f"(fmaxf(__uint_as_float(v[2 * i + 1]), 0.0f)));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i]) : "l"(x), "l"(w2));
                }
            }
            if (!alive) break;
            // The quarter's rows through shared memory: four warps write 32 columns of 32 rows each and store 8 whole rows each, in 16-byte
            // pieces from a row's first 16-byte boundary on and single elements at its ends.  (Every warp its own 32 columns, in words: at
            // odd row lengths 6000 cycles of a tile, three stores of two rows where here is one of two rows and its ends.)
            if (round > 0 && !(alive = wait(read, (round - 1) & 1, 7))) break;
#pragma unroll
            for (int c = 0; c < IRUN_COLS / 8; ++c) {
                uint32_t h2[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float x, y;
                    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(acc[c * 4 + i]));
                    h2[i] = half2_bits(x, y);
                }
                *reinterpret_cast<uint4*>(stage + lane * 256 + (((group * (IRUN_COLS / 8) + c) ^ (lane & 7)) << 4)) = make_uint4(h2[0], h2[1], h2[2], h2[3]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(wrote);
            if (!(alive = wait(wrote, round & 1, 8))) break;
            const int cols = min(ITC_T, a.Lk - k0), rows = min(32, a.Lq - (q0 + quarter * 32)), j = lane & 15;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = group * 8 + 2 * i + (lane >> 4);
                const uint8_t* line = stage + r * 256;
                __half* orow = out + ((int64_t)b * a.Lq + q0 + quarter * 32 + r) * a.Lk + k0;
                uint4 lo = *reinterpret_cast<const uint4*>(line + ((j ^ (r & 7)) << 4));
                if (aligned) {
                    if (r < rows && j * 8 < cols) *reinterpret_cast<uint4*>(orow + j * 8) = lo;
                    continue;
                }
                const uint4 hi = *reinterpret_cast<const uint4*>(line + ((((j + 1) & 15) ^ (r & 7)) << 4));
                const int first = (int)(-(reinterpret_cast<uintptr_t>(orow) >> 1)) & 7;             // elements before the row's first boundary
                // elements [first, first + 8) of lo and hi
                uint32_t x[7] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z};
                if (first & 4) { x[0] = x[2]; x[1] = x[3]; x[2] = x[4]; x[3] = x[5]; x[4] = x[6]; x[5] = hi.w; }
                if (first & 2) { x[0] = x[1]; x[1] = x[2]; x[2] = x[3]; x[3] = x[4]; x[4] = x[5]; }
                const int bits = (first & 1) * 16;
                lo = make_uint4(__funnelshift_r(x[0], x[1], bits), __funnelshift_r(x[1], x[2], bits), __funnelshift_r(x[2], x[3], bits),
                                __funnelshift_r(x[3], x[4], bits));
                const int whole = max(cols - first, 0) >> 3;
                if (r < rows) {
                    if (j < whole) *reinterpret_cast<uint4*>(orow + first + j * 8) = lo;
                    // the ends: lanes 0 - 7 before the first boundary, 8 - 15 behind the last whole piece
                    const int e = j < 8 ? j : first + whole * 8 + j - 8;
                    if (j < 8 ? e < min(first, cols) : e < cols)
                        orow[e] = *reinterpret_cast<const __half*>(line + (((e >> 3) ^ (r & 7)) << 4) + (e & 7) * 2);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(read);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == IRUN_MMA) {
        tc_fence_after();
        tc_dealloc(tmem, IRUN_BUFS * ITC_T);
    }
}

// Whether the persistent form takes the call, and then its launch (0: taken, -1: not, otherwise an error).
template <typename T>
static int indexer_run(const T* q, const T* k, const T* w, __half* out, int B, int Lq, int Lk, int H, int d, const int64_t* sq,
                       const int64_t* sk, const int64_t* sw, cudaStream_t st) {
    IndexerRun a;
    a.panels = (d + 63) / 64;
    const int places = IRUN_SLOT_BYTES / (a.panels * ITC_PANEL);   // 12 of 64 columns, 6 of 128
    a.k_slots = a.panels == 1 ? 3 : 2;
    a.q_slots = places - a.k_slots;
    if (H > a.q_slots) return -1;
    // dimensions of one element have no stride to speak of
    auto bytes = [](int64_t extent, int64_t stride) { return extent == 1 ? (int64_t)16 : stride * (int64_t)sizeof(T); };
    auto fits = [](int64_t b) { return b > 0 && b % 16 == 0 && b < (1LL << 39); };
    const int64_t qs[3] = {bytes(H, sq[2]), bytes(Lq, sq[1]), bytes(B, sq[0])}, ks[2] = {bytes(Lk, sk[1]), bytes(B, sk[0])};
    if ((d > 1 && (sq[3] != 1 || sk[2] != 1)) || !fits(qs[0]) || !fits(qs[1]) || !fits(qs[2]) || !fits(ks[0]) || !fits(ks[1]) ||
        (reinterpret_cast<uintptr_t>(q) & 15) != 0 || (reinterpret_cast<uintptr_t>(k) & 15) != 0)
        return -1;
    a.Lq = Lq; a.Lk = Lk; a.H = H;
    a.q_tiles = (Lq + ITC_T - 1) / ITC_T;
    a.k_tiles = (Lk + ITC_T - 1) / ITC_T;
    const int64_t tiles = (int64_t)B * a.q_tiles * a.k_tiles;
    if (tiles >= (1LL << 31)) return -1;
    a.tiles = (int)tiles;
    a.swb = sw[0]; a.swq = sw[1]; a.swh = sw[2];
    const CUtensorMapDataType type = std::is_same<T, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUtensorMap tq, tk;
    const uint64_t qd[4] = {(uint64_t)d, (uint64_t)H, (uint64_t)Lq, (uint64_t)B}, kd[3] = {(uint64_t)d, (uint64_t)Lk, (uint64_t)B};
    const uint64_t qst[3] = {(uint64_t)qs[0], (uint64_t)qs[1], (uint64_t)qs[2]}, kst[2] = {(uint64_t)ks[0], (uint64_t)ks[1]};
    const uint32_t qbox[4] = {64, 1, ITC_T, 1}, kbox[3] = {64, ITC_T, 1};
    if (encode_map(&tq, q, 4, qd, qst, qbox, type, CU_TENSOR_MAP_SWIZZLE_128B) || encode_map(&tk, k, 3, kd, kst, kbox, type, CU_TENSOR_MAP_SWIZZLE_128B))
        return -1;                                                  // (strides that the driver does not take)
    if (const int failed = allow_smem_once<indexer_run_kernel<T>>(IRUN_SMEM_BYTES)) return failed;
    const int grid = a.tiles < sm_count() ? a.tiles : sm_count();
    CINN_CHECK_CUDA(launch_dependent(indexer_run_kernel<T>, dim3(grid), dim3(IRUN_THREADS), IRUN_SMEM_BYTES, st, tq, tk, w, out, a));
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

template <typename T>
static int indexer_tc_typed(const T* q, const T* k, const T* w, __half* out, int B, int Lq, int Lk, int H, int d, const int64_t* sq,
                            const int64_t* sk, const int64_t* sw, cudaStream_t st) {
    IndexerArgs a;
    a.Lq = Lq; a.Lk = Lk; a.H = H; a.d = d;
    a.dpad = (d + 63) / 64 * 64;
    const int head_bytes = a.dpad / 64 * ITC_PANEL;
    a.heads_per_chunk = H < ITC_Q_BYTES / head_bytes ? H : ITC_Q_BYTES / head_bytes;
    a.sqb = sq[0]; a.sqq = sq[1]; a.sqh = sq[2]; a.sqd = sq[3];
    a.skb = sk[0]; a.skk = sk[1]; a.skd = sk[2];
    a.swb = sw[0]; a.swq = sw[1]; a.swh = sw[2];
    auto on16 = [](int64_t stride) { return (stride * (int64_t)sizeof(T)) % 16 == 0; };
    a.vec_q = d % 8 == 0 && sq[3] == 1 && on16(sq[0]) && on16(sq[1]) && on16(sq[2]) && (reinterpret_cast<uintptr_t>(q) & 15) == 0;
    a.vec_k = d % 8 == 0 && sk[2] == 1 && on16(sk[0]) && on16(sk[1]) && (reinterpret_cast<uintptr_t>(k) & 15) == 0;
    const size_t smem = (size_t)(a.heads_per_chunk + 1) * head_bytes + 1024 + 64;
    dim3 grid((unsigned)((Lk + ITC_T - 1) / ITC_T), (unsigned)((Lq + ITC_T - 1) / ITC_T), (unsigned)B);
    CINN_CHECK_ARG(grid.y <= 65535 && grid.z <= 65535, "lightning_indexer: too many queries or batches");
    CINN_CHECK_CUDA(cudaFuncSetAttribute(indexer_tc_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
    launch_dependent(indexer_tc_kernel<T>, grid, dim3(ITC_THREADS), smem, st, q, k, w, out, a);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

int read_indexer_status(int* out, int reset) {
    int v = 0;
    CINN_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_indexer_status, sizeof(int)));
    if (reset && v != 0) {
        int z = 0;
        CINN_CHECK_CUDA(cudaMemcpyToSymbol(g_indexer_status, &z, sizeof(int)));
    }
    *out = v;
    return CINN_OK;
}

template <typename T>
static int indexer_typed(const T* q, const T* k, const T* w, __half* out, int B, int Lq, int Lk, int H, int d, const int64_t* sq,
                         const int64_t* sk, const int64_t* sw, cudaStream_t st) {
    if (d <= ITC_MAX_D) {
        CINN_CHECK_ARG((Lq + ITC_T - 1) / ITC_T <= 65535 && B <= 65535, "lightning_indexer: too many queries or batches");
        if constexpr (sizeof(T) == 2) {
            const int rc = indexer_run<T>(q, k, w, out, B, Lq, Lk, H, d, sq, sk, sw, st);
            if (rc >= 0) return rc;
        }
        return indexer_tc_typed<T>(q, k, w, out, B, Lq, Lk, H, d, sq, sk, sw, st);
    }
    const size_t smem = ((size_t)d * (IDX_TK + 2) + (size_t)IDX_TQ * H * d) * sizeof(__half);
    CINN_CHECK_ARG(smem <= 160 * 1024, "lightning_indexer: %d heads of width %d need %zu bytes of shared memory (limit 163840)",
                   H, d, smem);
    CINN_CHECK_CUDA(cudaFuncSetAttribute(indexer_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
    dim3 grid((unsigned)((Lk + IDX_TK - 1) / IDX_TK), (unsigned)((Lq + IDX_TQ - 1) / IDX_TQ), (unsigned)B);
    CINN_CHECK_ARG(grid.y <= 65535 && grid.z <= 65535, "lightning_indexer: too many queries or batches");
    indexer_kernel<T><<<grid, 256, smem, st>>>(q, k, w, out, Lq, Lk, H, d, sq[0], sq[1], sq[2], sq[3], sk[0], sk[1], sk[2], sw[0],
                                               sw[1], sw[2]);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

int lightning_indexer(const void* q, const void* k, const void* w, int dtype, void* out, int64_t B, int64_t Lq, int64_t Lk,
                      int64_t H, int64_t d, const int64_t* q_strides, const int64_t* k_strides, const int64_t* w_strides,
                      cudaStream_t st) {
    CINN_CHECK_ARG(B >= 0 && Lq >= 0 && Lk >= 0 && H >= 1 && d >= 1, "lightning_indexer: bad shape");
    if (B == 0 || Lq == 0 || Lk == 0) return CINN_OK;
    CINN_CHECK_ARG(q && k && w && out && q_strides && k_strides && w_strides, "lightning_indexer: null pointer");
    CINN_CHECK_ARG(Lq < (1LL << 31) && Lk < (1LL << 31) && H < 4096 && d < 65536, "lightning_indexer: dimension too large");
    switch (dtype) {
        case CINN_BF16: return indexer_typed((const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)w, (__half*)out, (int)B, (int)Lq, (int)Lk, (int)H, (int)d, q_strides, k_strides, w_strides, st);
        case CINN_F16: return indexer_typed((const __half*)q, (const __half*)k, (const __half*)w, (__half*)out, (int)B, (int)Lq, (int)Lk, (int)H, (int)d, q_strides, k_strides, w_strides, st);
        case CINN_F32: return indexer_typed((const float*)q, (const float*)k, (const float*)w, (__half*)out, (int)B, (int)Lq, (int)Lk, (int)H, (int)d, q_strides, k_strides, w_strides, st);
        default: set_error("lightning_indexer: unknown dtype tag %d", dtype); return CINN_ERR_INVALID;
    }
}

}  // namespace cinn
