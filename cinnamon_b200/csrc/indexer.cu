// Lightning indexer logits: I[b, t, s] = sum_h relu(q[b, t, h, :] . k[b, s, :]) * w[b, t, h], fp16 result.
//
// Semantics of cinnamon's lightning_indexer_kernel / lightning_indexer_fused (src/kernels.py:321-433): the
// operands of the dot product are rounded to fp16 (:374), products are accumulated in fp32, ReLU and the head
// weights are applied in fp32 (:377), the logits are stored as fp16 (:381).
//
// Tensor-core kernel (rows up to 128 wide, the widths indexers have): one CTA computes 128 queries x 128 keys.  The
// inputs may have any strides and types, so they are not fetched by TMA: all threads read them (16 bytes at a time
// where the layout allows), round to fp16 and write the 128-byte-swizzled tiles the MMA reads.  One thread issues
// tcgen05.mma (kind::f16, 128 x 128 x d per head) into one of two 128-column tensor-memory buffers while eight warps
// fold the previous head's dot products, relu * w, into fp32 registers (64 per thread).  Queries of up to 64 KiB of
// heads are resident at a time, so two CTAs share an SM and one loads while the other computes.  Bound: two CUDA-core
// instructions per (query, key, head) next to the MMAs, and the write of the logits.
// Measured (8 x 1024 queries and keys, 4 heads of 64, bf16; the whole call): 439 us on the scalar kernel, 21 us here.
//
// Scalar kernel (wider rows): 16 queries x 64 keys per CTA.  The key tile is kept transposed in shared memory as fp16
// ([d][key], so the 16 lanes that share a query read 16 consecutive keys), the queries of all heads as fp16
// ([query][head][d], broadcast reads).  A thread owns one query and four keys: per head a d-long dot product for each
// of the four, then relu * w into the running sum.
#include "tcgen05.cuh"

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
            for (int s = 0; s < a.dpad / 16; ++s) {
                const uint32_t off = (s >> 2) * ITC_PANEL + (s & 3) * 32;
                tc_mma_f16(tmem + buf * ITC_T, make_smem_desc(smem_u32(sQ) + h * head_bytes + off, 16, 1024),
                           make_smem_desc(smem_u32(sK) + off, 16, 1024), make_idesc_f16(false, ITC_T, ITC_T), s > 0 ? 1u : 0u);
            }
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
    indexer_tc_kernel<T><<<grid, ITC_THREADS, smem, st>>>(q, k, w, out, a);
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
    if (d <= ITC_MAX_D) return indexer_tc_typed<T>(q, k, w, out, B, Lq, Lk, H, d, sq, sk, sw, st);
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
