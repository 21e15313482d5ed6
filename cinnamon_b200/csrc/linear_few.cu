// A linear without gradients on few rows (a prompt, a batch of generated tokens) as one kernel: the fp32 weight's 128 x 128 blocks
// and the activations' 1 x 128 tiles are quantised on their way into the MMA's operand tiles (src/kernels.py:41-132) and multiplied
// there (src/kernels.py:618-664).
//
// What has to move is the weight, once.  Quantised by a kernel of its own it moves 1.5 times (4 bytes read, 1 written, 1 read again),
// and both kernels of a small layer are launch latency.  A CTA takes 128 columns over a part of the reduction; the parts of a
// column tile are a cluster and add up through distributed shared memory, in order.  Per K block of 128 all 16 warps hold the
// block of the weight in registers (8 rows of a warp, 16 bytes per lane), agree on its amax, write e4m3 into the 128-byte-swizzled B tile,
// the rows of x into the A tile, and one warp issues the MMAs.  A CTA with one K block hands over its
// products as they are, with its rows' scales, and the cluster scales and adds in one step as the separate kernels do: the same bits.
// (Scaled before, each product was rounded once more: 0.0054 % of the results were not the exact sum in bf16, 0.0045 of the separate
// kernels'; 120 calls, 1 ... 128 rows, 256 ... 1024 columns.)  Without the loop over K blocks, the passes over the rows of x in step and the sums of
// the other CTAs asked for together: 1 x 512 -> 1024 5.8 -> 4.5 us and 128 x 512 -> 1024 8.5 -> 7.4 (back to back from a graph).  That is the form that linear_few_takes chooses.  A call of the entry point that has
// more K blocks than CTAs runs the other one: the next block's loads are in flight while one is converted, the product of the block
// before is scaled and added meanwhile, and every sum runs over whole K blocks in their order.
//
// All waits are bounded; cluster barriers are reached by every thread whatever a wait said.
#include "elements.cuh"
#include "tcgen05.cuh"
#include <cooperative_groups.h>

namespace cinn {

namespace few {

namespace cg = cooperative_groups;

__device__ int g_status = 0;               // 0, or (role << 8) | reason of a bounded wait that ran out

constexpr int WARPS = 16, THREADS = WARPS * 32;
constexpr int TILE = 128;                  // rows, columns and reduction of an operand tile
constexpr int TILE_BYTES = TILE * TILE;
constexpr int SMEM_BYTES = 4 * TILE_BYTES + 1024;      // two A and two B tiles; later 128 x 128 fp32 partial sums
constexpr int COLS = TILE / (WARPS / 4);   // columns of a promotion warp
constexpr int MAX_SLICES = 8;              // CTAs of a cluster: the portable limit

constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(TILE >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);

// byte `b` of row r of an operand tile: 128-byte rows, 16-byte chunks XOR-ed with the row
__device__ __forceinline__ uint32_t tile_off(int r, int b) { return (uint32_t)(r * 128 + ((((b >> 4) ^ r) & 7) << 4) + (b & 15)); }

// ONE: a K block per CTA, the form that linear_few_takes chooses; otherwise a run of them
template <typename TX, int DIV, bool ROUND, bool ONE>
__global__ void __launch_bounds__(THREADS, 1)
fp8_linear_few_kernel(const TX* __restrict__ x, int64_t ldx, const float* __restrict__ w, int64_t ldw, __nv_bfloat16* __restrict__ out,
                      int M, int N, int K) {
    constexpr int TMEM_COLS = (ONE ? 1 : 2) * TILE;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    __shared__ float s_red[2][WARPS], s_a[2][TILE];
    __shared__ float s_row[TILE];              // what the rows of this CTA's sums are multiplied with when the cluster adds them up
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t done0 = smem_u32(bars);
    volatile int* abort_flag = &abort_word;
    if (tid == 0) {
        abort_word = 0;
        for (int i = 0; i < 2; ++i) mbar_init(done0 + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tc_alloc(smem_u32(&tmem_slot), TMEM_COLS);        // (warp 0 has the barriers to set up)
    pdl_wait();
    if (warp == 1) pdl_trigger();
    const int slices = gridDim.x, slice = blockIdx.x, n0 = blockIdx.y * TILE;
    const int KB = (K + TILE - 1) / TILE, kb0 = ONE ? slice : KB * slice / slices, kb1 = ONE ? slice + 1 : KB * (slice + 1) / slices;
    const bool unscaled = ONE && slices > 1;               // products that stay as they are until they are added
    if (!ONE && tid < TILE) s_row[tid] = 1.0f;

    // the K block's piece of the weight: rows warp * 8 + i of the tile, 16 bytes per lane
    const float* wp = w + (int64_t)(n0 + warp * 8) * ldw + lane * 4;
    const int w_rows = min(8, N - n0 - warp * 8);
    float4 cur[8], nxt[ONE ? 1 : 8];
    auto fetch = [&](int kb, float4 (&r)[8]) {
        const bool live = kb < kb1 && kb * TILE + lane * 4 < K;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            r[i] = live && i < w_rows ? *reinterpret_cast<const float4*>(wp + (int64_t)i * ldw + kb * TILE) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    fetch(kb0, cur);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    const int quarter = warp & 3, group = warp >> 2;       // promotion: TMEM lane quarter, columns of the tile
    float acc[COLS], sb_old = 0.0f;
#pragma unroll
    for (int i = 0; i < COLS; ++i) acc[i] = 0.0f;
    bool alive = true;
    // adds K block number `it` of this CTA, scaled; sb: its weight scale
    auto promote = [&](int it, float sb) {
        const int buf = it & 1;
        const bool ok = mbar_wait_bounded(done0 + 8 * buf, (it >> 1) & 1, abort_flag, (8 << 8) | 1, &g_status);
        alive = __all_sync(0xffffffffu, ok) && alive;
        if (!alive || quarter * 32 >= M) return;
        tc_fence_after();
        float s = s_a[buf][quarter * 32 + lane] * sb;
        if (unscaled) {
            if (group == 0) s_row[quarter * 32 + lane] = s;
            s = 1.0f;
        }
        uint64_t s2;
        asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s));
#pragma unroll
        for (int c = 0; c < COLS; c += 16) {
            float v[16];
            tc_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + buf * TILE + group * COLS + c, v);
#pragma unroll
            for (int j = 0; j < 16; j += 2)
                asm("{\n\t.reg .b64 a, x;\n\t"
                    "mov.b64 a, {%0, %1};\n\t"
                    "mov.b64 x, {%2, %3};\n\t"
                    "fma.rn.f32x2 a, x, %4, a;\n\t"
                    "mov.b64 {%0, %1}, a;\n\t}"
                    : "+f"(acc[c + j]), "+f"(acc[c + j + 1]) : "f"(v[j]), "f"(v[j + 1]), "l"(s2));
        }
        tc_fence_before();
    };

    for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
        const int buf = it & 1;
        uint8_t* sA = smem + buf * TILE_BYTES;
        uint8_t* sB = smem + (2 + buf) * TILE_BYTES;
        if constexpr (!ONE) fetch(kb + 1, nxt);
        // the rows of x, a half-warp per 1 x 128 tile: 2-byte types are asked for here, so that they are there when the block is scaled
        const int sub = tid & 15, col = kb * TILE + sub * 8;
        constexpr bool EARLY = sizeof(TX) == 2;
        uint4 xr[EARLY ? TILE * 16 / THREADS : 1];
        if constexpr (EARLY) {
#pragma unroll
            for (int p = 0; p < TILE * 16 / THREADS; ++p) {
                const int r = p * (THREADS / 16) + (tid >> 4);
                xr[p] = r < M && col < K ? *reinterpret_cast<const uint4*>(x + (int64_t)r * ldx + col) : make_uint4(0u, 0u, 0u, 0u);
            }
        }
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            amax = fmaxf(fmaxf(fmaxf(amax, fabsf(cur[i].x)), fabsf(cur[i].y)), fmaxf(fabsf(cur[i].z), fabsf(cur[i].w)));
        amax = warp_max(amax);
        if (lane == 0) s_red[buf][warp] = amax;
        __syncthreads();
        amax = s_red[buf][0];
#pragma unroll
        for (int i = 1; i < WARPS; ++i) amax = fmaxf(amax, s_red[buf][i]);
        const float sb = scale_from_amax<DIV, false>(amax), db = divisor_of<DIV>(sb);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            *reinterpret_cast<uint32_t*>(sB + tile_off(warp * 8 + i, lane * 4)) =
                cvt_e4m3x4(scaled_clamped<DIV>(cur[i].x, db), scaled_clamped<DIV>(cur[i].y, db), scaled_clamped<DIV>(cur[i].z, db),
                           scaled_clamped<DIV>(cur[i].w, db));
        // `passes` of 32 rows in step, so that one's shuffles and quotients run under another's
        auto quantise_rows = [&](int first, auto passes) {
            constexpr int P = decltype(passes)::value;
            float a[P], v[P][8];
#pragma unroll
            for (int p = 0; p < P; ++p) {
                const int r = (first + p) * (THREADS / 16) + (tid >> 4);
                if constexpr (EARLY) {
                    Raw8<TX> raw;
                    raw.a = xr[first + p];
                    unpack_raw8<TX>(raw, v[p]);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[p][i] = 0.0f;
                    if (r < M && col < K) Elem<TX>::load8(x + (int64_t)r * ldx + col, v[p]);
                }
                a[p] = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i) a[p] = fmaxf(a[p], fabsf(v[p][i]));
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                for (int p = 0; p < P; ++p) a[p] = fmaxf(a[p], __shfl_xor_sync(0xffffffffu, a[p], o));
#pragma unroll
            for (int p = 0; p < P; ++p) {
                const int r = (first + p) * (THREADS / 16) + (tid >> 4);
                const float s = scale_from_amax<DIV, ROUND>(a[p]), d = divisor_of<DIV>(s);
                uint2 o2;
                o2.x = cvt_e4m3x4(scaled_clamped<DIV>(v[p][0], d), scaled_clamped<DIV>(v[p][1], d), scaled_clamped<DIV>(v[p][2], d),
                                  scaled_clamped<DIV>(v[p][3], d));
                o2.y = cvt_e4m3x4(scaled_clamped<DIV>(v[p][4], d), scaled_clamped<DIV>(v[p][5], d), scaled_clamped<DIV>(v[p][6], d),
                                  scaled_clamped<DIV>(v[p][7], d));
                *reinterpret_cast<uint2*>(sA + tile_off(r, sub * 8)) = o2;
                if (sub == 0) s_a[buf][r] = s;
            }
        };
        constexpr int PASSES = TILE * 16 / THREADS;
        if (!ONE || M <= THREADS / 16) {
#pragma unroll
            for (int p = 0; p < (ONE ? 1 : PASSES); ++p)
                if (p * (THREADS / 16) < M) quantise_rows(p, std::integral_constant<int, 1>{});
        } else if (M <= 2 * (THREADS / 16)) {
            quantise_rows(0, std::integral_constant<int, 2>{});
        } else {
            quantise_rows(0, std::integral_constant<int, PASSES>{});
        }
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (warp == 0) {
            tc_fence_after();
            const uint32_t lo = 1u << 16;
            tc_mma_f8_block<2>(tmem + buf * TILE, ((smem_u32(sA) >> 4) & 0x3FFF) | lo, ((smem_u32(sB) >> 4) & 0x3FFF) | lo, IDESC);
            tc_commit(done0 + 8 * buf);
        }
        if (!ONE && it > 0) promote(it - 1, sb_old);
        sb_old = sb;
        if constexpr (!ONE) {
#pragma unroll
            for (int i = 0; i < 8; ++i) cur[i] = nxt[i];
        }
    }
    if (kb1 > kb0) promote(kb1 - kb0 - 1, sb_old);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc(tmem, TMEM_COLS);
    }
    const int row = quarter * 32 + lane, c0 = n0 + group * COLS;
    if (slices == 1) {
        if (alive && row < M) {
            __nv_bfloat16* o = out + (int64_t)row * N + c0;
#pragma unroll
            for (int c = 0; c < COLS; c += 8) {
                __nv_bfloat162 h[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(acc[c + 2 * j], acc[c + 2 * j + 1]);
                if ((N & 7) == 0) {
                    if (c0 + c < N) *reinterpret_cast<uint4*>(o + c) = *reinterpret_cast<const uint4*>(h);
                } else {
                    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(h);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (c0 + c + j < N) o[c + j] = e[j];
                }
            }
        }
        return;
    }
    // partial sums of 512-byte rows, 16-byte chunks XOR-ed with the row, over the operand tiles
    if (row < M) {
#pragma unroll
        for (int c = 0; c < COLS; c += 4)
            *reinterpret_cast<float4*>(smem + row * 512 + ((((group * COLS + c) >> 2) ^ (row & 7)) << 4)) =
                make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int e = slice * THREADS + tid; e < M * 32; e += slices * THREADS) {
        const int r = e >> 5, c = e & 31, n = n0 + c * 4;
        // all of them asked for before the first is added: one round trip to the other SMs, not one after the other
        float4 part[MAX_SLICES];
        float f[MAX_SLICES];
#pragma unroll
        for (int s = 0; s < MAX_SLICES; ++s) {
            if (s >= slices) break;
            part[s] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(smem, s) + r * 512 + ((c ^ (r & 7)) << 4));
            f[s] = *cluster.map_shared_rank(&s_row[r], s);
        }
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < MAX_SLICES; ++s) {
            if (s >= slices) break;
            sum.x = fmaf(part[s].x, f[s], sum.x); sum.y = fmaf(part[s].y, f[s], sum.y);
            sum.z = fmaf(part[s].z, f[s], sum.z); sum.w = fmaf(part[s].w, f[s], sum.w);
        }
        __nv_bfloat162 h[2] = {__floats2bfloat162_rn(sum.x, sum.y), __floats2bfloat162_rn(sum.z, sum.w)};
        __nv_bfloat16* o = out + (int64_t)r * N + n;
        if ((N & 3) == 0) {
            if (n < N) *reinterpret_cast<uint2*>(o) = *reinterpret_cast<const uint2*>(h);
        } else {
            const __nv_bfloat16* v = reinterpret_cast<const __nv_bfloat16*>(h);
            for (int j = 0; j < 4; ++j)
                if (n + j < N) o[j] = v[j];
        }
    }
    cluster.sync();                                        // nobody leaves while its sums are being read
}

// Clusters of so many CTAs that run at once: a GPC holds whole ones only, and GPCs differ in their SMs.  Asked of the driver once per device.
static int clusters_at_once(int slices) {
    static std::atomic<int> known[64][MAX_SLICES + 1];
    constexpr auto kern = fp8_linear_few_kernel<__nv_bfloat16, CINN_DIV_FULL, false, true>;
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if ((n = known[dev][slices].load(std::memory_order_relaxed)) > 0) return n;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3((unsigned)slices, (unsigned)sm_count(), 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = slices;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (allow_smem_once<kern>(SMEM_BYTES) != CINN_OK || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    known[dev][slices].store(n, std::memory_order_relaxed);
    return n;
}

// CTAs that share a column tile's reduction: one per K block if their clusters all run at once and leave an eighth of the SMs (sizes that do
// not divide 16: a quarter) to what runs beside.  Sixteen clusters of eight were 128 CTAs of 148 and ran in two turns: 8 x 1024 -> 2048 12.5 us
// where the two kernels take 7.5.
static bool fits_at_once(int64_t tiles, int s) {
    return s == 1 || (tiles * s <= sm_count() * (16 % s == 0 ? 7 : 6) / 8 && tiles <= clusters_at_once(s));
}
static int slices_of(int64_t N, int64_t K) {
    const int64_t tiles = (N + TILE - 1) / TILE, KB = (K + TILE - 1) / TILE;
    int s = (int)(KB < MAX_SLICES ? KB : MAX_SLICES);
    while (!fits_at_once(tiles, s)) --s;
    return s;
}

template <typename TX, int DIV, bool ROUND, bool ONE>
static int launch_form(const TX* x, int64_t ldx, const float* w, int64_t ldw, __nv_bfloat16* out, int M, int N, int K, int slices,
                       cudaStream_t st) {
    constexpr auto kern = fp8_linear_few_kernel<TX, DIV, ROUND, ONE>;
    if (const int failed = allow_smem_once<kern>(SMEM_BYTES)) return failed;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)slices, (unsigned)((N + TILE - 1) / TILE), 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = slices;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    CINN_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, x, ldx, w, ldw, out, M, N, K));
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

template <typename TX, int DIV, bool ROUND>
static int launch(const TX* x, int64_t ldx, const float* w, int64_t ldw, __nv_bfloat16* out, int M, int N, int K, cudaStream_t st) {
    const int slices = slices_of(N, K);
    return (K + TILE - 1) / TILE == slices ? launch_form<TX, DIV, ROUND, true>(x, ldx, w, ldw, out, M, N, K, slices, st)
                                           : launch_form<TX, DIV, ROUND, false>(x, ldx, w, ldw, out, M, N, K, slices, st);
}

}  // namespace few

bool gemm_sms_capped();                                    // gemm.cu: other kernels are to run beside the multiplications

static inline bool on16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static bool fits(const void* x, int x_dtype, int64_t ldx_m, int64_t ldx_k, const void* w, int w_dtype, int64_t ldw_n, int64_t ldw_k, int64_t M,
                 int64_t N, int64_t K) {
    const int64_t item = x_dtype == CINN_F32 ? 4 : 2;
    return M >= 1 && M <= few::TILE && N >= 1 && N <= (1 << 22) && K >= 16 && K % 16 == 0 && K < (1LL << 24) && w_dtype == CINN_F32 &&
           (x_dtype == CINN_BF16 || x_dtype == CINN_F16 || x_dtype == CINN_F32) && ldx_k == 1 && ldw_k == 1 && ldx_m >= K && ldw_n >= K &&
           ldx_m * item % 16 == 0 && ldw_n % 4 == 0 && on16(x) && on16(w);
}

// Worth it where every CTA has one K block, for then the launch that it saves is what counts; with more, each block waits for its
// piece of the weight, where the quantiser's many CTAs stream them.  us a call, two kernels against this one, one block: weights that stay in
// L2, 4 x 1024 -> 1344 9.9 and 6.7, 128 x 512 -> 1024 9.7 and 8.1; every call another weight, 10.0 and 6.7, 9.7 and 8.4.  Two blocks, 7 x 2048 -> 1472
// 11.9 and 12.3, 99 x 1472 -> 1600 12.1 and 14.4; three, 117 x 2368 -> 768 12.0 and 18.5.
// Replayed from a CUDA graph the launch costs next to nothing and the exchange between the CTAs counts, which grows with the rows: 128 x 512 -> 1024
// 5.8 and 7.4, 64 5.7 and 5.8, 32 5.7 and 5.3, 128 x 1024 -> 1344 7.0 and 9.0, 32 6.6 and 6.3; without an exchange, 128 x 128 -> 8192, 6.0 and 5.3.
// So callers under capture take it for up to 32 rows, or for one K block in all (csrc/host/linear.cpp).
bool linear_few_takes(const void* x, int x_dtype, int64_t ldx_m, int64_t ldx_k, const void* w, int w_dtype, int64_t ldw_n, int64_t ldw_k,
                      int64_t M, int64_t N, int64_t K) {
    const int64_t KB = (K + few::TILE - 1) / few::TILE;
    return KB <= few::MAX_SLICES && fits(x, x_dtype, ldx_m, ldx_k, w, w_dtype, ldw_n, ldw_k, M, N, K) && !gemm_sms_capped() &&
           few::fits_at_once((N + few::TILE - 1) / few::TILE, (int)KB);
}

int linear_few(const void* x, int x_dtype, int64_t ldx, int round_scale, const float* w, int64_t ldw, void* out, int64_t M, int64_t N,
               int64_t K, int div_mode, cudaStream_t st) {
    CINN_CHECK_ARG(x && w && out && on16(out), "linear_few: null or unaligned pointer");
    CINN_CHECK_ARG(fits(x, x_dtype, ldx, 1, w, CINN_F32, ldw, 1, M, N, K), "linear_few: bad shape, type or alignment");
    CINN_CHECK_ARG(div_mode == CINN_DIV_FULL || div_mode == CINN_DIV_RN, "linear_few: unknown div_mode %d", div_mode);
    __nv_bfloat16* o = (__nv_bfloat16*)out;
    const int m = (int)M, n = (int)N, k = (int)K;
#define CINN_FEW(T)                                                                                                          \
    do {                                                                                                                     \
        const T* xt = (const T*)x;                                                                                           \
        if (div_mode == CINN_DIV_FULL)                                                                                       \
            return round_scale ? few::launch<T, CINN_DIV_FULL, true>(xt, ldx, w, ldw, o, m, n, k, st)                        \
                               : few::launch<T, CINN_DIV_FULL, false>(xt, ldx, w, ldw, o, m, n, k, st);                      \
        return round_scale ? few::launch<T, CINN_DIV_RN, true>(xt, ldx, w, ldw, o, m, n, k, st)                              \
                           : few::launch<T, CINN_DIV_RN, false>(xt, ldx, w, ldw, o, m, n, k, st);                            \
    } while (0)
    if (x_dtype == CINN_BF16) CINN_FEW(__nv_bfloat16);
    if (x_dtype == CINN_F16) CINN_FEW(__half);
    CINN_FEW(float);
#undef CINN_FEW
}

int read_linear_few_status(int* out, int reset) {
    int v = 0;
    CINN_CHECK_CUDA(cudaMemcpyFromSymbol(&v, few::g_status, sizeof(int)));
    if (reset && v != 0) {
        int z = 0;
        CINN_CHECK_CUDA(cudaMemcpyToSymbol(few::g_status, &z, sizeof(int)));
    }
    *out = v;
    return CINN_OK;
}

}  // namespace cinn
