// Sparse attention on the tensor cores: see attn_tc.cuh for what it trades against the gather kernels.
//
// Scratch (from the caller, one block per call): what the queries picked (Picks), the bf16 parts of the inputs and one
// flag word.  Everything is rebuilt on every call.  It is about as large as the tensors (32 x 8 x 1024 queries of 192 / 64 in
// fp32, 128 picks: 0.70 GB forward, 1.07 GB backward); a call that would need more than MAX_SCRATCH_BYTES takes the gathers.
//
// What a dense tile cannot express falls back on the device, without the host knowing: a key picked more than 255 times
// by one query, or results that are not finite (a NaN in a row nobody picked must not reach anyone, and 0 * NaN on a
// tensor core would let it) set the flag, and the gather kernel, launched behind with that flag as its condition,
// computes the whole call again.
#include <type_traits>
#include "attn_tc.cuh"
#include <atomic>
#include <cmath>

namespace cinn {
namespace atc {

__device__ int g_attn_status = 0;          // 0, or (role << 8) | reason of a bounded wait that ran out

// A bounded wait of a whole warp, with one verdict for all its lanes.
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, abort_flag, code, &g_attn_status));
}

// The MMA warp's end of a ring of panels.  (Asking for the next panel before this one's MMAs, so as to wait only if it is not
// there, delays the MMAs: 320 to 350 cycles per panel of four where the plain wait takes the MMAs' own 256.)
template <int RING> struct PanelRing {
    uint32_t full0, empty0, base;
    volatile int* abort_flag;
    int code;
    uint32_t slot, phase;
    bool alive;
    __device__ __forceinline__ PanelRing(uint32_t full, uint32_t empty, uint32_t panels, volatile int* flag, int reason)
        : full0(full), empty0(empty), base(panels), abort_flag(flag), code(reason), slot(0), phase(0), alive(true) {}
    // the next panel's address, and the slot to release once the MMAs that read it are issued
    __device__ __forceinline__ bool next(uint32_t& addr, uint32_t& taken) {
        if (!alive || !wait_warp(full0 + 8 * slot, phase, abort_flag, code)) return alive = false;
        tc_fence_after();
        addr = base + slot * PANEL;
        taken = slot;
        if (++slot == RING) { slot = 0; phase ^= 1u; }
        return true;
    }
    __device__ __forceinline__ void release(uint32_t taken) { tc_commit(empty0 + 8 * taken); }
};

// The four warps of a warpgroup meet at a barrier in shared memory (four arrivals): bounded, so that a warp that gave up
// leaves nobody behind.
struct WarpgroupBarrier {
    uint32_t bar, phase;
    volatile int* abort_flag;
    __device__ __forceinline__ bool sync(int code) {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
        return wait_warp(bar, phase++ & 1u, abort_flag, code);
    }
};

// ---------------------------------------------------------------------------
// what the queries picked
// ---------------------------------------------------------------------------
// One warp per query, in shared memory: the bits of its K indices, the running count of bits before every word, and from
// these the rank of every slot's key.  Bound by reading the indices: 33 MB at 32 x 1024 queries x 128.
__global__ void __launch_bounds__(128)
picks_kernel(const int64_t* __restrict__ idx, uint32_t* __restrict__ bits, uint16_t* __restrict__ rank, uint8_t* __restrict__ count,
             uint16_t* __restrict__ before_out, int* __restrict__ repeats, int* __restrict__ flag, int64_t n_rows, int L, int words, int K, int warps) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) uint32_t sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp >= warps) return;
    const int n_tiles = words / (T / 32);
    uint32_t* b = sm + (size_t)warp * (2 * words + K);
    uint32_t* before = b + words;
    uint32_t* cnt = before + words;
    for (int64_t w = (int64_t)blockIdx.x * warps + warp; w < n_rows; w += (int64_t)gridDim.x * warps) {
        const int64_t bt = w / L;
        const int t = (int)(w - bt * L);
        const int64_t* row = idx + w * K;
        for (int i = lane; i < words; i += 32) b[i] = 0u;
        for (int i = lane; i < K; i += 32) cnt[i] = 0u;
        __syncwarp();
        for (int j = lane; j < K; j += 32) {
            const int64_t i = row[j];
            if (i >= 0 && i <= t) atomicOr(b + (i >> 5), 1u << (i & 31));
        }
        __syncwarp();
        uint32_t carry = 0;
        for (int i0 = 0; i0 < words; i0 += 32) {
            const int i = i0 + lane;
            const uint32_t n = i < words ? __popc(b[i]) : 0u;
            uint32_t incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (i < words) {
                before[i] = carry + incl - n;
                bits[w * words + i] = b[i];
                before_out[w * words + i] = (uint16_t)before[i];
            }
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncwarp();
        for (int j = lane; j < K; j += 32) {
            const int64_t i = row[j];
            uint32_t r = 0xffffu;
            if (i >= 0 && i <= t) {
                r = before[i >> 5] + __popc(b[i >> 5] & ((1u << (i & 31)) - 1u));
                atomicAdd(cnt + r, 1u);
            }
            rank[w * K + j] = (uint16_t)r;
        }
        __syncwarp();
        uint32_t most = 0;
        for (int i = lane; i < K; i += 32) {
            most = max(most, cnt[i]);
            count[w * K + i] = (uint8_t)min(cnt[i], (uint32_t)MAX_COUNT);
        }
        if (most > 1) repeats[bt * n_tiles + t / T] = 1;
        if (most > MAX_COUNT) *flag = 1;
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// bf16 parts of the inputs: (parts, rows, dpad), columns beyond d are zero
// ---------------------------------------------------------------------------
template <typename U> __device__ __forceinline__ float widen(U v);
template <> __device__ __forceinline__ float widen<float>(float v) { return v; }
template <> __device__ __forceinline__ float widen<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float widen<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

struct SplitJob { const void* src; uint16_t* dst; int64_t rows; int d, dpad; };
struct SplitJobs { SplitJob job[4]; int n; };

// Bound by HBM: 4 bytes in and 6 out per fp32 element.
template <typename U, int NS>
__global__ void __launch_bounds__(256)
split_parts_kernel(const SplitJobs jobs) {
    pdl_wait();
    pdl_trigger();
    for (int n = 0; n < jobs.n; ++n) {
        const SplitJob jb = jobs.job[n];
        const U* src = static_cast<const U*>(jb.src);
        const int per_row = jb.dpad / 8;
        const int64_t total = jb.rows * per_row, plane = jb.rows * jb.dpad;
        const bool vec = jb.d % 8 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
        for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (int64_t)gridDim.x * 256) {
            const int64_t r = e / per_row;
            const int c = (int)(e - r * per_row) * 8;
            float v[8];
            const U* p = src + r * jb.d + c;
            if (vec && c < jb.d) {
                if constexpr (sizeof(U) == 4) {
                    const float4 a = __ldcs(reinterpret_cast<const float4*>(p)), b = __ldcs(reinterpret_cast<const float4*>(p) + 1);
                    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
                } else {
                    const uint4 raw = __ldcs(reinterpret_cast<const uint4*>(p));
                    const U* u = reinterpret_cast<const U*>(&raw);
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = widen<U>(u[i]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = c + i < jb.d ? widen<U>(p[i]) : 0.0f;
            }
            uint32_t w[3][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) split2(v[2 * i], v[2 * i + 1], w[0][i], w[1][i], w[2][i]);
#pragma unroll
            for (int s = 0; s < NS; ++s)
                *reinterpret_cast<uint4*>(jb.dst + s * plane + r * jb.dpad + c) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
        }
    }
}

// ---------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------
struct FwdArgs {
    Picks picks;
    float* out; void* out_cast; float* lse; float* attn; int* flag;
    int H, L, words, K, Dv, BH, n_tiles, group;   // words: 32-key words per query
    float scale;
    int out_cast_tag;                      // CINN_BF16 / CINN_F16: the output once more in that type (out_cast)
};

// Blocks walk the heads in groups, within a group from the tiles with the most work to those with the least: the long
// tiles of all its heads start first, and the heads in flight at a time (`group` of them, about three rounds of blocks)
// keep their operands in L2.
__device__ __forceinline__ void tile_of_block(int n_tiles, int BH, int group, int& tile, int& bh) {
    const int g = blockIdx.x / (group * n_tiles), r = blockIdx.x - g * group * n_tiles;
    const int heads = min(group, BH - g * group);
    tile = n_tiles - 1 - r / heads;
    bh = g * group + r % heads;
}

// Shared memory: queries [part][64-column panel] | ring of panels | barriers | row maxima on their way between two warps.
// With one part and many blocks two CTAs share an SM, each with one pair of softmax warpgroups: the first loads, the
// merge and the permutation of one run under the other's tiles (a CTA of two pairs spends 20 000 of its 55 000 cycles on them, at
// 8 x 8 x 1531 queries of 192).  Where that pays: one_pair.
// Three parts of 192 columns need most of an SM's shared memory for the queries alone.
template <int NS, int ND, int PAIRS_> struct FwdShape {
    static constexpr int PAIRS = PAIRS_;                   // of softmax warpgroups
    static constexpr int THREADS = (8 * PAIRS + 2) * 32;   // and a TMA warp, an MMA warp
    static constexpr int Q_PANELS = NS * ND;
    static constexpr int RING = PAIRS == 1 ? 6 - Q_PANELS : Q_PANELS > 6 ? 4 : 6;
    static constexpr int BAR_OFF = (Q_PANELS + RING) * PANEL;
    static constexpr int PAIR_OFF = BAR_OFF + 512;         // [round & 1][pair][half][row]
    static constexpr int LSE_OFF = PAIR_OFF + 4 * PAIRS * T * 4;
    static constexpr int BYTES = LSE_OFF + T * 4 + 1024;
};

// A key picked several times counts as often: p[i] times the next count for every bit i, the counts in the order of the bits.  At most
// sixteen of them, in five words that are all on their way before the first is used (past a row's counts they may hold the next
// row's bytes, or the scratch behind them).  Byte by byte behind a condition a warp waits for L2 at each of the sixteen columns: beside the
// operands of two CTAs there is hardly an L1.  11 heads of 2048 queries of 64 in bf16, 128 picks with repeats: 199 us a
// call so, 125 like this.
__device__ __forceinline__ void times_counts(float (&p)[16], uint32_t bit, const uint8_t*& count) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(count);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(at & ~(uintptr_t)3);
    const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3), w4 = __ldg(w + 4), by = (uint32_t)(at & 3) * 8;
    uint32_t c[5] = {__funnelshift_r(w0, w1, by), __funnelshift_r(w1, w2, by), __funnelshift_r(w2, w3, by), __funnelshift_r(w3, w4, by), 0u};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        p[i] *= (float)(c[0] & 0xffu);                    // (of a key that was not picked p is 0)
        if (bit & (1u << i)) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (4 * j < 15 - i) c[j] = __funnelshift_r(c[j], c[j + 1], 8);           // (the other words are past what is still to come)
        }
    }
    count += __popc(bit & 0xffffu);
}

// 16 columns of a thread's row: scores to probabilities relative to `m`, left as parts over the scores and beside them.  The
// picked raw scores go to `to` in passing when PUSH.  (32 columns at a time spilled.)
template <bool PUSH, bool REPEATS>
__device__ __forceinline__ void softmax_chunk(uint32_t t_s, uint32_t t_lead, uint32_t bit, float scale, float m,
                                              const uint8_t*& count, float*& to, uint64_t (&l)[2]) {
    uint32_t v[16];
    float p[16];
    ld16(t_s, v);
    ld_wait();
    const uint64_t sc = pair2(scale, scale), off = pair2(-m, -m), l2e = pair2(1.4426950408889634f, 1.4426950408889634f);
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        unpair2(mul2(fma2(pair2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), sc, off), l2e), p[i], p[i + 1]);
#pragma unroll
        for (int e = i; e < i + 2; ++e) {
            p[e] = exp2_fast(p[e]);
            if constexpr (PUSH) push_if(bit, 1u << e, to, __uint_as_float(v[e]), p[e]);
            else p[e] = bit & (1u << e) ? p[e] : 0.0f;
        }
    }
    if constexpr (REPEATS) times_counts(p, bit, count);
#pragma unroll
    for (int i = 0; i < 16; i += 2) l[(i >> 1) & 1] = add2(l[(i >> 1) & 1], pair2(p[i], p[i + 1]));
    store_parts16(t_s, t_lead, p);
}

// Raw scores by rank -> probabilities by slot, in place: rows of K slots, one warp of WARPS.  Every slot of a row is read
// before any of it is written.
template <int WARPS>
__device__ __forceinline__ void by_slot(const uint16_t* rank, float* attn, const float* lse, int rows, int K, float scale, int warp, int lane) {
    // (a caller's buffer may start on any 4-byte boundary: rows there go slot by slot)
    if (K >= 4 && K <= 512 && (K & (K - 1)) == 0 && (reinterpret_cast<uintptr_t>(attn) & 15) == 0) {
        // whole rows in batches of 512 slots, four in a row per lane and load
        const int log_k = 31 - __clz(K), end = rows << log_k;
#pragma unroll 1
        for (int e0 = warp * 512; e0 < end; e0 += WARPS * 512) {
            uint2 c[4];
            float4 x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) c[u] = __ldg(reinterpret_cast<const uint2*>(rank + min(e0 + u * 128 + lane * 4, end - 4)));
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = min(e0 + u * 128 + lane * 4, end - 4), row = e >> log_k;
                const float* from = attn + (row << log_k);
                const float z = lse[row];
                auto one = [&](uint32_t at) {
                    const float s = from[min((int)at, K - 1)];
                    return at == 0xffffu ? 0.0f : exp_fast(s * scale - z);
                };
                x[u] = make_float4(one(c[u].x & 0xffffu), one(c[u].x >> 16), one(c[u].y & 0xffffu), one(c[u].y >> 16));
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * 128 + lane * 4;
                if (e < end) *reinterpret_cast<float4*>(attn + e) = x[u];
            }
        }
        return;
    }
    // a warp takes sixteen pieces of 32 slots at a time with all loads in flight
    constexpr int U = MAX_SLOTS / 32;
    const int chunks = (K + 31) / 32, per = U / chunks;
    for (int k0 = warp; k0 < rows; k0 += WARPS * per) {                     // rows k0, k0 + WARPS, ...
        float v[U];
        uint32_t c[U];
        int rr = k0, j = lane;                            // piece u of the batch: its row and this lane's slot
        auto advance = [&] { if ((j += 32) >= chunks * 32) { j = lane; rr += WARPS; } };
        const int end = min(rows, k0 + WARPS * per);
#pragma unroll
        for (int u = 0; u < U; ++u, advance()) {
            // (loads from clamped places and a choice afterwards: behind a condition they would go one by one)
            const uint32_t x = rank[min(rr, end - 1) * K + min(j, K - 1)];
            c[u] = rr < end && j < K ? x : 0xffffu;
        }
        rr = k0; j = lane;
#pragma unroll
        for (int u = 0; u < U; ++u, advance()) {
            const float x = attn[min(rr, end - 1) * K + min((int)c[u], K - 1)] * scale;
            v[u] = c[u] != 0xffffu ? x : -INFINITY;
        }
        __syncwarp();
        rr = k0; j = lane;
#pragma unroll
        for (int u = 0; u < U; ++u, advance())
            if (rr < end && j < K) attn[rr * K + j] = exp_fast(v[u] - lse[rr]);
    }
}

// One CTA: 128 queries of one head and 64 value columns (blockIdx.z), over all key tiles up to the queries' own.  A pair of
// softmax warpgroups takes a key tile, a thread a query and half of the tile's keys; two pairs (of one CTA, which merge their
// maxima, sums and outputs at the end, or of two) keep out of each other's way, and while one turns scores into probabilities the
// tensor core works for the other.  A thread reads its 64 scores from tensor memory twice: for the maximum,
// which it exchanges with the thread of the other half, and to write exp(score - max) back as three bf16 parts, the A operand
// of P V, in the columns it has just read and 32 beside them, leaving the raw scores of the picked keys in the probabilities'
// output (by rank; permuted and normalised at the end).  256 columns per pair: 128 scores, 64 leading parts, 64 of output.
// Bound by the instructions per score (29, the merge and the permutation among them; they issue in 47 % of the cycles) and, in
// fp32, by the panels' way into shared memory: the operands of 72 MMAs and the 15 panels of a tile take 7300 cycles of its bandwidth.
// The call of 8 x 8 x 1531 queries of 192 in bf16 takes 229 us with two warpgroups per CTA, a thread per row, and 188 so (190 with two pairs);
// 256 heads of 947 in fp32 831 and 771.  (Skipping
// chunks that no query of a warp picked from: 2 % slower; the next chunk's scores in flight during this one's: 6 % slower, spills.)
// NS: bf16 parts of q, k, v; ND: 64-column panels of q and k.
template <int NS, int ND, int PAIRS>
__global__ void __launch_bounds__(FwdShape<NS, ND, PAIRS>::THREADS, 3 - PAIRS)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const FwdArgs a) {
    pdl_wait();
    using S = FwdShape<NS, ND, PAIRS>;
    constexpr int TMA_WARP = 8 * PAIRS, MMA_WARP = TMA_WARP + 1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sq = smem_u32(smem), ring = sq + S::Q_PANELS * PANEL;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::BAR_OFF);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + S::RING), qfull = smem_u32(bars + 2 * S::RING);
    const uint32_t sfull0 = qfull + 8, pready0 = qfull + 24, odone0 = qfull + 40;       // two each
    const uint32_t pair0 = odone0 + 16;                   // eight, one per two warps that share rows
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S::RING + 15);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* s_pair = reinterpret_cast<float*>(smem + S::PAIR_OFF);
    float* s_lse = reinterpret_cast<float*>(smem + S::LSE_OFF);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int qt, bh;
    tile_of_block(a.n_tiles, a.BH, a.group, qt, bh);
    const int n_qt = a.n_tiles, half = blockIdx.z;
    const int q0 = qt * T, n = qt + 1;                    // key tiles
    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < S::RING; ++i) { mbar_init(full0 + 8 * i, 1); mbar_init(empty0 + 8 * i, 1); }
        mbar_init(qfull, 1);
        for (int i = 0; i < 2; ++i) { mbar_init(sfull0 + 8 * i, 1); mbar_init(pready0 + 8 * i, 8); mbar_init(odone0 + 8 * i, 1); }
        for (int i = 0; i < 8; ++i) mbar_init(pair0 + 8 * i, 2);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        tc_alloc(smem_u32(tmem_slot), 256 * PAIRS);
        pdl_trigger();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == TMA_WARP) {
        if (lane == 0) {
            mbar_expect_tx(qfull, S::Q_PANELS * PANEL);
            for (int p = 0; p < NS; ++p)
                for (int c = 0; c < ND; ++c) tma_load_3d(&tmQ, qfull, sq + (p * ND + c) * PANEL, c * 64, q0, p * a.BH + bh);
            uint32_t it = 0;
            bool alive = true;
            auto fetch = [&](const CUtensorMap* m, int x, int y, int z) {
                const uint32_t s = it % S::RING, ph = (it / S::RING) & 1;
                if (!alive || !mbar_wait_bounded(empty0 + 8 * s, ph ^ 1, abort_flag, (8 << 8) | 1, &g_attn_status)) { alive = false; return; }
                mbar_expect_tx(full0 + 8 * s, PANEL);
                tma_load_3d(m, full0 + 8 * s, ring + s * PANEL, x, y, z);
                ++it;
            };
            auto keys = [&](int j) {
                if constexpr (NS > 1)
                    for (int c = 0; c < ND; ++c)
                        for (int p = NS - 1; p >= 0; --p) fetch(&tmK, c * 64, j * T, p * a.BH + bh);
                for (int c = 0; c < ND; ++c) fetch(&tmK, c * 64, j * T, bh);
            };
            for (int j = 0; j <= n && alive; ++j) {       // in the order in which the MMA warp takes them
                if (PAIRS > 1 && j < n) keys(j);
                if (j > 0)
                    for (int p = NS - 1; p >= 0; --p) fetch(&tmV, half * 64, (j - 1) * T, p * a.BH + bh);
                if (PAIRS == 1 && j < n) keys(j);
            }
            if (!alive) {                                 // abandoned: let the copies in flight land
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000LL) { }
            }
        }
    } else if (warp == MMA_WARP) {
        if (wait_warp(qfull, 0, abort_flag, (8 << 8) | 2)) {
            constexpr uint32_t id_s = make_idesc_f16(true, T, T), id_o = make_idesc_f16(true, T, 64, false, true);
            PanelRing<S::RING> panels(full0, empty0, ring, abort_flag, (8 << 8) | 3);
            // scores of key tile j, over the probabilities of the pair's tile before, whose product was issued before
            auto scores = [&](int j) {
                const uint32_t d = tmem + j % PAIRS * 256;
                bool first = true;
                // query parts [x_lo, x_hi] of column panel c against the ring's next key panel
                auto product = [&](int c, int x_hi, int x_lo) {
                    uint32_t kp, slot;
                    if (!panels.next(kp, slot)) return;
                    const uint32_t kd = panel_desc(kp);
                    uint32_t qd = panel_desc(sq + c * PANEL) + x_hi * ND * (PANEL >> 4);
                    for (int x = x_hi; x >= x_lo; --x) {
                        mma_panels(d, qd, kd, id_s, first);
                        first = false;
                        qd -= ND * (PANEL >> 4);
                    }
                    panels.release(slot);
                };
                // The tensor core truncates the running sum at every step, so the small products go first and the leading
                // ones, for which the keys' leading parts are fetched again, last: ND x 4 truncations at full size instead of
                // six times as many.
                if constexpr (NS > 1)
                    for (int c = 0; c < ND; ++c)
                        for (int p = NS - 1; p >= 0; --p) product(c, NS - 1 - p, p == 0 ? 1 : 0);
                for (int c = 0; c < ND; ++c) product(c, 0, 0);
                tc_commit(sfull0 + 8 * (j % PAIRS));
            };
            for (int j = 0; j <= n && panels.alive; ++j) {
                if (PAIRS > 1 && j < n) scores(j);
                if (j > 0 && panels.alive) {              // output of key tile j - 1
                    const int i = j - 1, w = i % PAIRS;
                    if (!wait_warp(pready0 + 8 * w, (i / PAIRS) & 1, abort_flag, (8 << 8) | 4)) break;
                    tc_fence_after();
                    const uint32_t base = tmem + w * 256;
                    bool first = NS > 1 || i < PAIRS;
                    for (int p = NS - 1; p >= 0; --p) {
                        uint32_t vp, slot;
                        if (!panels.next(vp, slot)) break;
                        const uint32_t vd = panel_desc(vp);
                        if (p == 0) { mma_part_at<2>(base + 192, base, base + 128, vd, id_o, first); first = false; }
                        if (p <= 1) { mma_part_at<1>(base + 192, base, base + 128, vd, id_o, first); first = false; }
                        mma_part_at<0>(base + 192, base, base + 128, vd, id_o, first);
                        first = false;
                        panels.release(slot);
                    }
                    if (i + PAIRS >= n) tc_commit(odone0 + 8 * w);
                }
                if (PAIRS == 1 && j < n) scores(j);
            }
        }
    } else {
        const int pair = warp >> 3, h = (warp >> 2) & 1, quarter = warp & 3, r = quarter * 32 + lane;
        const int t = q0 + r, b = bh / a.H;
        const bool live = t < a.L;
        const uint32_t base = tmem + ((uint32_t)(quarter * 32) << 16) + pair * 256;
        const uint32_t t_s = base + h * 64, t_lead = base + 128 + h * 32, t_o = base + 192 + h * 32;      // this half's
        const int64_t qrow = (int64_t)b * a.L + min(t, a.L - 1);
        const uint4* bits = reinterpret_cast<const uint4*>(a.picks.bits + qrow * a.words);
        const uint16_t* before = a.picks.before + qrow * a.words + h * 2;
        const bool repeats = a.picks.repeats[b * n_qt + qt] != 0;
        float* row = a.attn + ((int64_t)bh * a.L + min(t, a.L - 1)) * a.K;
        const uint8_t* counts = a.picks.count + qrow * a.K;
        float m = -INFINITY;
        uint64_t l2[2] = {0u, 0u};                        // (0, 0) each
        // With three parts a tile's output is added up here, rounded to nearest: the tensor core truncates, and over a long
        // row of tiles that would show in fp32.
        constexpr bool KEEP = NS > 1;
        uint64_t o_sum[KEEP ? 16 : 1];
#pragma unroll
        for (int i = 0; i < (KEEP ? 16 : 1); ++i) o_sum[i] = 0u;
        auto add_output = [&] {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float o[16];
                tc_ld16(t_o + c * 16, o);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    uint64_t& sum = o_sum[KEEP ? c * 8 + i : 0];
                    sum = add2(sum, pair2(o[2 * i], o[2 * i + 1]));
                }
            }
        };
        bool alive = true;
        // the larger of both halves' values, in both
        uint32_t rounds = 0;
        const uint32_t pair_bar = pair0 + 8 * (pair * 4 + quarter);
        auto exchange = [&](float& x) {
            float* slot = s_pair + ((rounds & 1) * PAIRS + pair) * 2 * T + r;
            slot[h * T] = x;
            __syncwarp();
            if (lane == 0) mbar_arrive(pair_bar);
            if (!wait_warp(pair_bar, rounds & 1, abort_flag, (8 << 8) | 7)) return false;
            x = fmaxf(x, slot[(h ^ 1) * T]);
            ++rounds;
            return true;
        };
        const uint4 none = make_uint4(0u, 0u, 0u, 0u);
        uint4 mine = live && pair < n ? __ldg(bits + pair) : none;
        uint32_t rank = pair < n ? __ldg(before + pair * 4) : 0u;
        const uint64_t scale2 = pair2(a.scale, a.scale);
        for (int j = pair; j < n; j += PAIRS) {
            const uint4 cur = mine;
            float* to = row + rank;                       // the next picked key's raw score goes here
            const uint8_t* count = counts + rank;
            if (j + PAIRS < n) {                          // the next tile's, in flight during this one
                mine = live ? __ldg(bits + j + PAIRS) : none;
                rank = __ldg(before + (j + PAIRS) * 4);
            }
            if (!wait_warp(sfull0 + 8 * pair, (j / PAIRS) & 1, abort_flag, (8 << 8) | 5)) { alive = false; break; }
            tc_fence_after();
            if constexpr (KEEP)
                if (j >= PAIRS) add_output();             // of the pair's tile before, issued before these scores
            // The reference point of the exponentials moves only when a picked score exceeds it by 5: sums stay below e^5 x K
            // and nothing is lost, the output is rescaled once or twice in a row's life.  The maximum of all the tile's scores
            // is cheaper than that of the picked ones (one instruction per score, not three) and says most times that no
            // row's point has to move.
            bool look = j < PAIRS;
            if (!look) {
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
                for (int c = 0; c < 2; ++c) {
                    uint32_t v[32];
                    ld32(t_s + c * 32, v);
                    ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float x, y;
                        unpair2(mul2(pair2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), scale2), x, y);
                        mx[(i >> 1) & 3] = fmaxf(mx[(i >> 1) & 3], fmaxf(x, y));
                    }
                }
                float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                if (!exchange(top)) { alive = false; break; }
                look = __any_sync(0xffffffffu, (cur.x | cur.y | cur.z | cur.w) != 0u && !(top <= m + 5.0f));
            }
            if (look) {
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
                for (int c = 0; c < 2; ++c) {
                    uint32_t v[32];
                    ld32(t_s + c * 32, v);
                    ld_wait();
                    const uint32_t bit = c == 0 ? (h ? cur.z : cur.x) : (h ? cur.w : cur.y);
#pragma unroll
                    for (int i = 0; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], bit & (1u << i) ? __uint_as_float(v[i]) * a.scale : -INFINITY);
                }
                float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                if (!exchange(mt)) { alive = false; break; }
                const bool move = mt > m + 5.0f || (m == -INFINITY && mt > -INFINITY);
                if (__any_sync(0xffffffffu, move)) {
                    const float mn = move ? mt : m;
                    const float f = m == -INFINITY ? 0.0f : __expf(m - mn);
                    const uint64_t f2 = pair2(f, f);
                    m = mn;
                    l2[0] = mul2(l2[0], f2);
                    l2[1] = mul2(l2[1], f2);
                    if constexpr (KEEP) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) o_sum[i] = mul2(o_sum[i], f2);
                    } else if (j >= PAIRS) {
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            float o[16];
                            uint32_t w[16];
                            tc_ld16(t_o + c * 16, o);
#pragma unroll
                            for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(o[i] * f);
                            st16(t_o + c * 16, w);
                        }
                    }
                }
            }
            const float mu = m == -INFINITY ? 0.0f : m;
            // (repeats are known per tile: inside a chunk, the choice cost the calls without any 1 %)
            auto chunks = [&](auto push, auto repeated) {
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    const uint32_t bit = (c < 2 ? (h ? cur.z : cur.x) : (h ? cur.w : cur.y)) >> (c & 1) * 16;
                    softmax_chunk<push.value, repeated.value>(t_s + c * 16, t_lead + c * 8, bit, a.scale, mu, count, to, l2);
                }
            };
            constexpr std::true_type yes;
            constexpr std::false_type no;
            if (half == 0) { if (repeats) chunks(yes, yes); else chunks(yes, no); }
            else if (repeats) chunks(no, yes);
            else chunks(no, no);
            st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(pready0 + 8 * pair);
        }
        const bool ran = n > pair;
        for (int i = 0; i < min(n, PAIRS) && alive; ++i) {                  // every product has been added, no panel is read any more
            alive = wait_warp(odone0 + 8 * i, 0, abort_flag, (8 << 8) | 6);
        }
        tc_fence_after();
        float o[32];
        if constexpr (KEEP) {
            if (ran && alive) add_output();
#pragma unroll
            for (int i = 0; i < 16; ++i) unpair2(o_sum[i], o[2 * i], o[2 * i + 1]);
        } else {
            uint32_t v[32];
            ld32(t_o, v);
            ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __uint_as_float(v[i]);
        }
        float l;
        {
            float x, y;
            unpair2(add2(l2[0], l2[1]), x, y);
            l = x + y;
        }
        // merge: each half leaves its sum in the operand panels, a second pair all its state
        float* merge = reinterpret_cast<float*>(smem);                   // [69][128], column r: conflict-free
        merge[(65 + pair * 2 + h) * T + r] = l;
        if (PAIRS > 1 && pair == 1) {
            if (h == 0) merge[64 * T + r] = ran ? m : -INFINITY;
            if (ran && alive) {
#pragma unroll
                for (int i = 0; i < 32; ++i) merge[(h * 32 + i) * T + r] = o[i];
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(256 * PAIRS) : "memory");
        if (pair == 0) {
            const float l0 = merge[65 * T + r] + merge[66 * T + r];
            const float m1 = PAIRS > 1 ? merge[64 * T + r] : -INFINITY, l1 = PAIRS > 1 ? merge[67 * T + r] + merge[68 * T + r] : 0.0f;
            const float mm = fmaxf(m, m1);
            const float f0 = m == -INFINITY ? 0.0f : __expf(m - mm), f1 = m1 == -INFINITY ? 0.0f : __expf(m1 - mm);
            const float sum = l0 * f0 + l1 * f1;
            const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;
            const float lse = sum > 0.0f ? mm + logf(sum) : 0.0f;
            // (no finite result can hide a sum that is not a number: with NaN scores only, the second pair's maximum stays
            // at -inf and its output is left out below)
            bool bad = sum != sum;
            const int col0 = half * 64 + h * 32, cols = min(32, a.Dv - col0);
            const int64_t orow = ((int64_t)bh * a.L + t) * a.Dv + col0;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const float o1 = m1 == -INFINITY ? 0.0f : merge[(h * 32 + i) * T + r] * f1;
                o[i] = (o[i] * f0 + o1) * inv;
                bad |= !(fabsf(o[i]) <= 3.4e38f);
            }
            if (live && alive && cols > 0) {
                if (cols == 32 && (a.Dv & 3) == 0) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        *reinterpret_cast<float4*>(a.out + orow + i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (i < cols) a.out[orow + i] = o[i];
                }
                if (a.out_cast) {
                    uint16_t* crow = static_cast<uint16_t*>(a.out_cast) + orow;
                    uint32_t w[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        if (a.out_cast_tag == CINN_BF16) {
                            const __nv_bfloat162 x = __floats2bfloat162_rn(o[2 * i], o[2 * i + 1]);
                            w[i] = *reinterpret_cast<const uint32_t*>(&x);
                        } else {
                            const __half2 x = __floats2half2_rn(o[2 * i], o[2 * i + 1]);
                            w[i] = *reinterpret_cast<const uint32_t*>(&x);
                        }
                    }
                    if (cols == 32 && (a.Dv & 7) == 0) {
#pragma unroll
                        for (int i = 0; i < 16; i += 4) *reinterpret_cast<uint4*>(crow + 2 * i) = make_uint4(w[i], w[i + 1], w[i + 2], w[i + 3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (i < cols) crow[i] = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
                    }
                }
            }
            if (live && bad) *a.flag = 1;
            if (h == 0) {
                s_lse[r] = lse;
                if (live && half == 0) a.lse[(int64_t)bh * a.L + t] = lse;
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(256 * PAIRS) : "memory");
        if (half == 0 && alive)
            by_slot<8 * PAIRS>(a.picks.rank + ((int64_t)b * a.L + q0) * a.K, a.attn + ((int64_t)bh * a.L + q0) * a.K, s_lse, min(T, a.L - q0), a.K,
                    a.scale, warp, lane);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        tc_dealloc(tmem, 256 * PAIRS);
    }
}

// ---------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------
// delta[row] = sum_d dO[row, d] * O[row, d]; one warp per row, bound by reading both
template <typename U>
__global__ void __launch_bounds__(256)
delta_kernel(const U* __restrict__ d_out, const float* __restrict__ out, float* __restrict__ delta, int64_t rows, int Dv) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    for (int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); w < rows; w += (int64_t)gridDim.x * 8) {
        float s = 0.0f;
        for (int d = lane; d < Dv; d += 32) s = fmaf(widen<U>(d_out[w * Dv + d]), out[w * Dv + d], s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) delta[w] = s;
    }
}

struct BwdArgs {
    Picks picks;
    const float* lse; const float* delta;
    float2* pd;                            // (B H, L, K) by rank: probability times count, and its score gradient
    void* dq; void* dk; void* dv;          // in `tag`'s type
    int* flag;
    int H, L, words, K, Dqk, Dv, BH, n_tiles, group, tag;
    float scale;
};

// 16 fp32 values of one row to `dst + col` (elements of `tag`'s type); the row has `width` columns
__device__ __forceinline__ void store_row16(void* dst, int64_t row, int col, int width, int tag, const float (&o)[16]) {
    if (tag == CINN_F32) {
        float* d = static_cast<float*>(dst) + row * width + col;
        if (col + 16 <= width && (width & 3) == 0) {
#pragma unroll
            for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(d + i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
        } else {
            for (int i = 0; i < 16; ++i)
                if (col + i < width) d[i] = o[i];
        }
    } else {
        uint16_t* d = static_cast<uint16_t*>(dst) + row * width + col;
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (tag == CINN_BF16) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(o[2 * i], o[2 * i + 1]);
                w[i] = *reinterpret_cast<const uint32_t*>(&h);
            } else {
                const __half2 h = __floats2half2_rn(o[2 * i], o[2 * i + 1]);
                w[i] = *reinterpret_cast<const uint32_t*>(&h);
            }
        }
        if (col + 16 <= width && (width & 7) == 0) {
            *reinterpret_cast<uint4*>(d) = make_uint4(w[0], w[1], w[2], w[3]);
            *reinterpret_cast<uint4*>(d + 8) = make_uint4(w[4], w[5], w[6], w[7]);
        } else {
            for (int i = 0; i < 16; ++i)
                if (col + i < width) d[i] = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
        }
    }
}

// fp32 gradients leave tensor memory every few hundred steps and are added up in global memory, rounded to nearest: the tensor
// core truncates its running sums at every step, which over thousands of queries would show in fp32.  A warpgroup takes
// pieces of 16 columns x 128 rows: registers, a slot of 8 KiB (64-byte swizzle), and a TMA store (the first time) or reduce;
// nobody reads the old values back.  (As loads, adds and stores of every thread's own row a flush took 20 000 cycles.)  Only
// this block touches these rows and a flush waits for the one before, so the sums are the same on every run.
constexpr int SLOT_COLS = 16, SLOT_BYTES = T * SLOT_COLS * 4;

// where(c): the map and first column of piece c.  All four warps of a warpgroup call it; slots: this warpgroup's.  False: given up.
template <int SLOTS, typename WHERE>
__device__ __forceinline__ bool flush_tma(uint32_t taddr, WarpgroupBarrier& all, int code, int c0, int c1, int step, uint32_t slots, int row, int plane, bool first,
                                          bool live, bool& bad, WHERE&& where) {
    const int quarter = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31, r = quarter * 32 + lane;
    const bool elected = quarter == 0 && lane == 0;
    if (elected && !first) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");      // the flush before has been added
    int n = 0;
#pragma unroll 1
    for (int c = c0; c < c1; c += step, ++n) {
        float o[16];
        tc_ld16(taddr + c * 16, o);
        const uint32_t slot = slots + (n % SLOTS) * SLOT_BYTES;
        if (elected && n >= SLOTS) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(SLOTS - 1) : "memory");
        if (!all.sync(code)) return false;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            bad |= live && !(fabsf(o[4 * i]) <= 3.4e38f && fabsf(o[4 * i + 1]) <= 3.4e38f && fabsf(o[4 * i + 2]) <= 3.4e38f &&
                             fabsf(o[4 * i + 3]) <= 3.4e38f);
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(slot + r * 64 + ((i ^ ((r >> 1) & 3)) << 4)), "f"(o[4 * i]),
                         "f"(o[4 * i + 1]), "f"(o[4 * i + 2]), "f"(o[4 * i + 3]) : "memory");
        }
        fence_async_smem();
        if (!all.sync(code)) return false;
        if (elected) {
            int x;
            const CUtensorMap* m = where(c, x);
            if (m) {
                if (first) tma_store_3d(m, slot, x, row, plane);
                else tma_add_3d(m, slot, x, row, plane);
            }
            tma_store_commit();
        }
    }
    if (elected) tma_store_wait_read();                    // the slots are free again
    return all.sync(code);
}

// Shared memory of the query pass: queries and output gradients resident, a ring of key / value panels.  Of three parts
// the smallest, which meets only the leading part of k and v, comes through the ring too: with everything resident two
// panels were left, and the copies' latency bounded the pass (1.40 ms at 32 x 8 x 1024 queries of 192 in fp32).
template <int NS, int ND, int NV> struct QPassShape {
    static constexpr int KEPT = NS > 1 ? 2 : 1;            // resident parts
    static constexpr int FIXED = KEPT * (ND + NV);
    static constexpr int RING = FIXED > 7 ? 13 - FIXED : 6;
    static constexpr int SLOT_OFF = (FIXED + RING) * PANEL;        // one slot per warpgroup
    static constexpr int BAR_OFF = SLOT_OFF + 2 * SLOT_BYTES;
    static constexpr int BYTES = BAR_OFF + 256 + 1024;
};

constexpr int QUERY_THREADS = 10 * 32;     // two vector warpgroups, TMA warp, MMA warp

// Query pass: one CTA per 128 queries of a head, over their key tiles.  S = q k^T and dP = dO v^T in tensor memory; a
// thread (a query, half of the tile's keys) turns them into p = exp(scale S - lse) and dS = p (dP - delta) scale, leaves
// both by rank for the key pass, and writes dS back as an A operand for dq += dS k.  (Collecting a row's values in shared
// memory to store them together took twice as long as these scattered stores.)  All of tensor memory: 128 columns of
// S under the second and third parts of dS, 128 of dP, 64 of dS's leading parts, 192 of dq.
template <int NS, int ND, int NV>
__global__ void __launch_bounds__(QUERY_THREADS, 1)
attn_bwd_query_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmG,
                      const __grid_constant__ CUtensorMap tmDQ, const BwdArgs a) {
    pdl_wait();
    using S = QPassShape<NS, ND, NV>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sq = smem_u32(smem), sg = sq + S::KEPT * ND * PANEL, ring = sq + S::FIXED * PANEL;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::BAR_OFF);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + S::RING), qfull = smem_u32(bars + 2 * S::RING);
    const uint32_t sfull = qfull + 8, dsready = qfull + 16, done = qfull + 24, taken = qfull + 32;
    constexpr int EVERY = 1;                              // fp32 gradients: tiles between two flushes
    const uint32_t group0 = qfull + 40;                   // the two warpgroups' own barriers
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S::RING + 7);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int qt, bh;
    tile_of_block(a.n_tiles, a.BH, a.group, qt, bh);
    const int q0 = qt * T, n = qt + 1;
    const bool flush = NS > 1 && a.tag == CINN_F32;
    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < S::RING; ++i) { mbar_init(full0 + 8 * i, 1); mbar_init(empty0 + 8 * i, 1); }
        mbar_init(qfull, 1); mbar_init(sfull, 1); mbar_init(dsready, 8); mbar_init(done, 1); mbar_init(taken, 8);
        for (int i = 0; i < 2; ++i) mbar_init(group0 + 8 * i, 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        tc_alloc(smem_u32(tmem_slot), 512);
        pdl_trigger();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot, t_s = tmem, t_dp = tmem + 128, t_lead = tmem + 256, t_dq = tmem + 320;

    if (warp == 8) {
        if (lane == 0) {
            mbar_expect_tx(qfull, S::FIXED * PANEL);
            for (int p = 0; p < S::KEPT; ++p) {
                for (int c = 0; c < ND; ++c) tma_load_3d(&tmQ, qfull, sq + (p * ND + c) * PANEL, c * 64, q0, p * a.BH + bh);
                for (int c = 0; c < NV; ++c) tma_load_3d(&tmG, qfull, sg + (p * NV + c) * PANEL, c * 64, q0, p * a.BH + bh);
            }
            uint32_t it = 0;
            bool alive = true;
            auto fetch = [&](const CUtensorMap* m, int x, int y, int z) {
                const uint32_t s = it % S::RING, ph = (it / S::RING) & 1;
                if (!alive || !mbar_wait_bounded(empty0 + 8 * s, ph ^ 1, abort_flag, (9 << 8) | 1, &g_attn_status)) { alive = false; return; }
                mbar_expect_tx(full0 + 8 * s, PANEL);
                tma_load_3d(m, full0 + 8 * s, ring + s * PANEL, x, y, z);
                ++it;
            };
            for (int j = 0; j < n && alive; ++j) {
                if constexpr (NS > 1)
                    for (int c = 0; c < ND; ++c) {
                        for (int p = NS - 1; p >= 0; --p) fetch(&tmK, c * 64, j * T, p * a.BH + bh);
                        fetch(&tmQ, c * 64, q0, 2 * a.BH + bh);
                    }
                for (int c = 0; c < ND; ++c) fetch(&tmK, c * 64, j * T, bh);
                for (int c = 0; c < NV; ++c) {
                    for (int p = NS - 1; p >= 0; --p) fetch(&tmV, c * 64, j * T, p * a.BH + bh);
                    if constexpr (NS > 1) fetch(&tmG, c * 64, q0, 2 * a.BH + bh);
                }
                for (int c = 0; c < ND; ++c)
                    for (int p = NS - 1; p >= 0; --p) fetch(&tmK, c * 64, j * T, p * a.BH + bh);
            }
            if (!alive) {                                 // abandoned: let the copies in flight land
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000LL) { }
            }
        }
    } else if (warp == 9) {
        if (wait_warp(qfull, 0, abort_flag, (9 << 8) | 2)) {
            constexpr uint32_t id_s = make_idesc_f16(true, T, T), id_o = make_idesc_f16(true, T, 64, false, true);
            PanelRing<S::RING> panels(full0, empty0, ring, abort_flag, (9 << 8) | 3);
            const bool& alive = panels.alive;
            // parts [x_lo, x_hi] of a resident panel (parts `stride` panels apart) against the ring's next panel; with
            // `small`, the panel after it holds the third part, which goes first
            auto product = [&](uint32_t d, uint32_t fixed, int stride, int x_hi, int x_lo, bool small, bool& first) {
                uint32_t bp, ap, slot, small_slot;
                if (!panels.next(bp, slot)) return;
                const uint32_t bd = panel_desc(bp);
                if (small) {
                    if (!panels.next(ap, small_slot)) return;
                    mma_panels(d, panel_desc(ap), bd, id_s, first);
                    first = false;
                    panels.release(small_slot);
                }
                uint32_t ad = panel_desc(fixed) + x_hi * stride * (PANEL >> 4);
                for (int x = x_hi; x >= x_lo; --x) {
                    mma_panels(d, ad, bd, id_s, first);
                    first = false;
                    ad -= stride * (PANEL >> 4);
                }
                panels.release(slot);
            };
            for (int j = 0; j < n && alive; ++j) {
                // (S overwrites the parts of dS that dq of tile j - 1 reads: issued after it, executed after it)
                bool first = true;
                if constexpr (NS > 1)
                    for (int c = 0; c < ND && alive; ++c) {
                        product(t_s, sq + c * PANEL, ND, 0, 0, false, first);                  // third part of k
                        if (alive) product(t_s, sq + c * PANEL, ND, 1, 0, false, first);       // second
                        if (alive) product(t_s, sq + c * PANEL, ND, 1, 1, true, first);        // leading, without q's leading part
                    }
                for (int c = 0; c < ND && alive; ++c) product(t_s, sq + c * PANEL, ND, 0, 0, false, first);
                first = true;
                for (int c = 0; c < NV && alive; ++c) {
                    if constexpr (NS > 1) {
                        product(t_dp, sg + c * PANEL, NV, 0, 0, false, first);
                        if (alive) product(t_dp, sg + c * PANEL, NV, 1, 0, false, first);
                        if (alive) product(t_dp, sg + c * PANEL, NV, 1, 0, true, first);
                    } else {
                        product(t_dp, sg + c * PANEL, NV, 0, 0, false, first);
                    }
                }
                if (!alive) break;
                tc_commit(sfull);
                if (!wait_warp(dsready, j & 1, abort_flag, (9 << 8) | 4)) break;
                const bool fresh = j == 0 || (flush && j % EVERY == 0);
                if (fresh && j > 0 && !wait_warp(taken, (j / EVERY - 1) & 1, abort_flag, (9 << 8) | 7)) break;
                tc_fence_after();
                for (int c = 0; c < ND && alive; ++c) {
                    first = fresh;
                    for (int p = NS - 1; p >= 0 && alive; --p) {
                        uint32_t kp, slot;
                        if (!panels.next(kp, slot)) break;
                        const uint32_t kd = panel_desc(kp);
                        const uint32_t d = t_dq + c * 64;
                        if (p == 0) { mma_part_at<2>(d, t_s, t_lead, kd, id_o, first); first = false; }
                        if (p <= 1) { mma_part_at<1>(d, t_s, t_lead, kd, id_o, first); first = false; }
                        mma_part_at<0>(d, t_s, t_lead, kd, id_o, first);
                        first = false;
                        panels.release(slot);
                    }
                }
                if (alive && (j + 1 == n || (flush && (j + 1) % EVERY == 0))) tc_commit(done);
            }
        }
    } else {
        const int h = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const int t = q0 + r, b = bh / a.H;
        const bool live = t < a.L;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const int64_t qrow = (int64_t)b * a.L + min(t, a.L - 1), row = (int64_t)bh * a.L + min(t, a.L - 1);
        const uint2* bits = reinterpret_cast<const uint2*>(a.picks.bits + qrow * a.words) + h;       // 64 keys of every tile
        const uint16_t* before = a.picks.before + qrow * a.words + h * 2;
        const bool repeats = a.picks.repeats[b * a.n_tiles + qt] != 0;
        const uint8_t* count = a.picks.count + qrow * a.K;
        const float lse = a.lse[row], delta = a.delta[row];
        float2* pdrow = a.pd + row * a.K;
        bool alive = true;
        uint2 mine = live ? __ldg(bits) : make_uint2(0u, 0u);
        uint32_t rank = __ldg(before);
        uint32_t rounds = 0;                              // sums of dq taken out so far
        bool bad = false;
        const uint32_t slots = smem_u32(smem + S::SLOT_OFF) + h * SLOT_BYTES;
        WarpgroupBarrier group{group0 + 8 * h, 0, abort_flag};
        auto take = [&] {
            if (!wait_warp(done, rounds & 1, abort_flag, (9 << 8) | 6)) return false;
            tc_fence_after();
            if (!flush_tma<1>(t_dq + lanes, group, (9 << 8) | 8, h, ND * 4, 2, slots, q0, bh, rounds == 0, live, bad,
                                        [&](int c, int& x) { x = c * 16; return x < a.Dqk ? &tmDQ : nullptr; })) return false;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(taken);
            ++rounds;
            return true;
        };
        for (int j = 0; j < n; ++j) {
            if (flush && j > 0 && j % EVERY == 0 && !take()) { alive = false; break; }
            const uint2 cur = mine;
            uint32_t at0 = rank;
            if (j + 1 < n) {
                mine = live ? __ldg(bits + (j + 1) * 2) : make_uint2(0u, 0u);
                rank = __ldg(before + (j + 1) * 4);
            }
            if (!wait_warp(sfull, j & 1, abort_flag, (9 << 8) | 5)) { alive = false; break; }
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                uint32_t sv[32], dv[32];
                ld32(t_s + lanes + h * 64 + c * 32, sv);
                ld32(t_dp + lanes + h * 64 + c * 32, dv);
                ld_wait();
                const uint32_t bit = c == 0 ? cur.x : cur.y;
                float p[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) p[i] = exp_fast(bit & (1u << i) ? fmaf(__uint_as_float(sv[i]), a.scale, -lse) : -INFINITY);
                if (repeats) {                            // a key picked several times counts as often
                    const uint8_t* cnt = count + at0;
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (bit & (1u << i)) p[i] *= (float)*cnt++;
                }
                // (one 8-byte store for both: the store unit takes a line per lane and instruction, and that bounds this phase)
                float2* pd = pdrow + at0;
                uint32_t at = 0;
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const uint32_t pick = bit & (1u << i);
                    const float ds = p[i] * (__uint_as_float(dv[i]) - delta) * a.scale;
                    store2_if(pd + at, p[i], ds, pick);
                    p[i] = pick ? ds : 0.0f;
                    at += (bit >> i) & 1u;
                }
                at0 += at;
                store_parts16(t_s + lanes + h * 64 + c * 32, t_lead + lanes + h * 32 + c * 16, p);
                store_parts16(t_s + lanes + h * 64 + c * 32 + 16, t_lead + lanes + h * 32 + c * 16 + 8, p + 16);
            }
            st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(dsready);
        }
        if (alive && flush) {
            take();
        } else if (alive && wait_warp(done, 0, abort_flag, (9 << 8) | 6)) {
            tc_fence_after();
#pragma unroll 1
            for (int c = h; c < ND * 4; c += 2) {
                float o[16];
                tc_ld16(t_dq + lanes + c * 16, o);
#pragma unroll
                for (int i = 0; i < 16; ++i) bad |= !(fabsf(o[i]) <= 3.4e38f);
                if (live && c * 16 < a.Dqk) store_row16(a.dq, row, c * 16, a.Dqk, a.tag, o);
            }
        }
        if (live && bad) *a.flag = 1;
        if (quarter == 0 && lane == 0) tma_store_wait_all();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        tc_dealloc(tmem, 512);
    }
}

// Shared memory of the key pass: a ring of stages, each 32 queries of every panel of q and dO.
template <int NS, int ND, int NV> struct KPassShape {
    static constexpr int SUB = 32 * 128;                   // 32 rows of a 64-column panel
    static constexpr int PANELS = NS * (ND + NV), STAGE = PANELS * SUB;
    static constexpr int STAGES = (12 * PANEL) / STAGE < 8 ? (12 * PANEL) / STAGE : 8;
    static constexpr int SLOT_OFF = STAGES * STAGE;
    static constexpr int BAR_OFF = SLOT_OFF + 4 * SLOT_BYTES;
    static constexpr int BYTES = BAR_OFF + 256 + 1024;
};

// Key pass: one CTA per 128 keys of a head, over the queries from the keys' own tile on, 32 at a time.  A thread owns a
// key; for a warp's 32 keys the bits of a query are one word, and the ranks of the keys it picked are consecutive, so
// that what the query pass left is read in short contiguous pieces, p and dS together.  Two warpgroups take half of a
// chunk's queries each and write them as A operands (48 columns for p, 48 for dS), two others the next chunk's; the tensor
// core adds dv += P^T dO, dk += dS^T q.  (p and dS apart, a warpgroup reading one of them for all 32 queries, and the flush
// before the gather: 859 us at 32 x 8 x 1024 queries of 192 in fp32, where this takes 716.)
constexpr int KEY_THREADS = 18 * 32;       // four producing warpgroups, TMA warp, MMA warp

template <int NS, int ND, int NV>
__global__ void __launch_bounds__(KEY_THREADS, 1)
attn_bwd_key_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmG,
                    const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDV, const BwdArgs a) {
    pdl_wait();
    using S = KPassShape<NS, ND, NV>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t ring = smem_u32(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::BAR_OFF);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + S::STAGES);
    const uint32_t ready0 = smem_u32(bars + 2 * S::STAGES), free0 = ready0 + 16;        // two each
    const uint32_t done = ready0 + 32, taken = ready0 + 40;
    constexpr int EVERY = 4;                               // fp32 gradients: chunks between two flushes
    const bool flush = NS > 1 && a.tag == CINN_F32;
    const uint32_t group0 = ready0 + 48;                   // the four warpgroups' own barriers
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S::STAGES + 10);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int kt, bh;
    tile_of_block(a.n_tiles, a.BH, a.group, kt, bh);
    kt = a.n_tiles - 1 - kt;                               // the first keys have the most queries
    const int k0 = kt * T, n = (a.n_tiles - kt) * 4;       // chunks of 32 queries
    if (tid == 0) {
        *abort_flag = 0;
        for (int i = 0; i < S::STAGES; ++i) { mbar_init(full0 + 8 * i, 1); mbar_init(empty0 + 8 * i, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(ready0 + 8 * i, 8); mbar_init(free0 + 8 * i, 1); }
        mbar_init(done, 1); mbar_init(taken, 16);
        for (int i = 0; i < 4; ++i) mbar_init(group0 + 8 * i, 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 17) {
        tc_alloc(smem_u32(tmem_slot), 512);
        pdl_trigger();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // columns: dk | dv | [operand p, dS][buffer] 48
    const uint32_t tmem = *tmem_slot, t_dk = tmem, t_dv = tmem + ND * 64, t_a = tmem + 320;

    if (warp == 16) {
        if (lane == 0) {
            bool alive = true;
            for (int i = 0; i < n && alive; ++i) {
                const uint32_t s = i % S::STAGES, ph = (i / S::STAGES) & 1;
                if (!mbar_wait_bounded(empty0 + 8 * s, ph ^ 1, abort_flag, (10 << 8) | 1, &g_attn_status)) { alive = false; break; }
                mbar_expect_tx(full0 + 8 * s, S::STAGE);
                uint32_t dst = ring + s * S::STAGE;
                const int y = k0 + i * 32;
                for (int p = 0; p < NS; ++p) {
                    for (int c = 0; c < NV; ++c, dst += S::SUB) tma_load_3d(&tmG, full0 + 8 * s, dst, c * 64, y, p * a.BH + bh);
                    for (int c = 0; c < ND; ++c, dst += S::SUB) tma_load_3d(&tmQ, full0 + 8 * s, dst, c * 64, y, p * a.BH + bh);
                }
            }
            if (!alive) {                                 // abandoned: let the copies in flight land
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000LL) { }
            }
        }
    } else if (warp == 17) {
        constexpr uint32_t id = make_idesc_f16(true, T, 64, false, true);
        bool alive = true;
        uint32_t s = 0, phase = 0;
        for (int i = 0; i < n; ++i) {
            const uint32_t buf = i & 1, stage = ring + s * S::STAGE, empty = empty0 + 8 * s;
            if (!wait_warp(full0 + 8 * s, phase, abort_flag, (10 << 8) | 2)) { alive = false; break; }
            const bool fresh = i == 0 || (flush && i % EVERY == 0);
            if (fresh && i > 0 && !wait_warp(taken, (i / EVERY - 1) & 1, abort_flag, (10 << 8) | 6)) { alive = false; break; }
            if (!wait_warp(ready0 + 8 * buf, (i >> 1) & 1, abort_flag, (10 << 8) | 3)) { alive = false; break; }
            tc_fence_after();
            if (++s == (uint32_t)S::STAGES) { s = 0; phase ^= 1u; }
#pragma unroll
            for (int op = 0; op < 2; ++op) {               // dv from p and dO, dk from dS and q
                const uint32_t at = t_a + (op * 2 + buf) * 48;
                for (int c = 0; c < (op ? ND : NV); ++c) {
                    const uint32_t d = (op ? t_dk : t_dv) + c * 64;
                    bool first = fresh;
#pragma unroll
                    for (int p = NS - 1; p >= 0; --p) {
                        const uint32_t bd = panel_desc(stage + (p * (ND + NV) + (op ? NV : 0) + c) * S::SUB);
                        if (p == 0) { mma_part_at<2, 2>(d, at, at + 32, bd, id, first); first = false; }
                        if (p <= 1) { mma_part_at<1, 2>(d, at, at + 32, bd, id, first); first = false; }
                        mma_part_at<0, 2>(d, at, at + 32, bd, id, first);
                        first = false;
                    }
                }
            }
            tc_commit(free0 + 8 * buf);
            tc_commit(empty);
            if (i + 1 == n || (flush && (i + 1) % EVERY == 0)) tc_commit(done);
        }
    } else {
        const int half = (warp >> 2) & 1, buf = warp >> 3, quarter = warp & 3, r = quarter * 32 + lane;
        const int s = k0 + r, b = bh / a.H;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const int word = (k0 >> 5) + quarter;
        const uint32_t* bits = a.picks.bits + ((int64_t)b * a.L) * a.words + word;
        const uint16_t* before = a.picks.before + ((int64_t)b * a.L) * a.words + word;
        const float2* src = a.pd + (int64_t)bh * a.L * a.K;
        const uint32_t below = (1u << lane) - 1u;
        bool alive = true;
        // this lane's query of the next chunk: its word for the warp's keys, and where that word's picks begin
        auto fetch = [&](int i, uint32_t& w, uint32_t& base) {
            const int t = k0 + i * 32 + lane, tc = min(t, a.L - 1);
            w = t < a.L ? __ldg(bits + (int64_t)tc * a.words) : 0u;
            base = (uint32_t)tc * a.K + __ldg(before + (int64_t)tc * a.words);
        };
        const int64_t row = (int64_t)bh * a.L + min(s, a.L - 1);
        uint32_t rounds = 0;                               // sums taken out so far
        WarpgroupBarrier group{group0 + 8 * (warp >> 2), 0, abort_flag};
        bool bad = false;
        auto take = [&] {
            if (!wait_warp(done, rounds & 1, abort_flag, (10 << 8) | 5)) return false;
            tc_fence_after();
            const int wg = warp >> 2;
            const bool ok = flush_tma<1>(t_dk + lanes, group, (10 << 8) | 7, wg, (ND + NV) * 4, 4,
                                                   smem_u32(smem + S::SLOT_OFF) + wg * SLOT_BYTES, k0, bh, rounds == 0, s < a.L, bad,
                                                   [&](int c, int& x) -> const CUtensorMap* {                // dk, then dv
                const bool is_v = c >= ND * 4;
                x = (is_v ? c - ND * 4 : c) * 16;
                if (x >= (is_v ? a.Dv : a.Dqk)) return nullptr;
                return is_v ? &tmDV : &tmDK;
            });
            if (!ok) return false;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(taken);
            ++rounds;
            return true;
        };
        uint32_t w_next, base_next;
        fetch(buf, w_next, base_next);
        for (int i = buf; i < n; i += 2) {
            const uint32_t w = w_next, base = base_next;
            if (i + 2 < n) fetch(i + 2, w_next, base_next);
            float vp[16], vd[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                const uint32_t wu = __shfl_sync(0xffffffffu, w, half * 16 + u);
                const uint32_t at = __shfl_sync(0xffffffffu, base, half * 16 + u) + __popc(wu & below);
                const float2 x = __ldg(src + min(at, (uint32_t)a.L * a.K - 1u));      // a lane that was not picked reads its neighbour's
                vp[u] = wu >> lane & 1u ? x.x : 0.0f;
                vd[u] = wu >> lane & 1u ? x.y : 0.0f;
            }
            // (with this chunk's values already here, the flush costs the tensor core its own time only)
            if (flush && i >= EVERY && i % EVERY == buf && !take()) { alive = false; break; }
            if (!wait_warp(free0 + 8 * buf, ((i >> 1) & 1) ^ 1, abort_flag, (10 << 8) | 4)) { alive = false; break; }
            tc_fence_after();
            store_parts16(t_a + lanes + buf * 48 + half * 16, t_a + lanes + buf * 48 + 32 + half * 8, vp);
            store_parts16(t_a + lanes + (2 + buf) * 48 + half * 16, t_a + lanes + (2 + buf) * 48 + 32 + half * 8, vd);
            st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready0 + 8 * buf);
        }
        if (alive && flush) {
            take();
        } else if (alive && wait_warp(done, 0, abort_flag, (10 << 8) | 5)) {
            tc_fence_after();
#pragma unroll 1
            for (int c = warp >> 2; c < (ND + NV) * 4; c += 4) {       // 16-column pieces of dk, then dv
                float o[16];
                tc_ld16(t_dk + lanes + c * 16, o);
#pragma unroll
                for (int i = 0; i < 16; ++i) bad |= !(fabsf(o[i]) <= 3.4e38f);
                const bool is_v = c >= ND * 4;
                const int col = (is_v ? c - ND * 4 : c) * 16, width = is_v ? a.Dv : a.Dqk;
                if (s < a.L && col < width) store_row16(is_v ? a.dv : a.dk, row, col, width, a.tag, o);
            }
        }
        if (s < a.L && bad) *a.flag = 1;
        if (quarter == 0 && lane == 0) tma_store_wait_all();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 17) {
        tc_fence_after();
        tc_dealloc(tmem, 512);
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static inline int64_t up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

// One call's shapes and where its scratch lies.
struct Plan {
    int64_t B, H, L, K, Dqk, Dv, BH, Lp;
    int dtype, ns, nd, dp, nv;             // parts; panels, padded width of q and k; 64-column panels of v
    bool direct;                           // bf16 rows TMA can read as they are: no copies
    int64_t bits_off, rank_off, count_off, before_off, flag_off, q_off, k_off, v_off, g_off, delta_off, pd_off, grads_off, bytes;
};

static Plan make_plan(int64_t B, int64_t H, int64_t L, int64_t K, int64_t Dqk, int64_t Dv, int dtype, bool backward) {
    Plan p{};
    p.B = B; p.H = H; p.L = L; p.K = K; p.Dqk = Dqk; p.Dv = Dv; p.BH = B * H; p.Lp = up(L, T);
    p.dtype = dtype;
    p.ns = dtype == CINN_BF16 ? 1 : PARTS;
    p.nd = (int)((Dqk + 63) / 64); p.dp = p.nd * 64; p.nv = (int)((Dv + 63) / 64);
    p.direct = dtype == CINN_BF16 && Dqk % 8 == 0 && Dv % 8 == 0;
    int64_t off = 0;
    auto take = [&](int64_t bytes) { const int64_t o = off; off += up(bytes, 256); return o; };
    p.flag_off = take(4 * (1 + B * (p.Lp / T)));          // the flag, then the tiles' `repeats`
    p.bits_off = take(B * L * p.Lp / 8);
    p.rank_off = take(B * L * K * 2);
    p.count_off = take(B * L * K);
    p.before_off = take(B * L * p.Lp / 32 * 2);
    if (backward) {
        p.delta_off = take(p.BH * L * 4);
        p.pd_off = take(p.BH * L * K * 8);
        if (!p.direct) p.g_off = take(p.ns * p.BH * L * p.nv * 64 * 2);
        // fp32 gradients for the fallback, where the caller's are not
        if (dtype != CINN_F32) p.grads_off = take(p.BH * L * (2 * Dqk + Dv) * 4);
    }
    if (!p.direct) {
        p.q_off = take(p.ns * p.BH * L * p.dp * 2);
        p.k_off = take(p.ns * p.BH * L * p.dp * 2);
        p.v_off = take(p.ns * p.BH * L * p.nv * 64 * 2);
    }
    p.bytes = off;
    return p;
}

// Whether the dense tiles are worth it: their time (the causal half of the tiles is visited, a constant number of cycles
// each that grows with the widths, and every query tile costs its start and its probabilities; what was picked and the parts come
// first) against the gathers' (K rows of Dqk + Dv elements per query and a constant per row).  The tiles take the larger of their number over
// the SMs and of the longest query tile's chain: with the sum of both, or the first alone, the estimate was 11 % off on average, with the
// larger 5 (backward).  Fitted to 420 calls, B = 1 ... 32, L = 256 ... 4052, K = 32 ... 256, widths 64 ... 192, bf16 and fp32.  On 400 others the way
// that is taken costs more than the faster one would by 0.1 (forward) and 0.2 % (backward) in bf16, 0.2 and 0.2 in fp32, at worst 1.17 times;
// with constants of a slower forward, fewer lengths and no chain by 7, 2, 3.4 and 4.4, at worst 2.5.  Gathers against tiles:
// 16 x 4 x 2286 queries, 64 picks of 64 / 128 in bf16 838 and 403 us, 4 x 8 x 3965,
// 64 of 192 / 128 861 and 581; backward 4 x 4 x 2033, 64 of 128 / 128 in fp32 549 and 428, 1 x 8 x 1965, 32 of 128 / 64 in bf16 131 and 176.
static std::atomic<int> g_mode{-1};         // -1: by the estimate; 0 / 1: never / wherever the tiles can (tests, measurements)
int set_mode(int mode) { return g_mode.exchange(mode); }

static bool dense_pays(const Plan& p, bool backward) {
    const int mode = g_mode.load(std::memory_order_relaxed);
    if (mode >= 0) return mode != 0;
    const double tiles = 0.5 * (double)(p.Lp / T) * (double)(p.Lp / T + 1) * (double)p.BH, q_tiles = (double)(p.Lp / T) * (double)p.BH;
    const bool parts = p.ns > 1, wide = p.dtype == CINN_F32;
    const double queries = (double)p.BH * p.L, row = (double)(p.Dqk + p.Dv), widths = p.dp + 64.0 * p.nv;
    const double gathered = queries * p.K * row * (wide ? 4 : 2), split = parts ? queries * (row + p.Dqk) * (wide ? 10 : 8) / 6.2e6 : 0.0;
    const double picked = 5.5e-6 * p.B * p.L * p.K;
    // cycles of a tile, how much of the longest query tile's chain counts, cycles of a query tile, microseconds before the tiles
    double tile, chain, query_tile, first, gather_us;
    if (!backward) {
        tile = parts ? 3740.0 + 34.2 * p.dp : 3610.0 + 4.28 * p.dp;
        chain = parts ? 0.81 : 0.76;
        query_tile = parts ? 3850.0 + 67.0 * p.K : 4900.0 + 50.1 * p.K;
        first = parts ? 17.7 + 1.75 * picked + 1.80 * split : 20.6 + 3.01 * picked;
        gather_us = wide ? 9.8 + gathered / 14.95e6 + queries * p.K / 43.8e3 : 12.1 + gathered / 10.15e6 + queries * p.K / 26.6e3;
    } else {
        tile = parts ? 9190.0 + 126.6 * widths : 9510.0 + 39.2 * widths;
        chain = parts ? 0.905 : 0.814;
        query_tile = parts ? 112.0 * p.K : 15160.0 + 117.6 * p.K;
        first = parts ? 26.8 + 0.84 * picked + 2.93 * split : 24.9 + 0.46 * picked;
        gather_us = wide ? 28.6 + gathered / 4.40e6 + queries * p.K / 76.2e3 : 42.6 + gathered / 2.76e6 + queries * p.K / 23.5e3;
    }
    const double ctas = backward ? 1.0 : (double)p.nv;      // a forward CTA computes 64 columns of the output
    const double all = ctas * tiles * tile / 148.0, longest = chain * (double)(p.Lp / T) * tile;
    double cycles = (all > longest ? all : longest) + ctas * q_tiles * query_tile / 148.0;
    if (!backward) {
        // With few queries a forward is one of them after the other: a query's picks on the gathers' side, and on the tiles' side, with CTAs for less
        // than half the SMs, the longest chain and its query tile.  Fitted to 280 calls of one sequence, 1 ... 8 heads, L = 256 ... 640, K = 32 ... 256: the way
        // taken costs 0.6 % more than the faster one, at worst 1.14 times (without this 5.8 %, 1.9 times); on 250 others of every size 0.65 %, 1.19 times
        // (0.86 %, 1.43).  us, gathers and tiles: 2 x 313 queries, 256 picks of 192 / 128 in fp32 101 and 53, 4 x 313, 128 picks 52 and 40, in bf16 39
        // and 29; 1 x 512, 128 picks of 192 / 64 39 and 46.
        const double one_query = 6.0 + p.K * row * (wide ? 4 : 2) / 4100.0 + (wide ? 0.0 : 0.055 * p.K) + gathered / (wide ? 14.95e6 : 10.15e6);
        if (one_query > gather_us) gather_us = one_query;
        if (ctas * q_tiles < 74.0)
            cycles = parts ? 0.664 * (double)(p.Lp / T) * tile + 1200.0 + 191.0 * p.K : 0.515 * (double)(p.Lp / T) * tile - 3980.0 + 117.0 * p.K;
        if (cycles < 0.0) cycles = 0.0;
    }
    return first + cycles / 1900.0 < gather_us;
}

static bool supported(int64_t B, int64_t H, int64_t L, int64_t K, int64_t Dqk, int64_t Dv) {
    return B * H * L > 0 && K >= 1 && K <= MAX_SLOTS && Dqk <= 192 && Dv <= 128 && L <= 12000 && B * H <= 65535 && B * H * L < (1LL << 31) / 4;
}

// a tenth of the memory: what a call may add to its tensors for the sake of speed
constexpr int64_t MAX_SCRATCH_BYTES = 16LL << 30;
static int64_t scratch_bytes(const Plan& p, bool backward) { return p.bytes <= MAX_SCRATCH_BYTES && dense_pays(p, backward) ? p.bytes : 0; }

static Picks picks_of(const Plan& p, const uint8_t* ws) {
    return {reinterpret_cast<const uint32_t*>(ws + p.bits_off), reinterpret_cast<const uint16_t*>(ws + p.rank_off), ws + p.count_off,
            reinterpret_cast<const uint16_t*>(ws + p.before_off), reinterpret_cast<const int*>(ws + p.flag_off) + 1};
}

// clears the flag and finds out what was picked
static int make_picks(const Plan& p, const int64_t* idx, uint8_t* ws, cudaStream_t st) {
    CINN_CHECK_CUDA(cudaMemsetAsync(ws + p.flag_off, 0, 4 * (1 + p.B * (p.Lp / T)), st));
    const int words = (int)(p.Lp / 32), warps = 4;
    const size_t smem = (size_t)warps * (2 * words + p.K) * 4;
    const int64_t rows = p.B * p.L;
    const int64_t want = (rows + warps - 1) / warps, cap = (int64_t)sm_count() * 16;
    const unsigned grid = (unsigned)(want < cap ? want : cap);
    int* flag = reinterpret_cast<int*>(ws + p.flag_off);
    launch_dependent(picks_kernel, dim3(grid), dim3(32 * warps), smem, st, idx, reinterpret_cast<uint32_t*>(ws + p.bits_off),
                                                 reinterpret_cast<uint16_t*>(ws + p.rank_off), ws + p.count_off,
                                                 reinterpret_cast<uint16_t*>(ws + p.before_off), flag + 1, flag, rows,
                                                 (int)p.L, words, (int)p.K, warps);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

static int split_parts(const SplitJobs& jobs, int dtype, cudaStream_t st) {
    const unsigned grid = (unsigned)sm_count() * 16;
    switch (dtype) {
        case CINN_F32: launch_dependent(split_parts_kernel<float, 3>, dim3(grid), dim3(256), 0, st, jobs); break;
        case CINN_F16: launch_dependent(split_parts_kernel<__half, 3>, dim3(grid), dim3(256), 0, st, jobs); break;
        default: launch_dependent(split_parts_kernel<__nv_bfloat16, 1>, dim3(grid), dim3(256), 0, st, jobs); break;
    }
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

// tensor maps of q, k, v (parts, heads, L, width), from the inputs themselves or from their parts
static int operand_map(const Plan& p, CUtensorMap* m, const void* direct, const uint8_t* parts, int64_t d, int64_t padded,
                       uint32_t box_rows = T) {
    if (p.direct)
        return encode_map_3d(m, direct, (uint64_t)d, (uint64_t)p.L, (uint64_t)p.BH, (uint64_t)d * 2, box_rows,
                             CU_TENSOR_MAP_DATA_TYPE_BFLOAT16);
    return encode_map_3d(m, parts, (uint64_t)padded, (uint64_t)p.L, (uint64_t)(p.ns * p.BH), (uint64_t)padded * 2, box_rows,
                         CU_TENSOR_MAP_DATA_TYPE_BFLOAT16);
}

static int head_group(const Plan& p) {
    const int64_t tiles = p.Lp / T, want = (3 * sm_count() + tiles - 1) / tiles;
    return (int)(want < p.BH ? want : p.BH);
}

template <int NS, int ND, int PAIRS>
static int launch_fwd_pairs(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdArgs& a, dim3 grid, cudaStream_t st) {
    using S = FwdShape<NS, ND, PAIRS>;
    auto kern = attn_fwd_kernel<NS, ND, PAIRS>;
    CINN_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::BYTES));
    launch_dependent(kern, dim3(grid), dim3(S::THREADS), S::BYTES, st, tq, tk, tv, a);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

// One pair of softmax warpgroups per CTA and two CTAs per SM, or two pairs in one CTA.  A block of one pair takes 1.4 times as long for
// its keys, and a call ends no sooner than a block of the last query tile has, so one pair needs more blocks per SM the longer the
// sequence is.  Up to three rounds of blocks, two rounds of one pair are as long as three of two.  Short blocks that all fit on the
// SMs at once are the exception, and with two value panels, of which one writes no probabilities, those of two rounds.
// Call times in us, one pair -> two (heads x queries of 192 | 64, bf16, 128 picks): 11 x 2048 102 -> 74, 18 x 2048 109 -> 94,
// 25 x 2048 133 -> 125, 38 x 2048 178 -> 176, 50 x 2048 211 -> 217, 85 x 512 92 -> 84, 150 x 512 123 -> 127, 296 x 128 53 -> 57.
static bool one_pair(int64_t blocks, int64_t n_tiles, int panels, int value_panels, int sms) {
    if (blocks <= sms) return false;
    if (blocks <= 2 * sms) return n_tiles <= 2 || (n_tiles <= 6 && panels + value_panels == 2 && 5 * blocks >= 6 * sms);
    if (blocks <= 3 * sms) return n_tiles <= 6 && value_panels == 2;
    return 8 * blocks > (24 + (n_tiles > 4 ? n_tiles - 4 : 0)) * sms;
}

// Heads per group of the forward: groups of one size, so that no small last one ends alone on its long blocks, with about three rounds of
// blocks each (six of half an SM for long sequences; on short ones that is up to 5 % slower).  Call times, three rounds and
// the rest in the last group -> this: 31 x 2048 queries of 192 198 -> 152 us with one pair, 62 x 2048 297 -> 256, 19 x 4096 362 -> 268.
static int forward_group(const Plan& p, bool one) {
    const int64_t tiles = p.Lp / T, want = ((one && tiles >= 12 ? 6 : 3) * sm_count() + tiles - 1) / tiles;
    const int64_t groups = (p.BH + want - 1) / want;
    return (int)((p.BH + groups - 1) / groups);
}

template <int NS, int ND>
static int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, FwdArgs& a, const Plan& p, cudaStream_t st) {
    const dim3 grid((unsigned)(p.Lp / T * p.BH), 1, (unsigned)p.nv);
    const bool one = NS == 1 && one_pair((int64_t)grid.x * grid.z, p.Lp / T, ND, p.nv, sm_count());
    a.group = forward_group(p, one);
    if constexpr (NS == 1)
        if (one) return launch_fwd_pairs<NS, ND, 1>(tq, tk, tv, a, grid, st);
    return launch_fwd_pairs<NS, ND, 2>(tq, tk, tv, a, grid, st);
}

int64_t forward_workspace_bytes(int64_t B, int64_t H, int64_t L, int64_t K, int64_t Dqk, int64_t Dv, int dtype) {
    if (!supported(B, H, L, K, Dqk, Dv)) return 0;
    const Plan p = make_plan(B, H, L, K, Dqk, Dv, dtype, false);
    return scratch_bytes(p, false);
}

// Returns the flag's device address in *flag: the gather kernel behind it runs when it is set.
int forward(const void* q, const void* k, const void* v, int dtype, const int64_t* idx, float* out, void* out_cast, float* lse,
            float* attn, int64_t B, int64_t H, int64_t L, int64_t K, int64_t Dqk, int64_t Dv, float scale, uint8_t* ws,
            const int** flag, cudaStream_t st) {
    const Plan p = make_plan(B, H, L, K, Dqk, Dv, dtype, false);
    auto al16 = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
    CINN_CHECK_ARG(!p.direct || (al16(q) && al16(k) && al16(v)), "sparse_attention: q, k and v must be 16-byte aligned");
    *flag = reinterpret_cast<const int*>(ws + p.flag_off);
    int rc = make_picks(p, idx, ws, st);
    if (rc) return rc;
    if (!p.direct) {
        SplitJobs jobs{};
        jobs.job[0] = {q, reinterpret_cast<uint16_t*>(ws + p.q_off), p.BH * L, (int)Dqk, p.dp};
        jobs.job[1] = {k, reinterpret_cast<uint16_t*>(ws + p.k_off), p.BH * L, (int)Dqk, p.dp};
        jobs.job[2] = {v, reinterpret_cast<uint16_t*>(ws + p.v_off), p.BH * L, (int)Dv, p.nv * 64};
        jobs.n = 3;
        rc = split_parts(jobs, dtype, st);
        if (rc) return rc;
    }
    CUtensorMap tq, tk, tv;
    if ((rc = operand_map(p, &tq, q, ws + p.q_off, Dqk, p.dp))) return rc;
    if ((rc = operand_map(p, &tk, k, ws + p.k_off, Dqk, p.dp))) return rc;
    if ((rc = operand_map(p, &tv, v, ws + p.v_off, Dv, p.nv * 64))) return rc;
    FwdArgs a{};
    a.picks = picks_of(p, ws);
    a.out = out; a.out_cast = out_cast; a.lse = lse; a.attn = attn; a.flag = reinterpret_cast<int*>(ws + p.flag_off);
    a.H = (int)H; a.L = (int)L; a.words = (int)(p.Lp / 32); a.K = (int)K; a.Dv = (int)Dv; a.BH = (int)p.BH; a.scale = scale;
    a.n_tiles = (int)(p.Lp / T);
    a.out_cast_tag = dtype;
    if (p.ns == 1) {
        switch (p.nd) {
            case 1: return launch_fwd<1, 1>(tq, tk, tv, a, p, st);
            case 2: return launch_fwd<1, 2>(tq, tk, tv, a, p, st);
            default: return launch_fwd<1, 3>(tq, tk, tv, a, p, st);
        }
    }
    switch (p.nd) {
        case 1: return launch_fwd<3, 1>(tq, tk, tv, a, p, st);
        case 2: return launch_fwd<3, 2>(tq, tk, tv, a, p, st);
        default: return launch_fwd<3, 3>(tq, tk, tv, a, p, st);
    }
}

template <int NS, int ND, int NV>
static int launch_bwd(const CUtensorMap (&m)[9], const BwdArgs& a, const Plan& p, cudaStream_t st) {
    auto qk = attn_bwd_query_kernel<NS, ND, NV>;
    auto kk = attn_bwd_key_kernel<NS, ND, NV>;
    const unsigned grid = (unsigned)(p.Lp / T * p.BH);
    CINN_CHECK_CUDA(cudaFuncSetAttribute(qk, cudaFuncAttributeMaxDynamicSharedMemorySize, QPassShape<NS, ND, NV>::BYTES));
    CINN_CHECK_CUDA(cudaFuncSetAttribute(kk, cudaFuncAttributeMaxDynamicSharedMemorySize, KPassShape<NS, ND, NV>::BYTES));
    launch_dependent(qk, dim3(grid), dim3(QUERY_THREADS), QPassShape<NS, ND, NV>::BYTES, st, m[0], m[1], m[2], m[3], m[6], a);
    CINN_CHECK_LAUNCH();
    launch_dependent(kk, dim3(grid), dim3(KEY_THREADS), KPassShape<NS, ND, NV>::BYTES, st, m[4], m[5], m[7], m[8], a);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

int64_t backward_workspace_bytes(int64_t B, int64_t H, int64_t L, int64_t K, int64_t Dqk, int64_t Dv, int dtype) {
    if (!supported(B, H, L, K, Dqk, Dv)) return 0;
    if (dtype == CINN_F32 && (Dqk % 4 != 0 || Dv % 4 != 0)) return 0;                // rows a TMA box cannot address
    const Plan p = make_plan(B, H, L, K, Dqk, Dv, dtype, true);
    return scratch_bytes(p, true);
}

// Gradients in `dtype` (dq, dk, dv written, not added to).  *flag as in forward; *fallback: fp32 buffers (dq | dk | dv) the
// gather kernel may use when it has to run.
int backward(const void* d_out, const float* out, const float* lse, const void* q, const void* k, const void* v, int dtype,
             const int64_t* idx, void* dq, void* dk, void* dv, int64_t B, int64_t H, int64_t L, int64_t K, int64_t Dqk, int64_t Dv,
             float scale, uint8_t* ws, const int** flag, float** fallback, cudaStream_t st) {
    const Plan p = make_plan(B, H, L, K, Dqk, Dv, dtype, true);
    *flag = reinterpret_cast<const int*>(ws + p.flag_off);
    *fallback = dtype != CINN_F32 ? reinterpret_cast<float*>(ws + p.grads_off) : nullptr;
    int rc = make_picks(p, idx, ws, st);
    if (rc) return rc;
    if (!p.direct) {
        SplitJobs jobs{};
        jobs.job[0] = {q, reinterpret_cast<uint16_t*>(ws + p.q_off), p.BH * L, (int)Dqk, p.dp};
        jobs.job[1] = {k, reinterpret_cast<uint16_t*>(ws + p.k_off), p.BH * L, (int)Dqk, p.dp};
        jobs.job[2] = {v, reinterpret_cast<uint16_t*>(ws + p.v_off), p.BH * L, (int)Dv, p.nv * 64};
        jobs.job[3] = {d_out, reinterpret_cast<uint16_t*>(ws + p.g_off), p.BH * L, (int)Dv, p.nv * 64};
        jobs.n = 4;
        rc = split_parts(jobs, dtype, st);
        if (rc) return rc;
    }
    float* delta = reinterpret_cast<float*>(ws + p.delta_off);
    const int64_t rows = p.BH * L, want = (rows + 7) / 8, cap = (int64_t)sm_count() * 32;
    const unsigned dgrid = (unsigned)(want < cap ? want : cap);
    switch (dtype) {
        case CINN_F32: launch_dependent(delta_kernel<float>, dim3(dgrid), dim3(256), 0, st, (const float*)d_out, out, delta, rows, (int)Dv); break;
        case CINN_F16: launch_dependent(delta_kernel<__half>, dim3(dgrid), dim3(256), 0, st, (const __half*)d_out, out, delta, rows, (int)Dv); break;
        default: launch_dependent(delta_kernel<__nv_bfloat16>, dim3(dgrid), dim3(256), 0, st, (const __nv_bfloat16*)d_out, out, delta, rows, (int)Dv); break;
    }
    CINN_CHECK_LAUNCH();
    CUtensorMap m[9];                                      // q, k, v, dO in boxes of 128 rows; q, dO in boxes of 32; dq, dk, dv
    if ((rc = operand_map(p, &m[0], q, ws + p.q_off, Dqk, p.dp))) return rc;
    if ((rc = operand_map(p, &m[1], k, ws + p.k_off, Dqk, p.dp))) return rc;
    if ((rc = operand_map(p, &m[2], v, ws + p.v_off, Dv, p.nv * 64))) return rc;
    if ((rc = operand_map(p, &m[3], d_out, ws + p.g_off, Dv, p.nv * 64))) return rc;
    if ((rc = operand_map(p, &m[4], q, ws + p.q_off, Dqk, p.dp, 32))) return rc;
    if ((rc = operand_map(p, &m[5], d_out, ws + p.g_off, Dv, p.nv * 64, 32))) return rc;
    m[6] = m[7] = m[8] = m[0];
    if (dtype == CINN_F32) {
        const struct { void* p; int64_t d; } outs[3] = {{dq, Dqk}, {dk, Dqk}, {dv, Dv}};
        for (int i = 0; i < 3; ++i)
            if ((rc = encode_map_3d(&m[6 + i], outs[i].p, (uint64_t)outs[i].d, (uint64_t)L, (uint64_t)p.BH, (uint64_t)outs[i].d * 4, T,
                                    CU_TENSOR_MAP_DATA_TYPE_FLOAT32, SLOT_COLS, CU_TENSOR_MAP_SWIZZLE_64B))) return rc;
    }
    BwdArgs a{};
    a.picks = picks_of(p, ws);
    a.lse = lse; a.delta = delta; a.pd = reinterpret_cast<float2*>(ws + p.pd_off);
    a.dq = dq; a.dk = dk; a.dv = dv; a.flag = reinterpret_cast<int*>(ws + p.flag_off);
    a.H = (int)H; a.L = (int)L; a.words = (int)(p.Lp / 32); a.K = (int)K; a.Dqk = (int)Dqk; a.Dv = (int)Dv; a.BH = (int)p.BH;
    a.n_tiles = (int)(p.Lp / T); a.group = head_group(p); a.tag = dtype; a.scale = scale;
#define CINN_ATB(NS, ND, NV) if (p.ns == NS && p.nd == ND && p.nv == NV) return launch_bwd<NS, ND, NV>(m, a, p, st)
    CINN_ATB(1, 1, 1); CINN_ATB(1, 2, 1); CINN_ATB(1, 3, 1); CINN_ATB(1, 1, 2); CINN_ATB(1, 2, 2); CINN_ATB(1, 3, 2);
    CINN_ATB(3, 1, 1); CINN_ATB(3, 2, 1); CINN_ATB(3, 3, 1); CINN_ATB(3, 1, 2); CINN_ATB(3, 2, 2); CINN_ATB(3, 3, 2);
#undef CINN_ATB
    set_error("sparse_attention: no tile kernel for %d + %d column panels", p.nd, p.nv);
    return CINN_ERR_INVALID;
}

}  // namespace atc

int read_attn_status(int* out, int reset) {
    int v = 0;
    CINN_CHECK_CUDA(cudaMemcpyFromSymbol(&v, atc::g_attn_status, sizeof(int)));
    if (reset && v != 0) {
        int z = 0;
        CINN_CHECK_CUDA(cudaMemcpyToSymbol(atc::g_attn_status, &z, sizeof(int)));
    }
    *out = v;
    return CINN_OK;
}

}  // namespace cinn
