// MoE routing on the device: top-k selection and the stable sort of (token, expert) pairs by expert.
//
// Replaces the chain of torch calls at the head of cinnamon's MoE.forward (src/layers.py:122-148):
// sigmoid, + expert_bias, topk, gather, normalise, sort by expert, token_indices, bincount.  Two or three launches:
//
//   route_topk_kernel     one warp per token: sigmoid scores, the k largest of score + bias (ties: the lower
//                         expert id), gates = score / (sum of the k scores + 1e-9); every CTA also leaves a histogram
//                         of the experts its tokens selected in the workspace
//   route_scan_kernel     one warp per expert: the running sum of those histograms over the CTAs (the histograms
//                         become offsets) -> counts.  With 32 CTAs or fewer the scatter kernel does this itself.
//   route_scatter_kernel  the same CTAs again: an exclusive scan of the counts gives every expert's first row, and every
//                         pair gets the next free row of its expert, pairs taken in (token, slot) order, so the order is
//                         that of a stable sort and the same on every run; writes token_indices / sorted_scores /
//                         sorted_experts, the experts' row ranges, and per token its k rows in ascending order with their
//                         gates (what the combine pass reads)
//
// The workspace (one int per CTA and expert, and one more per expert) is the only memory beyond inputs and outputs.
#include "common.cuh"
#include <mutex>

namespace cinn {

constexpr int ROUTE_MAX_TOKENS_PER_CTA = 128;
constexpr int ROUTE_FEW_CTAS = 32;             // up to here the scatter kernel sums the histograms itself
constexpr int64_t ROUTE_STATIC_MAX_INTS = 1 << 19;                     // 2 MiB: the built-in scratch (moe_route_static)

// Tokens per CTA, a power of two: as few as one per warp while that is at most five CTAs per SM, more for more tokens.  Selecting
// the top k is a serial chain of shuffles per token, so what counts is how many warps there are, until the histograms of every
// CTA cost more than the chains save; five per SM is where the measured lines cross (us at 8 / 16 / 32 / 64 / 128 tokens per CTA:
// 2048 tokens x 256 experts 27 / 29 / 41 / 66 / 116, 8192 x 64 37 / 31 / 31 / 39 / 64, 16384 x 256 82 / 67 / 64 / 78 / 121,
// 32768 x 256 150 / 117 / 104 / 107 / 137, 131072 x 256 539 / 414 / 346 / 322 / 330).  (Any multiple of 8 instead: 24 and 72 tokens
// are up to 11 % slower than 32 and 128 with 8 pairs a token, which the scatter takes 256 at a time.)  Fewer CTAs where their
// histograms would not fit the built-in scratch, so that it serves what it serves at 128 tokens per CTA.
static inline int route_tokens_per_cta(int64_t T, int E) {
    int64_t per = 8;
    while (per < ROUTE_MAX_TOKENS_PER_CTA &&
           (T > per * 5 * sm_count() || ((T + per - 1) / per + 1) * E > ROUTE_STATIC_MAX_INTS)) per *= 2;
    return (int)per;
}

template <typename L> __device__ __forceinline__ float logit(L v);
template <> __device__ __forceinline__ float logit<float>(float v) { return v; }
template <> __device__ __forceinline__ float logit<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float logit<__half>(__half v) { return __half2float(v); }

constexpr int ROUTE_MAX_EXPERTS = 1024;
constexpr int ROUTE_MAX_TOPK = 32;

template <int VPL, typename L>      // expert values per lane, E <= 32 * VPL
__global__ void __launch_bounds__(256)
route_topk_kernel(const L* __restrict__ logits, const float* __restrict__ bias, int T, int E, int top_k, int tokens_per_cta,
                  int* __restrict__ top_experts, float* __restrict__ top_gates, int* __restrict__ hist) {
    pdl_wait();
    pdl_trigger();
    __shared__ int s_hist[ROUTE_MAX_EXPERTS];
    for (int e = threadIdx.x; e < E; e += 256) s_hist[e] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t_begin = blockIdx.x * tokens_per_cta;
    const int t_end = min(t_begin + tokens_per_cta, T);
    float b[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i) b[i] = (lane + 32 * i < E) ? bias[lane + 32 * i] : 0.0f;
    for (int t = t_begin + warp; t < t_end; t += 8) {
        float s[VPL], sel[VPL];
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int e = lane + 32 * i;
            if (e < E) {
                const float x = logit<L>(logits[(int64_t)t * E + e]);
                s[i] = __fdiv_rn(1.0f, 1.0f + expf(-x));                  // torch.sigmoid in fp32
                sel[i] = s[i] + b[i];
                if (sel[i] != sel[i]) sel[i] = -INFINITY;                  // a NaN is never selected
            } else {
                s[i] = 0.0f;
                sel[i] = -INFINITY;
            }
        }
        float my_score = 0.0f;
        int my_expert = 0;
        for (int r = 0; r < top_k; ++r) {
            float best = -INFINITY;
            int best_e = 0x7fffffff;
#pragma unroll
            for (int i = 0; i < VPL; ++i)
                if (sel[i] > best) { best = sel[i]; best_e = lane + 32 * i; }
            if (best == -INFINITY) best_e = 0x7fffffff;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
                if (ov > best || (ov == best && oe < best_e)) { best = ov; best_e = oe; }
            }
            // fewer than k selectable experts (E < k, or NaNs): fall back to the lowest unused ids
            if (best_e == 0x7fffffff) best_e = r < E ? r : 0;
            float sc = 0.0f;
#pragma unroll
            for (int i = 0; i < VPL; ++i)
                if (lane + 32 * i == best_e) { sc = s[i]; sel[i] = -INFINITY; }
            sc = __shfl_sync(0xffffffffu, sc, best_e & 31);
            if (lane == r) { my_score = sc; my_expert = best_e; }
        }
        float sum = lane < top_k ? my_score : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane < top_k) {
            top_experts[(int64_t)t * top_k + lane] = my_expert;
            top_gates[(int64_t)t * top_k + lane] = __fdiv_rn(my_score, sum + 1e-9f);
            atomicAdd(&s_hist[my_expert], 1);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += 256) hist[(int64_t)blockIdx.x * E + e] = s_hist[e];
}

__global__ void __launch_bounds__(256)
route_scan_kernel(int* __restrict__ hist, int n_ctas, int E, int* __restrict__ totals) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31, e = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (e >= E) return;
    int carry = 0;
    for (int b0 = 0; b0 < n_ctas; b0 += 128) {               // four histograms per lane in flight
        int v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int b = b0 + u * 32 + lane;
            v[u] = b < n_ctas ? hist[(int64_t)b * E + e] : 0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int b = b0 + u * 32 + lane;
            int incl = v[u];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += x;
            }
            if (b < n_ctas) hist[(int64_t)b * E + e] = carry + incl - v[u];
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    if (lane == 0) totals[e] = carry;
}

// totals: per-expert counts from route_scan_kernel, with `hist` turned into offsets; null: hist still holds counts
__global__ void __launch_bounds__(256)
route_scatter_kernel(const int* __restrict__ top_experts, const float* __restrict__ top_gates, const int* __restrict__ hist,
                     const int* __restrict__ totals, int T, int E, int top_k, int tokens_per_cta, int64_t* __restrict__ token_indices,
                     float* __restrict__ sorted_scores, int64_t* __restrict__ sorted_experts, int64_t* __restrict__ counts,
                     int64_t* __restrict__ starts, int64_t* __restrict__ ends, int64_t* __restrict__ pair_pos,
                     float* __restrict__ pair_gate) {
    pdl_wait();
    pdl_trigger();
    __shared__ int s_next[ROUTE_MAX_EXPERTS];                                  // next free row of every expert
    __shared__ int s_warp[8];
    __shared__ int s_pos[ROUTE_MAX_TOKENS_PER_CTA * ROUTE_MAX_TOPK];
    {
        // thread i: experts 4 i .. 4 i + 3; their counts, the rows of earlier CTAs, and a scan of the counts
        int cnt[4], mine[4], sum = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = threadIdx.x * 4 + u;
            cnt[u] = 0; mine[u] = 0;
            if (e < E) {
                if (totals) {
                    cnt[u] = totals[e];
                    mine[u] = hist[(int64_t)blockIdx.x * E + e];
                } else {
                    for (int b = 0; b < (int)gridDim.x; ++b) {
                        const int v = hist[(int64_t)b * E + e];
                        if (b < (int)blockIdx.x) mine[u] += v;
                        cnt[u] += v;
                    }
                }
            }
            sum += cnt[u];
        }
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        int first = incl - sum;
        for (int w = 0; w < warp; ++w) first += s_warp[w];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = threadIdx.x * 4 + u;
            if (e < E) {
                s_next[e] = first + mine[u];
                if (blockIdx.x == 0) {
                    counts[e] = cnt[u];
                    if (starts) { starts[e] = first; ends[e] = first + cnt[u]; }
                }
                first += cnt[u];
            }
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t_begin = blockIdx.x * tokens_per_cta;
    const int n_tok = min(tokens_per_cta, T - t_begin);
    const int n_pairs = n_tok * top_k;
    const int64_t pair0 = (int64_t)t_begin * top_k;
    for (int base = 0; base < n_pairs; base += 256) {
        const int p = base + threadIdx.x;
        const bool live = p < n_pairs;
        const int e = live ? top_experts[pair0 + p] : -1 - lane;              // dead lanes match nobody
        const int turns = min(8, (n_pairs - base + 31) / 32);
        for (int w = 0; w < turns; ++w) {                                      // warps take their turn: (token, slot) order
            if (warp == w) {
                const unsigned peers = __match_any_sync(0xffffffffu, e);
                const int leader = __ffs(peers) - 1;
                int row = 0;
                if (live && lane == leader) {
                    row = s_next[e];
                    s_next[e] = row + __popc(peers);
                }
                row = __shfl_sync(0xffffffffu, row, leader) + __popc(peers & ((1u << lane) - 1u));
                if (live) {
                    s_pos[p] = row;
                    token_indices[row] = t_begin + p / top_k;
                    sorted_scores[row] = top_gates[pair0 + p];
                    sorted_experts[row] = e;
                }
            }
            __syncthreads();
        }
    }
    // per token: its rows in ascending order, gates alongside (insertion sort, k <= 32)
    for (int tl = threadIdx.x; tl < n_tok; tl += 256) {
        int pos[ROUTE_MAX_TOPK];
        float gate[ROUTE_MAX_TOPK];
        for (int j = 0; j < top_k; ++j) {
            const int v = s_pos[tl * top_k + j];
            const float g = top_gates[pair0 + tl * top_k + j];
            int i = j;
            while (i > 0 && pos[i - 1] > v) { pos[i] = pos[i - 1]; gate[i] = gate[i - 1]; --i; }
            pos[i] = v;
            gate[i] = g;
        }
        for (int j = 0; j < top_k; ++j) {
            pair_pos[(int64_t)(t_begin + tl) * top_k + j] = pos[j];
            pair_gate[(int64_t)(t_begin + tl) * top_k + j] = gate[j];
        }
    }
}

int64_t moe_route_workspace_ints(int64_t T, int E) {
    const int per = route_tokens_per_cta(T, E);
    return ((T + per - 1) / per) * (int64_t)E + E;
}

template <typename L>
static void launch_topk(const L* logits, const float* bias, int T, int E, int top_k, int per, int n_ctas, int* top_experts,
                        float* top_gates, int* hist, cudaStream_t st) {
#define CINN_TOPK(V) launch_dependent(route_topk_kernel<V, L>, dim3(n_ctas), dim3(256), 0, st, logits, bias, T, E, top_k, per, top_experts, top_gates, hist)
    if (E <= 32) CINN_TOPK(1);
    else if (E <= 64) CINN_TOPK(2);
    else if (E <= 128) CINN_TOPK(4);
    else if (E <= 256) CINN_TOPK(8);
    else if (E <= 512) CINN_TOPK(16);
    else CINN_TOPK(32);
#undef CINN_TOPK
}

// logits_dtype: CINN_F32, or a 16-bit type that is widened on load.  starts / ends (E each): null, or every expert's rows.
int moe_route(const void* logits, int logits_dtype, const float* bias, int64_t T, int E, int top_k, int* workspace, int* top_experts,
              float* top_gates, int64_t* token_indices, float* sorted_scores, int64_t* sorted_experts, int64_t* counts,
              int64_t* starts, int64_t* ends, int64_t* pair_pos, float* pair_gate, cudaStream_t st) {
    CINN_CHECK_ARG(T >= 0 && E >= 1 && E <= ROUTE_MAX_EXPERTS, "moe_route: 1 <= E <= %d experts (got %d)", ROUTE_MAX_EXPERTS, E);
    CINN_CHECK_ARG(top_k >= 1 && top_k <= ROUTE_MAX_TOPK && top_k <= E, "moe_route: 1 <= top_k <= min(E, %d) (got %d)",
                   ROUTE_MAX_TOPK, top_k);
    CINN_CHECK_ARG(T * (int64_t)top_k < (1LL << 31), "moe_route: too many (token, expert) pairs");
    CINN_CHECK_ARG(counts != nullptr && (starts == nullptr) == (ends == nullptr), "moe_route: null pointer");
    CINN_CHECK_ARG(logits_dtype == CINN_F32 || logits_dtype == CINN_BF16 || logits_dtype == CINN_F16, "moe_route: unknown dtype tag %d",
                   logits_dtype);
    if (T == 0) {
        CINN_CHECK_CUDA(cudaMemsetAsync(counts, 0, sizeof(int64_t) * E, st));
        if (starts) {
            CINN_CHECK_CUDA(cudaMemsetAsync(starts, 0, sizeof(int64_t) * E, st));
            CINN_CHECK_CUDA(cudaMemsetAsync(ends, 0, sizeof(int64_t) * E, st));
        }
        return CINN_OK;
    }
    CINN_CHECK_ARG(logits && bias && workspace && top_experts && top_gates && token_indices && sorted_scores &&
                   sorted_experts && pair_pos && pair_gate, "moe_route: null pointer");
    const int per = route_tokens_per_cta(T, E), n_ctas = (int)((T + per - 1) / per);
    int* hist = workspace;
    int* totals = n_ctas > ROUTE_FEW_CTAS ? workspace + (int64_t)n_ctas * E : nullptr;
    if (logits_dtype == CINN_F32) launch_topk((const float*)logits, bias, (int)T, E, top_k, per, n_ctas, top_experts, top_gates, hist, st);
    else if (logits_dtype == CINN_BF16) launch_topk((const __nv_bfloat16*)logits, bias, (int)T, E, top_k, per, n_ctas, top_experts, top_gates, hist, st);
    else launch_topk((const __half*)logits, bias, (int)T, E, top_k, per, n_ctas, top_experts, top_gates, hist, st);
    CINN_CHECK_LAUNCH();
    if (totals) {
        launch_dependent(route_scan_kernel, dim3((E + 7) / 8), dim3(256), 0, st, hist, n_ctas, E, totals);
        CINN_CHECK_LAUNCH();
    }
    launch_dependent(route_scatter_kernel, dim3(n_ctas), dim3(256), 0, st, top_experts, top_gates, hist, totals, (int)T, E, top_k, per, token_indices, sorted_scores,
                                                 sorted_experts, counts, starts, ends, pair_pos, pair_gate);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

// ---------------------------------------------------------------------------
// The same routing for callers that cannot hand over a workspace.  The scratch lives in a fixed array inside
// the library image: every GPU that loads the library holds these 2 MiB until the process exits.  All calls on
// a device share it, so two calls that overlap on that GPU (different streams, different threads) race; the
// routing kernels overwrite every word they later read, so nothing has to be cleared between calls.
// ---------------------------------------------------------------------------
static __device__ __align__(256) int g_route_scratch[ROUTE_STATIC_MAX_INTS];

constexpr int ROUTE_MAX_DEVICES = 64;
static std::mutex g_route_scratch_mutex;
static int* g_route_scratch_ptr[ROUTE_MAX_DEVICES] = {};               // device address of the array, per device

// In host code `g_route_scratch` is only a handle for the symbol, not an address a kernel can use; the device
// address is asked for once per device, with that device current.
static int route_scratch_address(int** out) {
    int dev = -1;
    CINN_CHECK_CUDA(cudaGetDevice(&dev));
    CINN_CHECK_ARG(dev >= 0 && dev < ROUTE_MAX_DEVICES, "moe_route_static: device ordinal %d is beyond %d", dev,
                   ROUTE_MAX_DEVICES);
    std::lock_guard<std::mutex> lock(g_route_scratch_mutex);
    if (g_route_scratch_ptr[dev] == nullptr) {
        void* p = nullptr;
        CINN_CHECK_CUDA(cudaGetSymbolAddress(&p, g_route_scratch));
        g_route_scratch_ptr[dev] = static_cast<int*>(p);
    }
    *out = g_route_scratch_ptr[dev];
    return CINN_OK;
}

int64_t moe_route_static_max_ints() { return ROUTE_STATIC_MAX_INTS; }

int moe_route_static(const float* logits, const float* bias, int64_t T, int E, int top_k, int* top_experts, float* top_gates,
                     int64_t* token_indices, float* sorted_scores, int64_t* sorted_experts, int64_t* counts,
                     int64_t* pair_pos, float* pair_gate, cudaStream_t st) {
    CINN_CHECK_ARG(T >= 0 && E >= 1 && E <= ROUTE_MAX_EXPERTS, "moe_route_static: 1 <= E <= %d experts (got %d)",
                   ROUTE_MAX_EXPERTS, E);
    const int64_t need = moe_route_workspace_ints(T, E);
    CINN_CHECK_ARG(need <= ROUTE_STATIC_MAX_INTS,
                   "moe_route_static: %lld tokens x %d experts need %lld ints of scratch, the built-in array holds %lld; "
                   "use cinn_moe_route with a workspace of your own",
                   (long long)T, E, (long long)need, (long long)ROUTE_STATIC_MAX_INTS);
    int* scratch = nullptr;
    int rc = route_scratch_address(&scratch);
    if (rc) return rc;
    return moe_route(logits, CINN_F32, bias, T, E, top_k, scratch, top_experts, top_gates, token_indices, sorted_scores,
                     sorted_experts, counts, nullptr, nullptr, pair_pos, pair_gate, st);
}

}  // namespace cinn
