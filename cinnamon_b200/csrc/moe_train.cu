// The small passes of the trainable MoE block (layers.MoE): gates and balance loss with their derivative, the bias update.
//
// The reference writes them as chains of torch calls on (tokens, experts) tensors (src/layers.py:111-148, 167-177); as such
// they were 40 of the block's 128 launches and as many passes over the scores.  Here a warp keeps a token's scores in
// registers: one pass for the balance loss, one for the derivative of gates and loss together.
#include "common.cuh"

namespace cinn {

namespace {

template <typename L> __device__ __forceinline__ float widen(L v);
template <> __device__ __forceinline__ float widen<float>(float v) { return v; }
template <> __device__ __forceinline__ float widen<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float widen<__half>(__half v) { return __half2float(v); }
template <typename L> __device__ __forceinline__ L narrow(float v);
template <> __device__ __forceinline__ float narrow<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 narrow<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half narrow<__half>(float v) { return __float2half_rn(v); }

__device__ __forceinline__ float sigmoid(float x) { return __fdiv_rn(1.0f, 1.0f + expf(-x)); }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

constexpr int BAL_TOKENS = 64;                 // tokens of one sequence per CTA
constexpr int MAX_E = 1024;

}  // namespace

// Per CTA (64 tokens of one sequence): the sum of the normalised scores and the number of selections of every expert.
// Warps add up in their order, so the sums are the same on every run.
template <int VPL, typename L>                 // scores per lane, E <= 32 * VPL
__global__ void __launch_bounds__(256)
balance_partial_kernel(const L* __restrict__ logits, const int* __restrict__ top_experts, float* __restrict__ part_p,
                       int* __restrict__ part_c, int seq, int chunks, int E, int top_k) {
    pdl_wait();
    pdl_trigger();
    __shared__ float s_p[MAX_E];
    __shared__ int s_c[MAX_E];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int e = threadIdx.x; e < E; e += 256) { s_p[e] = 0.0f; s_c[e] = 0; }
    __syncthreads();
    const int b = blockIdx.x / chunks, l0 = (blockIdx.x - b * chunks) * BAL_TOKENS, l1 = min(l0 + BAL_TOKENS, seq);
    float acc[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i) acc[i] = 0.0f;
    for (int l = l0 + warp; l < l1; l += 8) {
        const int64_t t = (int64_t)b * seq + l;
        float s[VPL], sum = 0.0f;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int e = lane + 32 * i;
            s[i] = e < E ? sigmoid(widen<L>(logits[t * E + e])) : 0.0f;
            sum += s[i];
        }
        sum = warp_sum(sum) + 1e-9f;
#pragma unroll
        for (int i = 0; i < VPL; ++i) acc[i] += s[i] / sum;
        for (int j = lane; j < top_k; j += 32) atomicAdd(&s_c[top_experts[t * top_k + j]], 1);
    }
    for (int w = 0; w < 8; ++w) {
        if (warp == w) {
#pragma unroll
            for (int i = 0; i < VPL; ++i)
                if (lane + 32 * i < E) s_p[lane + 32 * i] += acc[i];
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < E; e += 256) {
        part_p[(int64_t)blockIdx.x * E + e] = s_p[e];
        part_c[(int64_t)blockIdx.x * E + e] = s_c[e];
    }
}

// share[b, e] = selections * E / (k * seq);  loss = alpha * mean_b sum_e share[b, e] * mean score[b, e]
__global__ void __launch_bounds__(1024)
balance_finish_kernel(const float* __restrict__ part_p, const int* __restrict__ part_c, float* __restrict__ share,
                      float* __restrict__ loss, int batch, int seq, int chunks, int E, int top_k, float alpha) {
    pdl_wait();
    pdl_trigger();
    __shared__ float s_sum[32];
    float sum = 0.0f;
    for (int64_t i = threadIdx.x; i < (int64_t)batch * E; i += 1024) {
        const int b = (int)(i / E), e = (int)(i - (int64_t)b * E);
        float p = 0.0f;
        int c = 0;
#pragma unroll 4
        for (int u = 0; u < chunks; ++u) {
            p += part_p[((int64_t)b * chunks + u) * E + e];
            c += part_c[((int64_t)b * chunks + u) * E + e];
        }
        const float sh = (float)c * ((float)E / (float)((int64_t)top_k * seq));
        share[i] = sh;
        sum += sh * (p / (float)seq);
    }
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x < 32) {
        const float total = warp_sum(s_sum[threadIdx.x]);
        if (threadIdx.x == 0) *loss = alpha * (total / (float)batch);
    }
}

// d logits from the gradients of the gates (in the order of pair_pos) and of the balance loss (share null: no such loss):
//   gate_j = s_j / (sum of the chosen s + 1e-9),  loss = alpha / (B L) sum share s_e / (sum_e s_e + 1e-9),  s = sigmoid(logit)
// One warp per token.
template <int VPL, typename L>
__global__ void __launch_bounds__(256)
gates_backward_kernel(const L* __restrict__ logits, const int64_t* __restrict__ sorted_experts, const int64_t* __restrict__ pair_pos,
                      const float* __restrict__ d_gates, const float* __restrict__ share, const float* __restrict__ d_loss, float coef,
                      L* __restrict__ d_logits, int64_t T, int seq, int E, int top_k) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    for (int64_t t = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); t < T; t += (int64_t)gridDim.x * 8) {
        float s[VPL], ds[VPL], sum = 0.0f;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int e = lane + 32 * i;
            s[i] = e < E ? sigmoid(widen<L>(logits[t * E + e])) : 0.0f;
            ds[i] = 0.0f;
            sum += s[i];
        }
        if (share != nullptr && d_loss != nullptr) {
            const float c = coef * *d_loss;
            sum = warp_sum(sum) + 1e-9f;
            float g[VPL], dot = 0.0f;
#pragma unroll
            for (int i = 0; i < VPL; ++i) {
                const int e = lane + 32 * i;
                g[i] = e < E ? c * share[t / seq * E + e] : 0.0f;
                dot = fmaf(g[i], s[i], dot);
            }
            dot = warp_sum(dot);
#pragma unroll
            for (int i = 0; i < VPL; ++i) ds[i] = (g[i] - dot / sum) / sum;
        }
        // lane j: the token's j-th pair
        float my_s = 0.0f, my_g = 0.0f;
        int my_e = -1;
        if (lane < top_k) {
            my_e = (int)sorted_experts[pair_pos[t * top_k + lane]];
            my_g = d_gates ? d_gates[t * top_k + lane] : 0.0f;
            my_s = sigmoid(widen<L>(logits[t * E + my_e]));
        }
        const float chosen = warp_sum(my_s) + 1e-9f, dot = warp_sum(my_g * my_s);
        const float my_d = (my_g - dot / chosen) / chosen;
        for (int j = 0; j < top_k; ++j) {
            const int e = __shfl_sync(0xffffffffu, my_e, j);
            const float d = __shfl_sync(0xffffffffu, my_d, j);
#pragma unroll
            for (int i = 0; i < VPL; ++i)
                if (lane + 32 * i == e) ds[i] += d;
        }
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int e = lane + 32 * i;
            if (e < E) d_logits[t * E + e] = narrow<L>(ds[i] * (1.0f - s[i]) * s[i]);
        }
    }
}

// bias of over-used experts down by gamma, of the others up, clamped to [-1, 1] (src/layers.py:111-116)
__global__ void update_bias_kernel(const int64_t* __restrict__ counts, float* __restrict__ bias, int E, float expected, float gamma) {
    pdl_wait();
    pdl_trigger();
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        const float b = bias[e] + ((float)counts[e] > expected ? -gamma : gamma);
        bias[e] = fminf(fmaxf(b, -1.0f), 1.0f);
    }
}

static int check_scores(int64_t T, int E, int top_k, int dtype) {
    CINN_CHECK_ARG(T >= 0 && E >= 1 && E <= MAX_E && top_k >= 1 && top_k <= 32 && top_k <= E, "moe scores: bad shape");
    CINN_CHECK_ARG(dtype == CINN_F32 || dtype == CINN_BF16 || dtype == CINN_F16, "moe scores: unknown dtype tag %d", dtype);
    return CINN_OK;
}

#define CINN_VPL(CALL) \
    do { if (E <= 32) { CALL(1); } else if (E <= 64) { CALL(2); } else if (E <= 128) { CALL(4); } else if (E <= 256) { CALL(8); } \
         else if (E <= 512) { CALL(16); } else { CALL(32); } } while (0)

static inline int64_t balance_chunks(int64_t seq) { return (seq + BAL_TOKENS - 1) / BAL_TOKENS; }

int64_t balance_workspace_bytes(int64_t batch, int64_t seq, int E) { return batch * balance_chunks(seq) * E * 8; }

template <typename L>
static void launch_balance(const L* logits, const int* top, float* pp, int* pc, int batch, int seq, int chunks, int E, int top_k, cudaStream_t st) {
#define CINN_CALL(V) launch_dependent(balance_partial_kernel<V, L>, dim3(batch * chunks), dim3(256), 0, st, logits, top, pp, pc, seq, chunks, E, top_k)
    CINN_VPL(CINN_CALL);
#undef CINN_CALL
}

int balance_loss(const void* logits, int dtype, const int* top_experts, int64_t batch, int64_t seq, int E, int top_k, float alpha,
                 void* workspace, float* share, float* loss, cudaStream_t st) {
    int rc = check_scores(batch * seq, E, top_k, dtype);
    if (rc) return rc;
    CINN_CHECK_ARG(batch >= 1 && seq >= 1 && logits && top_experts && workspace && share && loss, "balance_loss: bad arguments");
    const int64_t chunks = balance_chunks(seq);
    CINN_CHECK_ARG(batch * chunks < (1LL << 31) && seq < (1LL << 31), "balance_loss: too many tokens");
    float* pp = static_cast<float*>(workspace);
    int* pc = reinterpret_cast<int*>(pp + batch * chunks * E);
    if (dtype == CINN_F32) launch_balance((const float*)logits, top_experts, pp, pc, (int)batch, (int)seq, (int)chunks, E, top_k, st);
    else if (dtype == CINN_BF16) launch_balance((const __nv_bfloat16*)logits, top_experts, pp, pc, (int)batch, (int)seq, (int)chunks, E, top_k, st);
    else launch_balance((const __half*)logits, top_experts, pp, pc, (int)batch, (int)seq, (int)chunks, E, top_k, st);
    CINN_CHECK_LAUNCH();
    launch_dependent(balance_finish_kernel, dim3(1), dim3(1024), 0, st, pp, pc, share, loss, (int)batch, (int)seq, (int)chunks, E, top_k, alpha);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

template <typename L>
static void launch_gates(const L* logits, const int64_t* se, const int64_t* pos, const float* dg, const float* share, const float* dl,
                         float coef, L* out, int64_t T, int seq, int E, int top_k, cudaStream_t st) {
    const int64_t want = (T + 7) / 8, cap = (int64_t)sm_count() * 16;
    const unsigned grid = (unsigned)(want < cap ? want : cap);
#define CINN_CALL(V) launch_dependent(gates_backward_kernel<V, L>, dim3(grid), dim3(256), 0, st, logits, se, pos, dg, share, dl, coef, out, T, seq, E, top_k)
    CINN_VPL(CINN_CALL);
#undef CINN_CALL
}

int gates_backward(const void* logits, int dtype, const int64_t* sorted_experts, const int64_t* pair_pos, const float* d_gates,
                   const float* share, const float* d_loss, float alpha, int64_t batch, int64_t seq, int E, int top_k, void* d_logits,
                   cudaStream_t st) {
    const int64_t T = batch * seq;
    int rc = check_scores(T, E, top_k, dtype);
    if (rc) return rc;
    if (T == 0) return CINN_OK;
    CINN_CHECK_ARG(logits && sorted_experts && pair_pos && d_logits, "gates_backward: null pointer");
    const float coef = alpha / ((float)batch * (float)seq);
    if (dtype == CINN_F32) launch_gates((const float*)logits, sorted_experts, pair_pos, d_gates, share, d_loss, coef, (float*)d_logits, T, (int)seq, E, top_k, st);
    else if (dtype == CINN_BF16) launch_gates((const __nv_bfloat16*)logits, sorted_experts, pair_pos, d_gates, share, d_loss, coef, (__nv_bfloat16*)d_logits, T, (int)seq, E, top_k, st);
    else launch_gates((const __half*)logits, sorted_experts, pair_pos, d_gates, share, d_loss, coef, (__half*)d_logits, T, (int)seq, E, top_k, st);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

int update_bias(const int64_t* counts, float* bias, int E, float expected, float gamma, cudaStream_t st) {
    CINN_CHECK_ARG(counts && bias && E >= 1, "update_bias: bad arguments");
    launch_dependent(update_bias_kernel, dim3(1), dim3(256), 0, st, counts, bias, E, expected, gamma);
    CINN_CHECK_LAUNCH();
    return CINN_OK;
}

}  // namespace cinn
