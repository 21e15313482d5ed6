// Native host path: what kernels.py does between two Python calls - output allocation, argument checks, the sequence of
// library calls - in C++.  A small FP8 layer is a handful of launches of a few microseconds each; done from Python, the
// ctypes calls, device contexts and torch.empty calls around them cost four times the kernels (77 us against 15 us of
// GPU time for 128 tokens through a 512 -> 1024 layer).
//
// The kernels stay behind the plain C ABI: this extension holds function pointers into the one loaded copy of
// libcinnamon_b200.so, handed over by Python when it binds the library.
#pragma once
#include <torch/extension.h>
#include <torch/csrc/Exceptions.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <exception>
#include <string>
#include "../../../include/cinnamon_b200.h"

namespace cinnhost {

using at::Tensor;

#define CINN_HOST_API(X)                                                                                            \
    X(cinn_last_error) X(cinn_quant_rowwise) X(cinn_quant_rowwise_dual) X(cinn_quant_rowwise_with_block)             \
    X(cinn_quant_rowwise_with_block_t) X(cinn_quant_rowwise_dual_padded) X(cinn_quant_rowwise_with_block_t_padded) X(cinn_quant_blockwise) X(cinn_quant_block_beside) X(cinn_quant_linear) X(cinn_transpose_bytes)     \
    X(cinn_requant_row_to_block) X(cinn_fp8_gemm_ws) X(cinn_fp8_gemm_pitched) X(cinn_fp8_gemm_workspace_bytes) \
    X(cinn_lightning_indexer)                                                                                           \
    X(cinn_sparse_attn_workspace_bytes) X(cinn_sparse_attn_fwd_ws) X(cinn_sparse_attn_bwd) X(cinn_sparse_attn_bwd_ws)                  \
    X(cinn_fp8_linear_few_takes) X(cinn_fp8_linear_few)                                                                   \
    X(cinn_moe_route_workspace_ints) X(cinn_moe_route_ranges) X(cinn_spread_rows) X(cinn_fp8_grouped_gemm)                \
    X(cinn_swiglu_quant_rowwise) X(cinn_moe_combine) X(cinn_moe_combine_add) X(cinn_moe_sum_add)                \
    X(cinn_swiglu_rounded) X(cinn_swiglu_rounded_backward) X(cinn_moe_balance_workspace_bytes) X(cinn_moe_balance_loss)     \
    X(cinn_moe_gates_backward) X(cinn_moe_update_bias) X(cinn_moe_combine_backward) X(cinn_swiglu_backward)                 \
    X(cinn_fp8_grouped_wgrad_fused_scratch_bytes) X(cinn_fp8_grouped_wgrad_fused) X(cinn_quant_segments_bytes) X(cinn_quant_rowwise_segments)             \
    X(cinn_fp8_grouped_wgrad_segments_scratch_bytes) X(cinn_fp8_grouped_wgrad_segments)                          \
    X(cinn_swiglu_rounded_quant_block_t) X(cinn_swiglu_rounded_backward_quant_dual) X(cinn_swiglu_quant_segments) X(cinn_fp8_grouped_wgrad_swiglu) X(cinn_fp8_grouped_gemm_dgrad) X(cinn_zero_rows_outside)

struct Api {
#define CINN_DECL(name) decltype(&::name) name = nullptr;
    CINN_HOST_API(CINN_DECL)
#undef CINN_DECL
};
extern Api api;
extern PyObject* library_error;                // _lib.LibraryError

// A status of the library as an exception: `invalid` becomes Python's AssertionError, the rest LibraryError.
struct CinnError : std::exception {
    std::string msg;
    bool invalid;
    CinnError(std::string m, bool inv) : msg(std::move(m)), invalid(inv) {}
    const char* what() const noexcept override { return msg.c_str(); }
};

inline void check(int status, const char* what) {
    if (status == 0) return;
    throw CinnError(std::string(what) + ": " + api.cinn_last_error() + " (status " + std::to_string(status) + ")", status == 1);
}
inline void require(bool ok, const char* what) {
    if (!ok) throw CinnError(what, true);
}

// Runs the body of a native backward: a CinnError in an autograd worker travels to the caller's thread as the Python
// exception it stands for.
template <typename F>
void as_python_error(F&& body) {
    try {
        body();
    } catch (const CinnError& e) {
        pybind11::gil_scoped_acquire gil;
        PyErr_SetString(e.invalid ? PyExc_AssertionError : library_error, e.what());
        python_error err;
        err.persist();
        throw err;
    }
}

constexpr at::ScalarType F8 = at::kFloat8_e4m3fn;
constexpr int TAG_BF16 = 0, TAG_F32 = 1, TAG_F16 = 2, TAG_F32_BF16 = 3;
inline int tag_of(at::ScalarType t) {           // -1: not a type the kernels read
    switch (t) {
        case at::kBFloat16: return TAG_BF16;
        case at::kFloat: return TAG_F32;
        case at::kHalf: return TAG_F16;
        default: return -1;
    }
}
inline Tensor readable(const Tensor& t) { return tag_of(t.scalar_type()) < 0 ? t.to(at::kFloat) : t; }

inline Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Device& dev) {
    return at::detail::empty_cuda(size, type, dev, std::nullopt);
}
// Whether a call goes through its autograd node: a gradient will be recorded, or an input carries a forward-mode tangent, which
// the node refuses (computed without it, the tangent would be dropped in silence).
template <typename... T>
bool takes_node(const T&... t) {
    return (at::GradMode::is_enabled() && (t.requires_grad() || ...)) || (t._fw_grad(/*level=*/0).defined() || ...);
}
inline int64_t up(int64_t a, int64_t b) { return (a + b - 1) / b; }
constexpr int64_t MAX_PADDED_ROWS = 65535 * 128;          // of the padded quantisers: row blocks that a launch takes
// Whether they read a matrix in place, in 16-byte pieces
inline bool padded_in_place(const Tensor& t) {
    return t.stride(1) == 1 && t.stride(0) >= t.size(1) && t.stride(0) % 8 == 0 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}
inline void* stream() { return at::cuda::getCurrentCUDAStream().stream(); }
// Whether the current stream's launches become nodes of a graph; the null stream, which eager programs run on, is not asked (0.2 us)
inline bool capturing() {
    return stream() != nullptr && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
}
inline float* f32(const Tensor& t);
Tensor gemm(const Tensor& a, const Tensor& sa, const Tensor& b, int layout, const Tensor& sb, int64_t sbk, int64_t sbn, int64_t M,
            int64_t N, int64_t K, at::ScalarType type, int tag);               // linear.cpp

struct Quantised { Tensor q, s; };
struct Linear {                                 // what an FP8 linear's forward leaves for its backward
    Tensor out, x, x_scale, w, w_scale, w_t;
    bool x_is_block = false, x_is_block_t = false;
};
Linear linear_forward(const Tensor& x, const Tensor& weight, bool round_scale, bool need_dgrad, bool need_wgrad, bool kmajor, int div,
                      const Tensor& w_q, const Tensor& w_s, const Tensor& w_qt);
// the rest of linear_forward once x is quantised: weight, product (into r.out)
void linear_multiply(Linear& r, const Tensor& xq, const Tensor& xs, const Tensor& wf, bool need_dgrad, bool kmajor, int div, const Tensor& w_q,
                     const Tensor& w_s, const Tensor& w_qt);
Tensor linear_inference(const Tensor& x, const Tensor& weight, bool round_scale, int div, bool one_kernel);
// (input gradients, weight gradient).  `parts` > 1: the weight is that many layers of equally many rows (a multiple of 128)
// stacked, and every layer's input gradient is returned by itself.
std::tuple<std::vector<Tensor>, Tensor> linear_backward(const Tensor& grad_out, Tensor x, Tensor x_scale, const Tensor& w,
                                                        const Tensor& w_scale, const Tensor& w_t, at::IntArrayRef x_shape,
                                                        bool round_scale, bool x_is_block, bool x_is_block_t,
                                                        at::ScalarType weight_dtype, bool kmajor, int div, bool want_gx,
                                                        bool want_gw, at::ScalarType gx_type, int parts = 1);
// the rest of it once the output gradient is quantised
std::tuple<std::vector<Tensor>, Tensor> linear_backward_quantised(const Quantised& g, const Quantised& g_t, int64_t M, Tensor x, Tensor x_scale,
                                                                  const Tensor& w, const Tensor& w_scale, const Tensor& w_t,
                                                                  at::IntArrayRef x_shape, bool x_is_block, bool x_is_block_t,
                                                                  at::ScalarType weight_dtype, bool kmajor, int div, bool want_gx,
                                                                  bool want_gw, at::ScalarType gx_type, int parts);

Quantised rowwise(const Tensor& x, bool round_scale, int div);                 // moe.cpp
Quantised swiglu_quantised(const Tensor& h12, int div);
Tensor grouped(const Quantised& x, const Quantised& w, const Tensor& starts, const Tensor& ends, at::ScalarType type = at::kBFloat16);
struct Routes {                                 // moe_route's outputs, in three tensors
    Tensor longs, floats, top;                  // token_indices | sorted_experts | pair_pos | counts | starts | ends; scores | pair_gate
    int64_t pairs = 0, E = 0;
    int64_t* part(int64_t at) const { return longs.data_ptr<int64_t>() + at; }
    int64_t* token_indices() const { return part(0); }
    int64_t* sorted_experts() const { return part(pairs); }
    int64_t* pos() const { return part(2 * pairs); }
    Tensor counts() const { return longs.narrow(0, 3 * pairs, E); }
    Tensor starts() const { return longs.narrow(0, 3 * pairs + E, E); }
    Tensor ends() const { return longs.narrow(0, 3 * pairs + 2 * E, E); }
    float* gates() const { return static_cast<float*>(floats.data_ptr()) + pairs; }
};
Routes route(const Tensor& logits, const Tensor& bias, int64_t top_k);
// refuses operands on other devices or of other widths, before anything is launched
void check_layer(const Tensor& x, const Tensor& router, const Tensor& bias, const Quantised& w12, const Quantised& w3);
Quantised spread(const Quantised& x, const Routes& r, int64_t top_k);
inline float* f32(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }

}  // namespace cinnhost
