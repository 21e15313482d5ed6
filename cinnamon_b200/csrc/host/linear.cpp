// FP8 linear: forward and both gradients of FP8MatmulFunction (reference src/kernels.py:731-794) as one native call
// each, and as a native autograd node.
#include "host.h"

namespace cinnhost {

Tensor gemm(const Tensor& a, const Tensor& sa, const Tensor& b, int layout, const Tensor& sb, int64_t sbk, int64_t sbn, int64_t M,
            int64_t N, int64_t K, at::ScalarType type, int tag) {
    Tensor out = empty({M, N}, type, a.device());
    const int64_t need = api.cinn_fp8_gemm_workspace_bytes(M, N, K, layout);       // few tiles, long reduction: cut along K
    Tensor ws = need ? empty({need}, at::kByte, a.device()) : Tensor();
    check(api.cinn_fp8_gemm_ws(a.data_ptr(), f32(sa), sa.stride(0), b.data_ptr(), f32(sb), sbk, sbn, out.data_ptr(), M, N, K, layout,
                               tag, need ? ws.data_ptr() : nullptr, need, stream()), "cinn_fp8_gemm");
    return out;
}

// What the kernels take for granted, refused on the host before anything is launched.  w_q, w_s: the weight's e4m3 copy, or
// undefined.
static void check_operands(const Tensor& x, const Tensor& weight, const Tensor& w_q, const Tensor& w_s) {
    require(x.is_cuda() && weight.is_cuda(), "Input must be on CUDA");
    require(weight.device() == x.device(), "FP8 linear: input and weight must be on the same device");
    require(x.dim() >= 1 && weight.dim() == 2 && weight.size(1) == x.size(-1),
            "FP8 linear: the weight must be a matrix as wide as the input's last dimension");
    TORCH_CHECK(x.numel() > 0, "FP8 linear: the input has no rows");
    if (!w_q.defined()) return;
    require(w_s.defined() && w_q.device() == x.device() && w_s.device() == x.device() && w_q.sizes() == weight.sizes() && w_q.is_contiguous() &&
                w_q.scalar_type() == F8 && w_s.scalar_type() == at::kFloat && w_s.dim() == 2 && w_s.size(0) == up(weight.size(0), 128) &&
                w_s.size(1) == up(weight.size(1), 128), "FP8 linear: the quantised copy does not belong to the weight");
}

Linear linear_forward(const Tensor& x, const Tensor& weight, bool round_scale, bool need_dgrad, bool need_wgrad, bool kmajor, int div,
               const Tensor& w_q, const Tensor& w_s, const Tensor& w_qt) {
    check_operands(x, weight, w_q, w_s);
    c10::cuda::CUDAGuard guard(x.device());
    const at::Device dev = x.device();
    const int64_t K = x.size(-1), N = weight.size(0);
    Tensor xf = readable(x.dim() == 2 ? x : x.reshape({-1, K}));
    const int64_t M = xf.size(0), nkb = up(K, 128);
    // A weight of another type is converted here, before the activations' quantiser is enqueued: the weight's quantiser runs
    // beside that one and waits for nothing it reads.
    const Tensor wf = w_q.defined() ? Tensor() : readable(weight);
    Linear r;
    // When the weight will want a gradient, the block re-quantisation of the saved activations comes out of the same
    // pass over x; it is written with the token axis contiguous, since the weight gradient reduces over tokens, and padded
    // to a multiple of 16 with zeros, which change no sum.
    const int64_t Mp = up(M, 16) * 16;
    r.x_is_block = need_wgrad && K % 16 == 0;
    r.x_is_block_t = r.x_is_block && kmajor && (Mp == M || M <= MAX_PADDED_ROWS);
    Tensor xq = empty({M, K}, F8, dev), xs = empty({M, nkb}, at::kFloat, dev);
    if (r.x_is_block) {
        if (xf.stride(1) != 1) xf = xf.contiguous();
        if (r.x_is_block_t && Mp != M && xf.stride(0) >= K && !padded_in_place(xf)) xf = xf.clone(at::MemoryFormat::Contiguous);
        r.x = r.x_is_block_t ? empty({K, Mp}, F8, dev) : empty({M, K}, F8, dev);
        r.x_scale = empty({up(M, 128), nkb}, at::kFloat, dev);
        check((!r.x_is_block_t ? api.cinn_quant_rowwise_with_block
                               : Mp == M ? api.cinn_quant_rowwise_with_block_t : api.cinn_quant_rowwise_with_block_t_padded)(
                  xf.data_ptr(), tag_of(xf.scalar_type()), M, K, xf.stride(0), xq.data_ptr(), f32(xs), r.x.data_ptr(), f32(r.x_scale),
                  round_scale, div, stream()), "cinn_quant_rowwise_with_block");
    } else {
        check(api.cinn_quant_rowwise(xf.data_ptr(), tag_of(xf.scalar_type()), M, K, xf.stride(0), xf.stride(1), xq.data_ptr(), f32(xs),
                                     128, round_scale, div, stream()), "cinn_quant_rowwise");
        r.x = xq;
        r.x_scale = xs;
    }
    linear_multiply(r, xq, xs, wf, need_dgrad, kmajor, div, w_q, w_s, w_qt);
    if (x.dim() != 2) {
        auto shape = x.sizes().vec();
        shape.back() = N;
        r.out = r.out.view(shape);
    }
    return r;
}

// wf: the weight in a type the quantiser reads (undefined with w_q)
void linear_multiply(Linear& r, const Tensor& xq, const Tensor& xs, const Tensor& wf, bool need_dgrad, bool kmajor, int div, const Tensor& w_q,
                     const Tensor& w_s, const Tensor& w_qt) {
    const at::Device dev = xq.device();
    const int64_t M = xq.size(0), K = xq.size(1), N = (w_q.defined() ? w_q : wf).size(0);
    if (w_q.defined()) {
        r.w = w_q;
        r.w_scale = w_s;
        r.w_t = w_qt;
    } else {
        r.w = empty({N, K}, F8, dev);
        r.w_scale = empty({up(N, 128), up(K, 128)}, at::kFloat, dev);
        // the input gradient multiplies by the weight with N as the reduction axis: the byte-transposed copy it reads
        // comes out of the same pass
        if (kmajor && need_dgrad && N % 16 == 0 && K % 4 == 0 && wf.stride(1) == 1 && wf.stride(0) % 4 == 0) {
            r.w_t = empty({K, N}, F8, dev);
        }
        // beside the activations' quantiser just enqueued
        check(api.cinn_quant_block_beside(wf.data_ptr(), tag_of(wf.scalar_type()), N, K, wf.stride(0), wf.stride(1), r.w.data_ptr(),
                                          r.w_t.defined() ? r.w_t.data_ptr() : nullptr, f32(r.w_scale), 0, div, stream()),
              "cinn_quant_blockwise");
    }
    r.out = gemm(xq, xs, r.w, 0, r.w_scale, r.w_scale.stride(1), r.w_scale.stride(0), M, N, K, at::kBFloat16, TAG_BF16);
}

std::tuple<std::vector<Tensor>, Tensor> linear_backward(const Tensor& grad_out, Tensor x, Tensor x_scale, const Tensor& w,
                                                        const Tensor& w_scale, const Tensor& w_t, at::IntArrayRef x_shape,
                                                        bool round_scale, bool x_is_block, bool x_is_block_t,
                                                        at::ScalarType weight_dtype, bool kmajor, int div, bool want_gx,
                                                        bool want_gw, at::ScalarType gx_type, int parts) {
    c10::cuda::CUDAGuard guard(w.device());
    const at::Device dev = w.device();
    const int64_t N = w.size(0);
    Tensor g = readable(grad_out.dim() == 2 ? grad_out : grad_out.reshape({-1, grad_out.size(-1)}));
    if (g.stride(1) != 1) g = g.contiguous();
    int64_t M = g.size(0);
    const int64_t Mp = up(M, 16) * 16;
    // The token axis is the reduction axis of the weight gradient: a ragged count is padded with zeros, which change neither an
    // amax nor a sum, by the quantiser; where that cannot be, and for activations saved with their tokens outermost, by a copy.
    // (12654 tokens, 1280 -> 3520: 75 of 325 us were such copies.)
    int64_t rows = M;
    if (Mp != M) {
        if (N % 8 != 0 || M > MAX_PADDED_ROWS) {
            g = at::constant_pad_nd(g, {0, 0, 0, Mp - M});
            rows = Mp;
        } else if (!padded_in_place(g)) {
            g = g.clone(at::MemoryFormat::Contiguous);
        }
        if (!x_is_block_t) x = at::constant_pad_nd(x.view(at::kByte), {0, 0, 0, Mp - M}).view(F8);
        if (!x_is_block) x_scale = at::constant_pad_nd(x_scale, {0, 0, 0, Mp - M}, 1.0);
    }
    Tensor gq = empty({rows, N}, F8, dev), gs = empty({rows, up(N, 128)}, at::kFloat, dev);
    Tensor gqt = empty({N, Mp}, F8, dev), gst = empty({N, up(Mp, 128)}, at::kFloat, dev);
    check((rows == Mp ? api.cinn_quant_rowwise_dual : api.cinn_quant_rowwise_dual_padded)(
              g.data_ptr(), tag_of(g.scalar_type()), rows, N, g.stride(0), gq.data_ptr(), f32(gs), gqt.data_ptr(), f32(gst), round_scale, div,
              stream()), "cinn_quant_rowwise_dual");
    return linear_backward_quantised({gq, gs}, {gqt, gst}, M, x, x_scale, w, w_scale, w_t, x_shape, x_is_block, x_is_block_t, weight_dtype, kmajor,
                                     div, want_gx, want_gw, gx_type, parts);
}

// g: the output gradient quantised along its features (M rows at least), g_t: along the tokens, (N, M rounded up to 16)
std::tuple<std::vector<Tensor>, Tensor> linear_backward_quantised(const Quantised& g, const Quantised& g_t, int64_t M, Tensor x, Tensor x_scale,
                                                                  const Tensor& w, const Tensor& w_scale, const Tensor& w_t,
                                                                  at::IntArrayRef x_shape, bool x_is_block, bool x_is_block_t,
                                                                  at::ScalarType weight_dtype, bool kmajor, int div, bool want_gx,
                                                                  bool want_gw, at::ScalarType gx_type, int parts) {
    const at::Device dev = w.device();
    const int64_t N = w.size(0), K = w.size(1), Mp = g_t.q.size(1);
    const Tensor &gq = g.q, &gs = g.s, &gqt = g_t.q, &gst = g_t.s;
    // (the reference's input gradient is bf16 and autograd casts it to the input's type: fp32 holds those values)
    const int gx_tag = gx_type == at::kFloat ? TAG_F32_BF16 : TAG_BF16;
    std::vector<Tensor> gx(parts);
    if (want_gx) {
        const bool k_major = N % 16 == 0 && (kmajor || w_t.defined());
        Tensor wt = w_t;
        if (k_major && !wt.defined()) {
            wt = empty({K, N}, F8, dev);
            check(api.cinn_transpose_bytes(w.data_ptr(), w.stride(0), wt.data_ptr(), N, K, stream()), "cinn_transpose_bytes");
        }
        const int64_t n = N / parts;                // reduction length of a part: columns of gq and wt, rows of w
        const int64_t need = api.cinn_fp8_gemm_workspace_bytes(M, K, n, k_major ? 0 : 1);
        Tensor ws = need ? empty({need}, at::kByte, dev) : Tensor();
        for (int p = 0; p < parts; ++p) {
            Tensor out = empty({M, K}, gx_type, dev);
            const uint8_t* b = static_cast<const uint8_t*>(k_major ? wt.data_ptr() : w.data_ptr()) + p * n * (k_major ? 1 : K);
            check(api.cinn_fp8_gemm_pitched(static_cast<const uint8_t*>(gq.data_ptr()) + p * n, N, f32(gs) + p * (n / 128), gs.stride(0), b,
                                            k_major ? N : K, f32(w_scale) + p * (n / 128) * w_scale.stride(0), w_scale.stride(0),
                                            w_scale.stride(1), out.data_ptr(), M, K, n, k_major ? 0 : 1, gx_tag,
                                            need ? ws.data_ptr() : nullptr, need, stream()), "cinn_fp8_gemm");
            gx[p] = x_shape.size() != 2 ? out.reshape(x_shape) : out;
        }
    }
    if (!want_gw) return {gx, Tensor()};
    if (!x_is_block) {
        Tensor xb = empty({Mp, K}, F8, dev), xbs = empty({up(Mp, 128), up(K, 128)}, at::kFloat, dev);
        x = x.contiguous();
        x_scale = x_scale.contiguous();
        check(api.cinn_requant_row_to_block(x.data_ptr(), f32(x_scale), Mp, K, xb.data_ptr(), f32(xbs), 0, div, stream()),
              "cinn_requant_row_to_block");
        x = xb;
        x_scale = xbs;
    }
    // the reference returns a bf16 gradient that autograd casts to the master weight's type: the GEMM writes those values
    const bool w32 = weight_dtype == at::kFloat;
    Tensor gw = gemm(gqt, gst, x, x_is_block_t ? 0 : 1, x_scale, x_scale.stride(0), x_scale.stride(1), N, K, Mp,
                     w32 ? at::kFloat : at::kBFloat16, w32 ? TAG_F32_BF16 : TAG_BF16);
    return {gx, gw};
}


// Without gradients nothing but the result outlives the call: one launch for few rows (one_kernel), else one scratch buffer and one
// launch for both quantisers.
Tensor linear_inference(const Tensor& x, const Tensor& weight, bool round_scale, int div, bool one_kernel) {
    check_operands(x, weight, Tensor(), Tensor());
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t K = x.size(-1), N = weight.size(0), nkb = up(K, 128);
    const Tensor xf = readable(x.dim() == 2 ? x : x.reshape({-1, K})), wf = readable(weight);
    const int64_t M = xf.size(0);
    auto shape = x.sizes().vec();
    shape.back() = N;
    Tensor out = empty(shape, at::kBFloat16, x.device());
    // under capture the launch that the one kernel saves costs next to nothing, and with many rows the two are shorter (csrc/linear_few.cu)
    const auto pays = [&] { return M <= 32 || K <= 128 || !capturing(); };
    if (one_kernel && M <= 128 && K <= 1024 && api.cinn_fp8_linear_few_takes(xf.data_ptr(), tag_of(xf.scalar_type()), xf.stride(0), xf.stride(1), wf.data_ptr(),
                                      tag_of(wf.scalar_type()), wf.stride(0), wf.stride(1), M, N, K) && pays()) {
        check(api.cinn_fp8_linear_few(xf.data_ptr(), tag_of(xf.scalar_type()), xf.stride(0), round_scale, f32(wf), wf.stride(0),
                                      out.data_ptr(), M, N, K, div, stream()), "cinn_fp8_linear_few");
        return out;
    }
    const auto room = [](int64_t bytes) { return (bytes + 255) / 256 * 256; };
    const int64_t o_xs = room(M * K), o_wq = o_xs + room(4 * M * nkb), o_ws = o_wq + room(N * K), o_part = o_ws + room(4 * up(N, 128) * nkb);
    const int64_t need = api.cinn_fp8_gemm_workspace_bytes(M, N, K, 0);            // few tiles, long reduction: cut along K
    Tensor buf = empty({o_part + need}, at::kByte, x.device());
    uint8_t* b = buf.data_ptr<uint8_t>();
    float *xs = reinterpret_cast<float*>(b + o_xs), *ws = reinterpret_cast<float*>(b + o_ws);
    check(api.cinn_quant_linear(xf.data_ptr(), tag_of(xf.scalar_type()), xf.stride(0), xf.stride(1), b, xs, round_scale, wf.data_ptr(),
                                tag_of(wf.scalar_type()), wf.stride(0), wf.stride(1), b + o_wq, ws, M, N, K, div, stream()),
          "cinn_quant_linear");
    check(api.cinn_fp8_gemm_ws(b, xs, nkb, b + o_wq, ws, 1, nkb, out.data_ptr(), M, N, K, 0, TAG_BF16, need ? b + o_part : nullptr, need,
                               stream()), "cinn_fp8_gemm");
    return out;
}

namespace {

struct CachedWeight { Tensor q, s, q_t; };      // a weight already in e4m3 (undefined: quantise it here), handed around the node's tensors

class LinearNode : public torch::autograd::Function<LinearNode> {
public:
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const Tensor& weight, bool round_scale, bool kmajor,
                          int64_t div, const CachedWeight* wq) {
        Linear r = linear_forward(x, weight, round_scale, x.requires_grad(), weight.requires_grad(), kmajor, (int)div, wq->q, wq->s,
                                     wq->q_t);
        ctx->save_for_backward({r.x, r.x_scale, r.w, r.w_scale, r.w_t});
        ctx->saved_data["x_shape"] = x.sizes().vec();
        ctx->saved_data["flags"] = (int64_t)((round_scale ? 1 : 0) | (r.x_is_block ? 2 : 0) | (r.x_is_block_t ? 4 : 0) | (kmajor ? 8 : 0) |
                                             ((int64_t)div << 4) | ((int64_t)weight.scalar_type() << 8) |
                                             (x.scalar_type() == at::kFloat ? 1 << 16 : 0));
        return r.out;
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        auto s = ctx->get_saved_variables();
        const int64_t f = ctx->saved_data["flags"].toInt();
        std::vector<Tensor> gx(1);
        Tensor gw;
        as_python_error([&] {
            std::tie(gx, gw) = linear_backward(grads[0], s[0], s[1], s[2], s[3], s[4], ctx->saved_data["x_shape"].toIntVector(), f & 1,
                                                  f & 2, f & 4, (at::ScalarType)(f >> 8 & 255), f & 8, (f >> 4) & 15, ctx->needs_input_grad(0),
                                                  ctx->needs_input_grad(1), f >> 16 & 1 ? at::kFloat : at::kBFloat16);
        });
        return {gx[0], gw, Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

Tensor or_none(const c10::optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); }

}  // namespace

void bind_linear(pybind11::module_& m) {
    using OptT = c10::optional<Tensor>;
    // (out, x, x_scale, w, w_scale, w_t or None, x_is_block, x_is_block_t)
    m.def("linear_forward", [](const Tensor& x, const Tensor& w, bool round_scale, bool need_dgrad, bool need_wgrad, bool kmajor, int div) {
        Linear r = linear_forward(x, w, round_scale, need_dgrad, need_wgrad, kmajor, div, Tensor(), Tensor(), Tensor());
        return std::make_tuple(r.out, r.x, r.x_scale, r.w, r.w_scale, r.w_t.defined() ? OptT(r.w_t) : OptT(), r.x_is_block, r.x_is_block_t);
    });
    m.def("linear_backward", [](const Tensor& g, const Tensor& x, const Tensor& xs, const Tensor& w, const Tensor& ws, const OptT& wt,
                                const std::vector<int64_t>& x_shape, bool round_scale, bool x_is_block, bool x_is_block_t, bool w_fp32,
                                bool kmajor, int div) {
        auto [gx, gw] = linear_backward(g, x, xs, w, ws, or_none(wt), x_shape, round_scale, x_is_block, x_is_block_t,
                                        w_fp32 ? at::kFloat : at::kBFloat16, kmajor, div, true, true, at::kBFloat16);
        return std::make_tuple(gx[0], gw);
    });
    // the differentiable call; without gradients to record nothing is saved and no gradient copies are made
    m.def("linear", [](const Tensor& x, const Tensor& w, bool round_scale, bool kmajor, int div, const OptT& wq, const OptT& ws,
                       const OptT& wqt) {
        const CachedWeight cached{or_none(wq), or_none(ws), or_none(wqt)};
        if (takes_node(x, w))
            return LinearNode::apply(x, w, round_scale, kmajor, (int64_t)div, &cached);
        if (!cached.q.defined()) return linear_inference(x, w, round_scale, div, true);
        return linear_forward(x, w, round_scale, false, false, kmajor, div, cached.q, cached.s, cached.q_t).out;
    });
}

}  // namespace cinnhost
