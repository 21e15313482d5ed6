// The trainable MoE block (layers.MoE, layers.SwiGLU) as two native autograd nodes: the shared expert, and router + routed
// experts + combine.  Written as modules and torch calls the block was 128 launches and 2.7 ms of host time per step at 32 x
// 1024 tokens of 512; as nodes it also stops converting and copying between its parts:
//   - w1 and w2 of a shared expert share one quantisation of x and one of their output gradients, and one GEMM forward and
//     for the weight gradients
//   - tokens are quantised once and their bytes spread to the experts' rows (forward); the rows' gradients come home as one
//     gather pass with the router's part added in it (backward), where autograd's index_select needed an atomic index_add
//   - expert outputs stay in bf16 up to the combine pass, their gradients likewise
//   - gates and balance loss have a kernel for their derivative (csrc/moe_train.cu)
#include "host.h"

namespace cinnhost {

namespace {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// ---------------------------------------------------------------------------------------------------------------------
// shared expert: w3(silu(w1 x) * w2 x) on FP8 linears (reference src/layers.py:15-31 after convert_to_fp8)
// ---------------------------------------------------------------------------------------------------------------------
struct SwiGLUOptions { bool round12, round3, kmajor; int div; };

Tensor swiglu_rounded(const Tensor& h12) {
    const int64_t T = h12.size(0), I = h12.size(1) / 2;
    Tensor h = empty({T, I}, h12.scalar_type(), h12.device());
    check(api.cinn_swiglu_rounded(h12.data_ptr(), h.data_ptr(), tag_of(h12.scalar_type()), T, I, stream()), "cinn_swiglu");
    return h;
}

// Whether SwiGLU can be part of the quantisers next to it, and pays.  It saves a launch and a pass over memory, but a piece of 128 x 128 takes a CTA
// 8 - 10 us, two to an SM at a time: where the pieces do not fill a turn, or just begin a second, the separate passes are shorter.  us from a graph, in
// the quantisers and by itself, forward, dense and routed backward (with its product): 32 pieces 7.6 and 6.1, 10.0 and 6.1, 25.1 and 21.8; 192 10.3
// and 10.2, 14.0 and 12.5, 30.1 and 28.8; 256 10.8 and 11.4, 14.7 and 14.9, 31.5 and 33.2; 384 17.4 and 15.7, 23.5 and 21.3, 48.5 and 48.1; 512 20.9 and
// 19.3, 27.7 and 28.8, 54.7 and 57.3; 2048 67 and 71, 96 and 105, 155 and 166.  Outside a graph a block so small waits for the host, which has a launch
// less to make.
bool swiglu_in_quantisers(const Tensor& h12, bool kmajor, int div) {
    const int64_t T = h12.size(0), I = h12.size(1) / 2, pieces = up(T, 128) * (I / 128);
    const int64_t sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
    if (!(pieces > 3 * sms || (pieces >= 192 && pieces <= 2 * sms)) && capturing()) return false;
    return kmajor && div == CINN_DIV_FULL && h12.element_size() == 2 && tag_of(h12.scalar_type()) >= 0 && T >= 1 && T <= MAX_PADDED_ROWS &&
           I >= 128 && I % 128 == 0 && (reinterpret_cast<uintptr_t>(h12.data_ptr()) & 15) == 0;
}

// Whether the copy of the activations in the experts' tiles may be kept for the backward in place of the row-wise bytes.  It holds up to
// 128 rows more per expert: no more than there are rows, or than an eighth of the experts' e4m3 weights, which are kept as well.  (2048 rows of
// 7168 over 64 experts of 4096 outputs: 73 MB in place of 15, beside weights of 1.9 GB; over 64 of 512, 2048 rows stay row-wise.)
bool segments_fit(int64_t rows, int64_t experts, int64_t d_out) {
    return experts >= 1 && experts <= 1024 && up(rows, 128) + experts <= 65535 && (128 * experts <= rows || 8 * 128 <= d_out);
}

// linear_forward(swiglu_rounded(h12), w, ...) of a weight that wants its gradient
Linear swiglu_linear_forward(const Tensor& h12, const Tensor& w, bool round_scale, bool need_dgrad, int div) {
    const at::Device dev = h12.device();
    const int64_t T = h12.size(0), I = h12.size(1) / 2;
    const Tensor wf = readable(w);
    Linear r;
    r.x_is_block = r.x_is_block_t = true;
    r.x = empty({I, up(T, 16) * 16}, F8, dev);
    r.x_scale = empty({up(T, 128), I / 128}, at::kFloat, dev);
    const Tensor xq = empty({T, I}, F8, dev), xs = empty({T, I / 128}, at::kFloat, dev);
    check(api.cinn_swiglu_rounded_quant_block_t(h12.data_ptr(), tag_of(h12.scalar_type()), T, I, xq.data_ptr(), f32(xs), r.x.data_ptr(),
                                                f32(r.x_scale), round_scale, stream()), "cinn_swiglu_rounded_quant_block_t");
    linear_multiply(r, xq, xs, wf, need_dgrad, true, div, Tensor(), Tensor(), Tensor());
    return r;
}

// x comes in twice, once for w2 and once for w1: each of the two layers returns an input gradient of its own, rounded to bf16
// as the layer by itself rounds it, and autograd adds them up in the order in which it would for two layers.  (One product over
// [dh1 dh2] [w1; w2] rounds once and is 20 us faster at 32768 tokens, but then the block's gradient depends on whether a
// hook, a traced call or a compiled one takes it through its layers: 2e-3 of the gradient.)
struct SwiGLUNode : public torch::autograd::Function<SwiGLUNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor&, const Tensor& w1, const Tensor& w2, const Tensor& w3,
                          const SwiGLUOptions* o) {
        c10::cuda::CUDAGuard guard(x.device());
        const bool gx = x.requires_grad(), g12 = w1.requires_grad() || w2.requires_grad(), g3 = w3.requires_grad(), any = gx || g12;
        const Linear a = linear_forward(x, at::cat({w1, w2}), o->round12, gx, g12, o->kmajor, o->div, Tensor(), Tensor(), Tensor());
        const Tensor h12 = a.out.view({-1, a.out.size(-1)});
        const Linear b = g3 && swiglu_in_quantisers(h12, o->kmajor, o->div)
            ? swiglu_linear_forward(h12, w3, o->round3, any, o->div)
            : linear_forward(swiglu_rounded(h12), w3, o->round3, any, g3, o->kmajor, o->div, Tensor(), Tensor(), Tensor());
        ctx->set_materialize_grads(false);
        if (any || g3) {
            ctx->save_for_backward({a.x, a.x_scale, a.w, a.w_scale, a.w_t, h12, b.x, b.x_scale, b.w, b.w_scale, b.w_t});
            ctx->saved_data["x_shape"] = x.sizes().vec();
            auto flags = [&](bool round, const Linear& l, const Tensor& w) {
                return (int64_t)((round ? 1 : 0) | (l.x_is_block ? 2 : 0) | (l.x_is_block_t ? 4 : 0) | (o->kmajor ? 8 : 0) | (o->div << 4) |
                                 ((int)w.scalar_type() << 8));
            };
            ctx->saved_data["a"] = flags(o->round12, a, w1);
            ctx->saved_data["b"] = flags(o->round3, b, w3);
            ctx->saved_data["x32"] = x.scalar_type() == at::kFloat;
        }
        auto shape = x.sizes().vec();
        shape.back() = w3.size(0);
        return b.out.view(shape);
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        auto s = ctx->get_saved_variables();
        const bool gx = ctx->needs_input_grad(0), g12 = ctx->needs_input_grad(2) || ctx->needs_input_grad(3), g3 = ctx->needs_input_grad(4);
        std::vector<Tensor> dx(2), dh(1);
        Tensor d1, d2, d3;
        // (the block's output is not part of what is differentiated, its balance loss alone is: no gradient, not a zero one)
        if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
        as_python_error([&] {
            auto back = [&](int64_t f, const Tensor& g, int at, at::IntArrayRef shape, bool want_x, bool want_w, at::ScalarType type,
                            int parts) {
                return linear_backward(g, s[at], s[at + 1], s[at + 2], s[at + 3], s[at + 4], shape, f & 1, f & 2, f & 4,
                                       (at::ScalarType)(f >> 8 & 255), f & 8, (int)(f >> 4 & 15), want_x, want_w, type, parts);
            };
            const Tensor& h12 = s[5];
            const int64_t T = h12.size(0), I = h12.size(1) / 2;
            auto split = [&](const Tensor& d12) {
                if (!g12) return;
                const auto halves = at::unsafe_split(d12, I, 0);
                d1 = halves[0];
                d2 = halves[1];
            };
            std::tie(dh, d3) = back(ctx->saved_data["b"].toInt(), grads[0], 6, {T, I}, gx || g12, g3, at::kBFloat16, 1);
            if (!(gx || g12)) return;
            c10::cuda::CUDAGuard guard(h12.device());
            const int64_t f = ctx->saved_data["a"].toInt();
            const auto x_type = ctx->saved_data["x32"].toBool() ? at::kFloat : at::kBFloat16;
            Tensor d12;
            if (swiglu_in_quantisers(h12, f & 8, (int)(f >> 4 & 15)) && (!g12 || f & 4)) {
                const Quantised g{empty({T, 2 * I}, F8, h12.device()), empty({T, 2 * I / 128}, at::kFloat, h12.device())};
                const Quantised g_t{empty({2 * I, up(T, 16) * 16}, F8, h12.device()), empty({2 * I, up(T, 128)}, at::kFloat, h12.device())};
                check(api.cinn_swiglu_rounded_backward_quant_dual(h12.data_ptr(), dh[0].data_ptr(), tag_of(h12.scalar_type()), T, I, g.q.data_ptr(),
                                                                  f32(g.s), g_t.q.data_ptr(), f32(g_t.s), f & 1, stream()),
                      "cinn_swiglu_rounded_backward_quant_dual");
                std::tie(dx, d12) = linear_backward_quantised(g, g_t, T, s[0], s[1], s[2], s[3], s[4], ctx->saved_data["x_shape"].toIntVector(), f & 2,
                                                              f & 4, (at::ScalarType)(f >> 8 & 255), f & 8, (int)(f >> 4 & 15), gx, g12, x_type, 2);
                split(d12);
                return;
            }
            Tensor dh12 = empty({T, 2 * I}, h12.scalar_type(), h12.device());
            check(api.cinn_swiglu_rounded_backward(h12.data_ptr(), dh[0].data_ptr(), dh12.data_ptr(), tag_of(h12.scalar_type()), T, I, stream()),
                  "cinn_swiglu_backward");
            std::tie(dx, d12) = back(f, dh12, 0, ctx->saved_data["x_shape"].toIntVector(), gx, g12, x_type, 2);
            split(d12);
        });
        return {dx[1], dx[0], d1, d2, d3, Tensor()};
    }
};

// ---------------------------------------------------------------------------------------------------------------------
// router, routed experts, combine (reference src/layers.py:56-87, 118-179)
// ---------------------------------------------------------------------------------------------------------------------
struct BlockOptions {
    Tensor bias;                               // (E,) fp32
    Quantised w12, w3;                         // the expert weights in e4m3
    int64_t top_k, batch;
    double alpha;                              // balance loss, 0 = none
    at::ScalarType router_type;                // what the router multiplies in (autocast's type, or x's)
    int div;
    Tensor counts;                             // out: rows per expert
};

// gradients of grouped(x, w) given dy; `covered`: the experts' ranges cover every row (else the others' gradients are zero).
// xs undefined: xq holds the segments that the forward's quantiser left.  h12: dy is the gradient of SwiGLU's result, not of the product
std::tuple<Tensor, Tensor> grouped_backward(const Tensor& dy, const Tensor& xq, const Tensor& xs, const Tensor& wq, const Tensor& ws,
                                            const Tensor& starts, const Tensor& ends, at::ScalarType w_type, bool want_x,
                                            at::ScalarType x_type, int div, bool covered = true, const Tensor& h12 = Tensor()) {
    const int64_t R = dy.size(0), E = wq.size(0), d_out = wq.size(1), d_in = wq.size(2);
    const at::Device dev = dy.device();
    const int64_t *st = starts.data_ptr<int64_t>(), *en = ends.data_ptr<int64_t>();
    const bool segments = !xs.defined();
    const int64_t need = segments ? api.cinn_fp8_grouped_wgrad_segments_scratch_bytes(R, E, d_out)
                                  : api.cinn_fp8_grouped_wgrad_fused_scratch_bytes(R, E, d_in, d_out);
    Tensor scratch = empty({need}, at::kByte, dev), dw = empty({E, d_out, d_in}, w_type, dev);
    Tensor gq = empty({R, d_out}, F8, dev), gs = empty({R, d_out / 128}, at::kFloat, dev);
    const bool one_pass = dy.scalar_type() != at::kFloat;          // both quantisations of dy from one pass: 2-byte gradients
    void* rows_q = one_pass ? gq.data_ptr() : nullptr;
    float* rows_s = one_pass ? f32(gs) : nullptr;
    const int dw_tag = w_type == at::kFloat ? TAG_F32_BF16 : TAG_BF16;
    if (h12.defined())
        check(api.cinn_fp8_grouped_wgrad_swiglu(h12.data_ptr(), dy.data_ptr(), tag_of(dy.scalar_type()), xq.data_ptr(), f32(xs), st, en, E, R, d_in,
                                                d_out / 2, scratch.data_ptr(), need, dw.data_ptr(), dw_tag, rows_q, rows_s, stream()),
              "cinn_fp8_grouped_wgrad_swiglu");
    else if (segments)
        check(api.cinn_fp8_grouped_wgrad_segments(dy.data_ptr(), tag_of(dy.scalar_type()), xq.data_ptr(), E, R, d_in, d_out, scratch.data_ptr(),
                                                  need, dw.data_ptr(), dw_tag, div, rows_q, rows_s, stream()), "cinn_fp8_grouped_wgrad_segments");
    else
        check(api.cinn_fp8_grouped_wgrad_fused(dy.data_ptr(), tag_of(dy.scalar_type()), xq.data_ptr(), f32(xs), st, en, E, R, d_in, d_out,
                                               scratch.data_ptr(), need, dw.data_ptr(), dw_tag, div, rows_q, rows_s, stream()),
              "cinn_fp8_grouped_wgrad_fused");
    Tensor dx;
    if (want_x) {
        if (!one_pass) {
            const Quantised g = rowwise(dy, false, div);
            gq = g.q;
            gs = g.s;
        }
        dx = empty({R, d_in}, x_type, dev);
        if (!covered) {
            check(api.cinn_zero_rows_outside(dx.data_ptr(), R, d_in * dx.element_size(), st, en, E, stream()), "cinn_zero_rows_outside");
        }
        check(api.cinn_fp8_grouped_gemm_dgrad(gq.data_ptr(), f32(gs), wq.data_ptr(), f32(ws), st, en, E, R, d_in, d_out, dx.data_ptr(),
                                              tag_of(x_type), stream()), "cinn_fp8_grouped_gemm_dgrad");
    }
    return {dx, dw};
}

struct BlockNode : public torch::autograd::Function<BlockNode> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& router, const Tensor& w12, const Tensor& w3,
                                 const Tensor& addend, BlockOptions* o) {
        c10::cuda::CUDAGuard guard(x.device());
        at::AutoDispatchBelowAutograd below;
        const at::Device dev = x.device();
        const int64_t T = x.size(0), d = x.size(1), E = router.size(0), k = o->top_k, seq = T / o->batch;
        const Tensor xr = x.to(o->router_type), wr = router.to(o->router_type);
        const Tensor logits = at::mm(xr, wr.t());
        const Routes r = route(logits, o->bias, k);
        const Tensor starts = r.starts(), ends = r.ends();
        const Quantised rows = spread(rowwise(x, false, o->div), r, k);
        const Tensor h12 = grouped(rows, o->w12, starts, ends);
        // Where a backward will come, the weight gradient's copy of the activations comes out of the same pass; it is kept in place of
        // the row-wise bytes (h.s undefined: h.q holds the segments).
        Quantised h;
        Tensor out;
        const bool segments = (w12.requires_grad() || w3.requires_grad() || x.requires_grad()) && swiglu_in_quantisers(h12, true, o->div) &&
                              r.pairs > 0 && h12.size(1) % 512 == 0 && d % 256 == 0 && segments_fit(r.pairs, E, d);
        if (segments) {
            const int64_t I = h12.size(1) / 2, bytes = api.cinn_quant_segments_bytes(r.pairs, E, I);
            const Quantised hq{empty({r.pairs, I}, F8, dev), empty({r.pairs, I / 128}, at::kFloat, dev)};
            h.q = empty({bytes}, at::kByte, dev);
            check(api.cinn_swiglu_quant_segments(h12.data_ptr(), tag_of(h12.scalar_type()), r.pairs, I, starts.data_ptr<int64_t>(),
                                                 ends.data_ptr<int64_t>(), E, hq.q.data_ptr(), f32(hq.s), h.q.data_ptr(), bytes, stream()),
                  "cinn_swiglu_quant_segments");
            out = grouped(hq, o->w3, starts, ends);
        } else {
            h = swiglu_quantised(h12, o->div);
            out = grouped(h, o->w3, starts, ends);
        }
        Tensor y = empty({T, d}, at::kFloat, dev);
        check(api.cinn_moe_combine_add(out.data_ptr(), TAG_BF16, r.pos(), r.gates(), addend.data_ptr(), tag_of(addend.scalar_type()), f32(y),
                                       T, r.pairs, (int)k, d, stream()), "cinn_moe_combine_add");
        Tensor share, loss;
        if (o->alpha > 0) {
            share = empty({o->batch, E}, at::kFloat, dev);
            loss = empty({}, at::kFloat, dev);
            Tensor ws = empty({api.cinn_moe_balance_workspace_bytes(o->batch, seq, (int)E)}, at::kByte, dev);
            check(api.cinn_moe_balance_loss(logits.data_ptr(), tag_of(logits.scalar_type()), r.top.data_ptr<int>(), o->batch, seq, (int)E,
                                            (int)k, (float)o->alpha, ws.data_ptr(), f32(share), f32(loss), stream()), "cinn_moe_balance_loss");
        }
        o->counts = r.counts();
        ctx->save_for_backward({xr, wr, logits, r.longs, r.floats, rows.q, rows.s, h12, h.q, h.s, out, o->w12.q, o->w12.s, o->w3.q, o->w3.s,
                                share});
        ctx->saved_data["n"] = std::vector<int64_t>{k, o->batch, o->div, (int64_t)x.scalar_type(), (int64_t)router.scalar_type(),
                                                    (int64_t)w12.scalar_type(), (int64_t)w3.scalar_type(), (int64_t)addend.scalar_type()};
        ctx->saved_data["alpha"] = o->alpha;
        ctx->set_materialize_grads(false);
        if (loss.defined()) return {y, loss};
        return {y};
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        auto s = ctx->get_saved_variables();
        const auto n = ctx->saved_data["n"].toIntVector();
        const int64_t k = n[0], batch = n[1];
        const int div = (int)n[2];
        const auto type = [&](int i) { return (at::ScalarType)n[i]; };
        const float alpha = (float)ctx->saved_data["alpha"].toDouble();
        Tensor dx, d_router, dw12, dw3, d_add;
        as_python_error([&] {
            const Tensor &xr = s[0], &wr = s[1], &logits = s[2], &h12 = s[7], &out = s[10];
            c10::cuda::CUDAGuard guard(xr.device());
            const at::Device dev = xr.device();
            const int64_t T = xr.size(0), d = xr.size(1), E = wr.size(0), seq = T / batch;
            Routes r;
            r.longs = s[3]; r.floats = s[4]; r.pairs = T * k; r.E = E;
            const Tensor starts = r.starts(), ends = r.ends();
            const bool want_x = ctx->needs_input_grad(0), want_r = ctx->needs_input_grad(1), want_12 = ctx->needs_input_grad(2);
            const bool want_3 = ctx->needs_input_grad(3);
            Tensor d_gates, d_rows;
            if (grads[0].defined()) {
                const Tensor dy = grads[0].to(at::kFloat).contiguous();
                if (ctx->needs_input_grad(4)) d_add = dy.to(type(7));
                if (want_x || want_r || want_12 || want_3) {
                    Tensor d_out = empty({r.pairs, d}, at::kBFloat16, dev);
                    d_gates = empty({T, k}, at::kFloat, dev);
                    check(api.cinn_moe_combine_backward(out.data_ptr(), TAG_BF16, r.pos(), r.gates(), f32(dy), d_out.data_ptr(), f32(d_gates),
                                                        T, r.pairs, (int)k, d, stream()), "cinn_moe_combine_backward");
                    const bool below = want_x || want_12;
                    Tensor dh;
                    std::tie(dh, dw3) = grouped_backward(d_out, s[8], s[9], s[13], s[14], starts, ends, type(6), below, at::kBFloat16, div);
                    d_out.reset();
                    if (below) {
                        const int64_t I = h12.size(1) / 2;
                        if (!s[9].defined()) {             // the widths and the division flavour were found to fit in the forward
                            std::tie(d_rows, dw12) = grouped_backward(dh, s[5], s[6], s[11], s[12], starts, ends, type(5), want_x, type(3), div,
                                                                      true, h12);
                        } else {
                            Tensor dh12 = empty({r.pairs, 2 * I}, at::kBFloat16, dev);
                            check(api.cinn_swiglu_backward(h12.data_ptr(), dh.data_ptr(), dh12.data_ptr(), TAG_BF16, r.pairs, I, stream()),
                                  "cinn_swiglu_backward");
                            std::tie(d_rows, dw12) = grouped_backward(dh12, s[5], s[6], s[11], s[12], starts, ends, type(5), want_x,
                                                                      type(3), div);
                        }
                    }
                }
            }
            const bool loss = grads.size() > 1 && grads[1].defined();
            Tensor dxr;
            if ((want_x || want_r) && (loss || d_gates.defined())) {
                Tensor d_logits = empty({T, E}, logits.scalar_type(), dev);
                const Tensor dl = loss ? grads[1].to(at::kFloat) : Tensor();
                check(api.cinn_moe_gates_backward(logits.data_ptr(), tag_of(logits.scalar_type()), r.sorted_experts(), r.pos(),
                                                  d_gates.defined() ? f32(d_gates) : nullptr, loss ? f32(s[15]) : nullptr,
                                                  loss ? f32(dl) : nullptr, alpha, batch, seq, (int)E, (int)k, d_logits.data_ptr(), stream()),
                      "cinn_moe_gates_backward");
                if (want_r) d_router = at::mm(d_logits.t(), xr).to(type(4));
                if (want_x) dxr = at::mm(d_logits, wr);
            }
            if (want_x && d_rows.defined()) {
                dx = empty({T, d}, at::kFloat, dev);
                check(api.cinn_moe_sum_add(d_rows.data_ptr(), tag_of(d_rows.scalar_type()), r.pos(), dxr.data_ptr(), tag_of(dxr.scalar_type()),
                                           f32(dx), T, r.pairs, (int)k, d, stream()), "cinn_moe_sum_add");
            } else {
                dx = dxr;
            }
            if (dx.defined()) dx = dx.to(type(3));
        });
        return {dx, d_router, dw12, dw3, d_add, Tensor()};
    }
};

// ---------------------------------------------------------------------------------------------------------------------
// moe_grouped_gemm (reference src/kernels.py:526-581) with its gradients
// ---------------------------------------------------------------------------------------------------------------------
struct GroupedNode : public torch::autograd::Function<GroupedNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x_in, const Tensor& w, const Tensor& starts_in, const Tensor& ends_in,
                          const Quantised* wq, at::ScalarType type, int64_t div) {
        c10::cuda::CUDAGuard guard(x_in.device());
        at::AutoDispatchBelowAutograd below;
        const Tensor x = readable(x_in), starts = starts_in.to(at::kLong).contiguous(), ends = ends_in.to(at::kLong).contiguous();
        const int64_t R = x.size(0), E = wq->q.size(0), d = x.dim() == 2 ? x.size(1) : 0;
        // Where the weight gradient can be had (its widths are multiples of 256) its copy of x comes out of the forward's pass.
        const bool segments = w.requires_grad() && x.dim() == 2 && x.element_size() == 2 && x.is_contiguous() && R > 0 && d == wq->q.size(2) &&
                              d % 256 == 0 && wq->q.size(1) % 256 == 0 && segments_fit(R, E, wq->q.size(1)) &&
                              starts.numel() == E && ends.numel() == E && (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15) == 0;
        Quantised xq;
        if (segments) {
            const int64_t bytes = api.cinn_quant_segments_bytes(R, E, d);
            Tensor seg = empty({bytes}, at::kByte, x.device());
            xq = {empty({R, d}, F8, x.device()), empty({R, d / 128}, at::kFloat, x.device())};
            check(api.cinn_quant_rowwise_segments(x.data_ptr(), tag_of(x.scalar_type()), R, d, starts.data_ptr<int64_t>(), ends.data_ptr<int64_t>(),
                                                  E, xq.q.data_ptr(), f32(xq.s), seg.data_ptr(), bytes, (int)div, stream()),
                  "cinn_quant_rowwise_segments");
            ctx->save_for_backward({seg, Tensor(), wq->q, wq->s, starts, ends});
        } else {
            xq = rowwise(x, false, (int)div);
            ctx->save_for_backward({xq.q, xq.s, wq->q, wq->s, starts, ends});
        }
        ctx->saved_data["n"] = std::vector<int64_t>{(int64_t)x_in.scalar_type(), (int64_t)w.scalar_type(), div};
        return grouped(xq, *wq, starts, ends, type);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        auto s = ctx->get_saved_variables();
        const auto n = ctx->saved_data["n"].toIntVector();
        Tensor dx, dw;
        as_python_error([&] {
            c10::cuda::CUDAGuard guard(s[2].device());
            const Tensor dy = readable(grads[0]).contiguous();
            const auto x_type = (at::ScalarType)n[0], w_type = (at::ScalarType)n[1];
            const auto dx_type = tag_of(x_type) < 0 ? at::kFloat : x_type;
            const auto dw_type = w_type == at::kBFloat16 ? at::kBFloat16 : at::kFloat;
            std::tie(dx, dw) = grouped_backward(dy, s[0], s[1], s[2], s[3], s[4], s[5], dw_type, ctx->needs_input_grad(0), dx_type, (int)n[2],
                                                false);
            if (dx.defined()) dx = dx.to(x_type);
            dw = dw.to(w_type);
        });
        return {dx, dw, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

}  // namespace

void bind_moe_train(pybind11::module_& m) {
    m.def("swiglu_block", [](const Tensor& x, const Tensor& w1, const Tensor& w2, const Tensor& w3, bool round12, bool round3, bool kmajor,
                             int div) {
        // Nothing is kept for a backward; with gradients or without, the same numbers.  Its linears quantise and multiply in two launches on any
        // number of rows: the one-kernel form has the same bits, but this call's five launches are part of what it promises.
        if (!takes_node(x, w1, w2, w3)) {
            const Tensor h12 = linear_inference(x, at::cat({w1, w2}), round12, div, false);
            c10::cuda::CUDAGuard guard(x.device());
            Tensor y = linear_inference(swiglu_rounded(h12.view({-1, h12.size(-1)})), w3, round3, div, false);
            auto shape = x.sizes().vec();
            shape.back() = w3.size(0);
            return y.view(shape);
        }
        const SwiGLUOptions o{round12, round3, kmajor, div};
        return SwiGLUNode::apply(x, x, w1, w2, w3, &o);
    });
    m.def("grouped_gemm", [](const Tensor& x, const Tensor& w, const Tensor& starts, const Tensor& ends, const Tensor& w_q, const Tensor& w_s,
                             int tag, int div) {
        const Quantised q{w_q, w_s};
        const auto type = tag == TAG_BF16 ? at::kBFloat16 : (tag == TAG_F16 ? at::kHalf : at::kFloat);
        if (at::GradMode::is_enabled() && (x.requires_grad() || w.requires_grad()))
            return GroupedNode::apply(x, w, starts, ends, &q, type, (int64_t)div);
        c10::cuda::CUDAGuard guard(x.device());
        return grouped(rowwise(readable(x), false, div), q, starts.to(at::kLong).contiguous(), ends.to(at::kLong).contiguous(), type);
    });
    // (y, balance loss or None, rows per expert)
    m.def("moe_block", [](const Tensor& x, const Tensor& router, const Tensor& w12, const Tensor& w3, const Tensor& addend,
                          const Tensor& bias, const Tensor& w12_q, const Tensor& w12_s, const Tensor& w3_q, const Tensor& w3_s, int64_t top_k,
                          int64_t batch, double alpha, bool cast_router, int div) {
        check_layer(x, router, bias, {w12_q, w12_s}, {w3_q, w3_s});
        require(addend.device() == x.device() && addend.sizes() == x.sizes(), "MoE: the shared experts' output does not fit the input");
        BlockOptions o{bias, {w12_q, w12_s}, {w3_q, w3_s}, top_k, batch, alpha,
                       cast_router ? at::autocast::get_autocast_dtype(at::kCUDA) : x.scalar_type(), div, Tensor()};
        auto r = BlockNode::apply(x, router, w12, w3, addend, &o);
        return std::make_tuple(r[0], r.size() > 1 ? c10::optional<Tensor>(r[1]) : c10::optional<Tensor>(), o.counts);
    });
    m.def("moe_update_bias", [](Tensor bias, const Tensor& counts, double expected, double gamma) {
        c10::cuda::CUDAGuard guard(bias.device());
        check(api.cinn_moe_update_bias(counts.data_ptr<int64_t>(), f32(bias), (int)bias.numel(), (float)expected, (float)gamma, stream()),
              "cinn_moe_update_bias");
        bias.unsafeGetTensorImpl()->bump_version();
    });
}

}  // namespace cinnhost
