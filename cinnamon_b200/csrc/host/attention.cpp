// Sparse attention over index lists (reference src/kernels.py:1189-1312): forward and backward as one native call each,
// and as a native autograd node.
#include "host.h"

namespace cinnhost {

namespace {

// The tiles' scratch; undefined where they need none, or where there is no room for it: the gather kernels, which need none,
// compute the call then.
Tensor scratch(int64_t bytes, const at::Device& dev) {
    if (!bytes) return Tensor();
    try {
        return empty({bytes}, at::kByte, dev);
    } catch (const c10::OutOfMemoryError&) {
        return Tensor();
    }
}

struct Attention { Tensor out, attn, q, k, v, idx, out32, lse; };

Attention forward(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& idx_in, double scale) {
    require(q_in.is_cuda() && k_in.is_cuda() && v_in.is_cuda() && idx_in.is_cuda(), "Inputs must be on CUDA");
    c10::cuda::CUDAGuard guard(q_in.device());
    const at::Device dev = q_in.device();
    const at::ScalarType in = q_in.scalar_type(), work = tag_of(in) < 0 ? at::kFloat : in;
    Attention r;
    r.q = q_in.to(work).contiguous();
    r.k = k_in.to(work).contiguous();
    r.v = v_in.to(work).contiguous();
    r.idx = idx_in.to(at::kLong).contiguous();
    const int64_t B = r.q.size(0), H = r.q.size(1), L = r.q.size(2), Dqk = r.q.size(3), Dv = r.v.size(-1), K = r.idx.size(-1);
    r.out32 = empty({B, H, L, Dv}, at::kFloat, dev);
    r.lse = empty({B, H, L}, at::kFloat, dev);
    r.attn = empty({B, H, L, K}, at::kFloat, dev);
    const bool cast = work != at::kFloat;
    r.out = cast ? empty({B, H, L, Dv}, work, dev) : r.out32;
    int64_t need = api.cinn_sparse_attn_workspace_bytes(B, H, L, K, Dqk, Dv, tag_of(work), 0);
    const Tensor ws = scratch(need, dev);
    if (!ws.defined()) need = 0;
    check(api.cinn_sparse_attn_fwd_ws(r.q.data_ptr(), r.k.data_ptr(), r.v.data_ptr(), tag_of(work), r.idx.data_ptr<int64_t>(), f32(r.out32),
                                      cast ? r.out.data_ptr() : nullptr, f32(r.lse), f32(r.attn), B, H, L, K, Dqk, Dv, (float)scale,
                                      need ? ws.data_ptr() : nullptr, need, stream()), "cinn_sparse_attn_fwd");
    if (in != work) r.out = r.out32.to(in);
    return r;
}

std::tuple<Tensor, Tensor, Tensor> backward(const Tensor& grad_out, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                                            const Tensor& out32, const Tensor& lse, double scale, at::ScalarType in) {
    c10::cuda::CUDAGuard guard(q.device());
    const int64_t B = q.size(0), H = q.size(1), L = q.size(2), Dqk = q.size(3), Dv = v.size(-1), K = idx.size(-1);
    Tensor g = grad_out.contiguous();
    const int tag = tag_of(q.scalar_type());
    const int64_t need = api.cinn_sparse_attn_workspace_bytes(B, H, L, K, Dqk, Dv, tag, 1);
    const auto odd = [](const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) != 0; };
    const bool tiles = need && g.scalar_type() == q.scalar_type() && !(odd(q) || odd(k) || odd(v) || odd(g));
    if (const Tensor ws = scratch(tiles ? need : 0, q.device()); ws.defined()) {
        Tensor gq = empty({B, H, L, Dqk}, q.scalar_type(), q.device()), gk = empty({B, H, L, Dqk}, q.scalar_type(), q.device());
        Tensor gv = empty({B, H, L, Dv}, q.scalar_type(), q.device());
        check(api.cinn_sparse_attn_bwd_ws(g.data_ptr(), f32(out32), f32(lse), q.data_ptr(), k.data_ptr(), v.data_ptr(), tag,
                                          idx.data_ptr<int64_t>(), gq.data_ptr(), gk.data_ptr(), gv.data_ptr(), B, H, L, K, Dqk, Dv,
                                          (float)scale, ws.data_ptr(), need, stream()), "cinn_sparse_attn_bwd");
        if (in == q.scalar_type()) return {gq, gk, gv};
        return {gq.to(in), gk.to(in), gv.to(in)};
    }
    if (g.scalar_type() != q.scalar_type() && g.scalar_type() != at::kFloat) g = g.to(at::kFloat);
    Tensor gq = empty({B, H, L, Dqk}, at::kFloat, q.device());
    Tensor gk = empty({B, H, L, Dqk}, at::kFloat, q.device()).zero_();            // accumulated into
    Tensor gv = empty({B, H, L, Dv}, at::kFloat, q.device()).zero_();
    check(api.cinn_sparse_attn_bwd(g.data_ptr(), tag_of(g.scalar_type()), f32(out32), f32(lse), q.data_ptr(), k.data_ptr(), v.data_ptr(),
                                   tag_of(q.scalar_type()), idx.data_ptr<int64_t>(), f32(gq), f32(gk), f32(gv), B, H, L, K, Dqk, Dv,
                                   (float)scale, stream()), "cinn_sparse_attn_bwd");
    return {gq.to(in), gk.to(in), gv.to(in)};
}

// Lightning indexer logits (reference src/kernels.py:392-433); q (B, Lq, H, d), k (B, Lk, d), w (B, Lq, H), any strides
Tensor indexer(const Tensor& q_in, const Tensor& k_in, const Tensor& w_in) {
    require(q_in.is_cuda() && k_in.is_cuda() && w_in.is_cuda(), "Inputs must be on CUDA");
    c10::cuda::CUDAGuard guard(q_in.device());
    const at::ScalarType in = q_in.scalar_type(), work = tag_of(in) < 0 ? at::kFloat : in;
    const Tensor q = q_in.to(work), k = k_in.to(work), w = w_in.to(work);
    Tensor out = empty({q.size(0), q.size(1), k.size(1)}, at::kHalf, q.device());
    check(api.cinn_lightning_indexer(q.data_ptr(), k.data_ptr(), w.data_ptr(), tag_of(work), out.data_ptr(), q.size(0), q.size(1), k.size(1),
                                     q.size(2), q.size(3), q.strides().data(), k.strides().data(), w.strides().data(), stream()),
          "cinn_lightning_indexer");
    return out;
}

class AttentionNode : public torch::autograd::Function<AttentionNode> {
public:
    static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v,
                                                  const Tensor& idx, double scale) {
        Attention r = cinnhost::forward(q, k, v, idx, scale);
        ctx->save_for_backward({r.q, r.k, r.v, r.idx, r.out32, r.lse});
        ctx->saved_data["scale"] = scale;
        ctx->saved_data["dtype"] = (int64_t)q.scalar_type();
        ctx->mark_non_differentiable({r.attn});
        return {r.out, r.attn};
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        auto s = ctx->get_saved_variables();
        Tensor gq, gk, gv;
        as_python_error([&] {
            std::tie(gq, gk, gv) = cinnhost::backward(grads[0], s[0], s[1], s[2], s[3], s[4], s[5], ctx->saved_data["scale"].toDouble(),
                                                      (at::ScalarType)ctx->saved_data["dtype"].toInt());
        });
        return {gq, gk, gv, Tensor(), Tensor()};
    }
};

}  // namespace

void bind_attention(pybind11::module_& m) {
    m.def("indexer", &indexer);
    // (out, attention weights, then what the backward takes: q, k, v, idx, out in fp32, lse)
    m.def("attention_forward", [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, double scale) {
        Attention r = forward(q, k, v, idx, scale);
        return std::make_tuple(r.out, r.attn, r.q, r.k, r.v, r.idx, r.out32, r.lse);
    });
    m.def("attention_backward", [](const Tensor& g, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, const Tensor& out32,
                                   const Tensor& lse, double scale, const Tensor& like) {
        return backward(g, q, k, v, idx, out32, lse, scale, like.scalar_type());
    });
    m.def("attention", [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, double scale) {
        if (takes_node(q, k, v)) {
            auto r = AttentionNode::apply(q, k, v, idx, scale);
            return std::make_tuple(r[0], r[1]);
        }
        Attention r = forward(q, k, v, idx, scale);
        return std::make_tuple(r.out, r.attn);
    });
}

}  // namespace cinnhost
