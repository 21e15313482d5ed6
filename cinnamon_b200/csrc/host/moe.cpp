// The MoE layer on one GPU, forward only (moe.ExpertParallelMoE): router, routing, routed experts, shared expert and the
// combine pass as one native call.  Generating for 64 sequences the layer is 0.7 ms of kernels; driven from Python, its
// calls took 0.47 ms of host time, more than the kernels around the grouped GEMMs could hide.
#include "host.h"

namespace cinnhost {

Quantised rowwise(const Tensor& x, bool round_scale, int div) {
    const int64_t M = x.size(0), K = x.size(1);
    Quantised r{empty({M, K}, F8, x.device()), empty({M, up(K, 128)}, at::kFloat, x.device())};
    check(api.cinn_quant_rowwise(x.data_ptr(), tag_of(x.scalar_type()), M, K, x.stride(0), x.stride(1), r.q.data_ptr(), f32(r.s), 128,
                                 round_scale, div, stream()), "cinn_quant_rowwise");
    return r;
}

Quantised swiglu_quantised(const Tensor& h12, int div) {
    const int64_t T = h12.size(0), I = h12.size(1) / 2;
    Quantised r{empty({T, I}, F8, h12.device()), empty({T, up(I, 128)}, at::kFloat, h12.device())};
    check(api.cinn_swiglu_quant_rowwise(h12.data_ptr(), tag_of(h12.scalar_type()), T, I, r.q.data_ptr(), f32(r.s), div, stream()),
          "cinn_swiglu_quant_rowwise");
    return r;
}

Tensor grouped(const Quantised& x, const Quantised& w, const Tensor& starts, const Tensor& ends, at::ScalarType type) {
    const int64_t T = x.q.size(0), E = w.q.size(0), d_out = w.q.size(1), d_in = w.q.size(2);
    Tensor out = empty({T, d_out}, type, x.q.device());
    check(api.cinn_fp8_grouped_gemm(x.q.data_ptr(), f32(x.s), w.q.data_ptr(), f32(w.s), starts.data_ptr<int64_t>(),
                                    ends.data_ptr<int64_t>(), E, T, d_in, d_out, out.data_ptr(), tag_of(type), stream()),
          "cinn_fp8_grouped_gemm");
    return out;
}

void check_layer(const Tensor& x, const Tensor& router, const Tensor& bias, const Quantised& w12, const Quantised& w3) {
    const auto dev = x.device();
    require(x.is_cuda() && router.is_cuda() && bias.is_cuda(), "Inputs must be on CUDA");
    require(router.device() == dev && bias.device() == dev && w12.q.device() == dev && w3.q.device() == dev && w12.s.device() == dev &&
                w3.s.device() == dev, "MoE: input, router and experts must be on the same device");
    const int64_t E = router.size(0), d = x.size(1);
    require(router.size(1) == d && bias.numel() == E && w12.q.size(0) == E && w3.q.size(0) == E && w12.q.size(2) == d &&
                w3.q.size(1) == d && w12.q.size(1) == 2 * w3.q.size(2), "MoE: the widths of input, router and experts do not fit together");
}

Routes route(const Tensor& logits_in, const Tensor& bias, int64_t top_k) {
    const Tensor logits = readable(logits_in).contiguous(), b = bias.to(at::kFloat).contiguous();
    const int64_t T = logits.size(0), E = logits.size(1);
    const at::Device dev = logits.device();
    Routes r;
    r.pairs = T * top_k;
    r.E = E;
    r.longs = empty({3 * r.pairs + 3 * E}, at::kLong, dev);
    r.floats = empty({2 * r.pairs}, at::kFloat, dev);
    r.top = empty({r.pairs}, at::kInt, dev);
    Tensor ws = empty({std::max<int64_t>(1, api.cinn_moe_route_workspace_ints(T, (int)E))}, at::kInt, dev);
    Tensor top_gates = empty({r.pairs}, at::kFloat, dev);
    check(api.cinn_moe_route_ranges(logits.data_ptr(), tag_of(logits.scalar_type()), f32(b), T, (int)E, (int)top_k, ws.data_ptr<int>(),
                                    r.top.data_ptr<int>(), f32(top_gates), r.token_indices(), f32(r.floats), r.sorted_experts(),
                                    r.part(3 * r.pairs), r.part(3 * r.pairs + E), r.part(3 * r.pairs + 2 * E), r.pos(), r.gates(),
                                    stream()), "cinn_moe_route");
    return r;
}

// quantised tokens to the rows of their pairs
Quantised spread(const Quantised& x, const Routes& r, int64_t top_k) {
    const int64_t T = x.q.size(0), d = x.q.size(1), ns = x.s.size(1);
    Quantised rows{empty({r.pairs, d}, F8, x.q.device()), empty({r.pairs, ns}, at::kFloat, x.q.device())};
    check(api.cinn_spread_rows(x.q.data_ptr(), f32(x.s), r.pos(), rows.q.data_ptr(), f32(rows.s), T, r.pairs, (int)top_k, d, ns, stream()),
          "cinn_spread_rows");
    return rows;
}

namespace {

// A GEMM that is not cut along K: a rank of an expert-parallel job runs the shared expert on its share of the tokens, and a token
// gets the same bits there as on one GPU with all of them.  (Cut along K, the layer takes 910 us instead of 916 for 64 tokens of
// 7168 and 256 experts.)
Tensor gemm_whole(const Tensor& a, const Tensor& sa, const Tensor& b, const Tensor& sb, int64_t M, int64_t N, int64_t K) {
    Tensor out = empty({M, N}, at::kBFloat16, a.device());
    check(api.cinn_fp8_gemm_ws(a.data_ptr(), f32(sa), sa.stride(0), b.data_ptr(), f32(sb), sb.stride(1), sb.stride(0), out.data_ptr(), M, N, K, 0,
                               TAG_BF16, nullptr, 0, stream()), "cinn_fp8_gemm");
    return out;
}

// x (T, d), contiguous; router (E, d) in the type the logits are computed in; the weights as FP8Experts and FP8SwiGLU hold
// them.  Returns (T, d) fp32.
Tensor forward(const Tensor& x, const Tensor& router, const Tensor& bias, int64_t top_k, const Quantised& w12, const Quantised& w3,
               const Quantised& sw12, const Quantised& sw3, bool shared_round, int div) {
    check_layer(x, router, bias, w12, w3);
    require(!sw12.q.defined() || (sw12.q.device() == x.device() && sw12.q.size(1) == x.size(1) && sw3.q.size(0) == x.size(1) &&
                                  sw12.q.size(0) == 2 * sw3.q.size(1)), "MoE: the shared expert does not fit the input");
    c10::cuda::CUDAGuard guard(x.device());
    at::NoGradGuard no_grad;
    const at::Device dev = x.device();
    const int64_t T = x.size(0), d = x.size(1), E = router.size(0);
    const Quantised xq = rowwise(x, false, div);
    Tensor shared;
    if (sw12.q.defined()) {
        const Quantised xs = shared_round ? rowwise(x, true, div) : xq;
        const int64_t I2 = sw12.q.size(0);
        const Quantised h = swiglu_quantised(gemm_whole(xs.q, xs.s, sw12.q, sw12.s, T, I2, d), div);
        shared = gemm_whole(h.q, h.s, sw3.q, sw3.s, T, d, I2 / 2);
    }
    Tensor logits = at::mm(x, router.to(x.scalar_type()).t());
    const Routes r = route(logits, bias, top_k);
    const Tensor starts = r.starts(), ends = r.ends();
    const int64_t pairs = r.pairs, *pos = r.pos();
    Quantised rows = spread(xq, r, top_k);
    Tensor h12 = grouped(rows, w12, starts, ends);
    rows = Quantised{};
    const Quantised h = swiglu_quantised(h12, div);
    h12.reset();
    const Tensor out = grouped(h, w3, starts, ends);
    Tensor y = empty({T, d}, at::kFloat, dev);
    if (shared.defined())
        check(api.cinn_moe_combine_add(out.data_ptr(), TAG_BF16, pos, r.gates(), shared.data_ptr(), TAG_BF16, f32(y), T, pairs,
                                       (int)top_k, d, stream()), "cinn_moe_combine_add");
    else
        check(api.cinn_moe_combine(out.data_ptr(), TAG_BF16, pos, r.gates(), f32(y), T, pairs, (int)top_k, d, stream()),
              "cinn_moe_combine");
    return y;
}

}  // namespace

void bind_moe(pybind11::module_& m) {
    using OptT = c10::optional<Tensor>;
    m.def("moe_forward", [](const Tensor& x, const Tensor& router, const Tensor& bias, int64_t top_k, const Tensor& w12_q, const Tensor& w12_s,
                            const Tensor& w3_q, const Tensor& w3_s, const OptT& sw12_q, const OptT& sw12_s, const OptT& sw3_q,
                            const OptT& sw3_s, bool shared_round, int div) {
        auto get = [](const OptT& t) { return t.has_value() ? *t : Tensor(); };
        return forward(x, router, bias, top_k, {w12_q, w12_s}, {w3_q, w3_s}, {get(sw12_q), get(sw12_s)}, {get(sw3_q), get(sw3_s)},
                       shared_round, div);
    });
}

}  // namespace cinnhost
