"""The calls this framework is used for, as timed cases over the public entry points.

Each case is one call (or one forward + backward) that a training or serving program makes:

  linear_fwd     ``FP8Linear`` without gradients: evaluation, prefill and small-batch inference
  linear_train   ``FP8Linear`` forward and both gradients: a training step's share of one layer
  grouped_train  ``moe_grouped_gemm`` over ragged experts, forward and both gradients
  moe_serve      ``ExpertParallelMoE`` on one GPU: routing, routed experts, shared expert, combine
  moe_train      the trainable ``layers.MoE`` block under bf16 autocast, forward and every gradient
  attn_fwd       ``sparse_attention`` without gradients
  attn_train     ``sparse_attention`` forward and the gradients of q, k and v
  indexer        ``lightning_indexer_fused``: the logits that choose the keys

Sizes are those of the repository's benchmark configurations (a 512-wide model trained on 32 x 1024 tokens, a
7168-wide feed-forward and attention projections on 16384 tokens, 256 experts on 32768 tokens) and of its tests;
``draw`` spreads over the ranges between them.
"""
import math

import numpy as np
import torch

from cinnamon_b200 import kernels as K
from cinnamon_b200 import layers, moe

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
ITEM = {"bf16": 2, "fp32": 4}


def listed():
    return [
        # a projection of a narrow model on a short prompt: launches and host work are all there is
        dict(name="linear_prompt", kind="linear_fwd", tokens=128, d_in=512, d_out=1024, round_scale=False),
        # the benchmark's single-layer forward: one 4096-token sequence through a narrow feed-forward
        dict(name="linear_4096", kind="linear_fwd", tokens=4096, d_in=512, d_out=2048, round_scale=False),
        # the narrow model's shared-expert projection in training: 32 x 1024 tokens, power-of-two scales
        dict(name="linear_train_narrow", kind="linear_train", tokens=32768, d_in=512, d_out=1024, round_scale=True),
        # the joint latent projection of wide attention: few output columns, not a multiple of 128
        dict(name="linear_train_latent", kind="linear_train", tokens=16384, d_in=7168, d_out=576, round_scale=False),
        # the wide feed-forward layer of the headline benchmark
        dict(name="linear_train_ffn", kind="linear_train", tokens=16384, d_in=7168, d_out=18432, round_scale=False),
        # up-projection of one rank's 32 experts in training, about 1024 rows each, ragged
        dict(name="grouped_train", kind="grouped_train", experts=32, rows=32768, d_in=7168, d_out=4096),
        # the whole MoE layer on a prefill batch with a strongly skewed router (the benchmark's bias ~ N(0, 1))
        dict(name="moe_prefill", kind="moe_serve", tokens=32768, experts=256, d=7168, inter=2048, top_k=8, bias_std=1.0),
        # the same layer generating for 64 sequences: a couple of rows per expert, every expert's weights are read
        dict(name="moe_decode", kind="moe_serve", tokens=64, experts=256, d=7168, inter=2048, top_k=8, bias_std=0.1),
        # the narrow model's MoE block in training
        dict(name="moe_train_narrow", kind="moe_train", batch=32, seq=1024, experts=16, d=512, hidden=1024, top_k=2),
        # the narrow model's attention in training: fp32 tensors, 192-wide queries and keys, 64-wide values
        dict(name="attn_train", kind="attn_train", batch=32, heads=8, seq=1024, topk=128, d_qk=192, d_v=64, dtype="fp32"),
        # evaluation on prompts of an odd length in bf16
        dict(name="attn_eval_ragged", kind="attn_fwd", batch=8, heads=8, seq=1531, topk=128, d_qk=192, d_v=64, dtype="bf16"),
        # indexer logits of the narrow model: four heads of 64
        dict(name="indexer", kind="indexer", batch=8, seq=1024, heads=4, d=64, dtype="bf16"),
    ]


def _log(rng, lo, hi, step=1):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step
    return min(max(v, lo), hi)


def draw(rng):
    while True:
        case = _draw(rng)
        if _cost(case) <= 1.0:
            return case


def _draw(rng):
    kind = rng.choice(["linear_fwd", "linear_fwd", "linear_train", "linear_train", "grouped_train", "moe_serve", "moe_serve",
                       "moe_train", "attn_train", "attn_fwd", "indexer"])
    if kind in ("linear_fwd", "linear_train"):
        # widths in steps of 64 as projections have them (576, 1536, 7168 ...), any number of tokens
        return dict(kind=kind, tokens=_log(rng, 1 if kind == "linear_fwd" else 256, 32768), d_in=_log(rng, 256, 7168, 64),
                    d_out=_log(rng, 256, 18432, 64), round_scale=rng.random() < 0.3)
    if kind == "grouped_train":
        return dict(kind=kind, experts=rng.choice([8, 16, 32, 64]), rows=_log(rng, 2048, 65536), d_in=_log(rng, 512, 7168, 256),
                    d_out=_log(rng, 512, 4096, 256))
    if kind == "moe_serve":
        return dict(kind=kind, tokens=_log(rng, 1, 32768), experts=rng.choice([64, 128, 256]), d=_log(rng, 1024, 7168, 256),
                    inter=_log(rng, 512, 2048, 128), top_k=rng.choice([2, 4, 6, 8]), bias_std=rng.choice([0.0, 0.1, 1.0]))
    if kind == "moe_train":
        return dict(kind=kind, batch=rng.choice([2, 4, 8, 16, 32]), seq=_log(rng, 128, 2048), experts=rng.choice([8, 16, 32, 64]),
                    d=_log(rng, 512, 2048, 256), hidden=_log(rng, 1024, 4096, 512), top_k=rng.choice([2, 4, 6]))
    if kind in ("attn_train", "attn_fwd"):
        return dict(kind=kind, batch=rng.choice([1, 2, 4, 8, 16, 32]), heads=rng.choice([4, 8, 16]), seq=_log(rng, 256, 4096),
                    topk=rng.choice([32, 64, 128, 256]), d_qk=rng.choice([64, 128, 192]), d_v=rng.choice([64, 128]),
                    dtype=rng.choice(["bf16", "fp32"]))
    return dict(kind=kind, batch=rng.choice([1, 2, 4, 8, 16, 32]), seq=_log(rng, 256, 4096), heads=rng.choice([2, 4, 8]),
                d=rng.choice([64, 128]), dtype=rng.choice(["bf16", "fp32"]))


def _cost(case):
    """Work of a drawn case as a share of what the largest listed case of such calls does."""
    k = case["kind"]
    if k.startswith("linear"):
        return case["tokens"] * case["d_in"] * case["d_out"] / (16384 * 7168 * 18432)
    if k == "grouped_train":
        return max(case["rows"] * case["d_in"] * case["d_out"] / (32768 * 7168 * 4096),
                   case["experts"] * case["d_in"] * case["d_out"] / (32 * 7168 * 4096))
    if k == "moe_serve":
        return 1.0
    if k == "moe_train":
        return case["batch"] * case["seq"] * case["top_k"] * case["d"] * case["hidden"] / (16 * 32 * 1024 * 2 * 512 * 1024)
    if k.startswith("attn"):
        queries = case["batch"] * case["heads"] * case["seq"]
        return max(queries * case["topk"] * (case["d_qk"] + case["d_v"]) / (32 * 8 * 1024 * 128 * 256),
                   queries * case["seq"] / (32 * 8 * 1024 * 4096))
    return case["batch"] * case["seq"] ** 2 * case["heads"] * case["d"] / (32 * 2048 ** 2 * 4 * 64)


# ---------------------------------------------------------------------------------------------------------------------
# inputs and objects a program holds before the call
# ---------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _weights(shape, g, dtype):
    return torch.randn(shape, generator=g, device=DEV, dtype=dtype).mul_(0.02)


def prepare(case, seed):
    g = _gen(seed)
    return dict(_PREPARE[case["kind"]](case, g, seed), kind=case["kind"])


def _prepare_linear(c, g, seed):
    torch.manual_seed(seed)
    with torch.device(DEV):
        layer = K.FP8Linear(c["d_in"], c["d_out"], round_scale=c["round_scale"])
    s = dict(layer=layer, x=torch.randn(c["tokens"], c["d_in"], generator=g, device=DEV, dtype=torch.bfloat16))
    if c["kind"] == "linear_train":
        s["x"].requires_grad_(True)
        s["dy"] = torch.randn(c["tokens"], c["d_out"], generator=g, device=DEV, dtype=torch.bfloat16)
    return s


def _ragged(rows, experts, g):
    """Ends and starts of ragged row ranges: shares around the mean as a mildly unbalanced router gives them."""
    share = torch.rand(experts, generator=g, device=DEV) + 0.5
    ends = (share.cumsum(0) / share.sum() * rows).round().long()
    ends[-1] = rows
    return torch.cat([ends.new_zeros(1), ends[:-1]]), ends


def _prepare_grouped(c, g, seed):
    starts, ends = _ragged(c["rows"], c["experts"], g)
    return dict(x=torch.randn(c["rows"], c["d_in"], generator=g, device=DEV, dtype=torch.bfloat16).requires_grad_(True),
                w=_weights((c["experts"], c["d_out"], c["d_in"]), g, torch.float32).requires_grad_(True), starts=starts, ends=ends,
                dy=torch.randn(c["rows"], c["d_out"], generator=g, device=DEV, dtype=torch.bfloat16))


def _prepare_moe_serve(c, g, seed):
    E, d, inter = c["experts"], c["d"], c["inter"]
    bf16 = torch.bfloat16
    shared = moe.FP8SwiGLU(_weights((inter, d), g, bf16), _weights((inter, d), g, bf16), _weights((d, inter), g, bf16))
    layer = moe.ExpertParallelMoE(_weights((E, d), g, torch.float32), torch.randn(E, generator=g, device=DEV) * c["bias_std"],
                                  _weights((E, 2 * inter, d), g, bf16), _weights((E, d, inter), g, bf16), c["top_k"], shared=shared)
    return dict(layer=layer, x=torch.randn(c["tokens"], d, generator=g, device=DEV, dtype=bf16))


def _prepare_moe_train(c, g, seed):
    torch.manual_seed(seed)
    with torch.device(DEV):
        block = layers.MoE(c["experts"], 1, c["top_k"], c["d"], c["hidden"], 2, 0.001, 0.01)
    block = K.convert_to_fp8(block).train()
    shape = (c["batch"], c["seq"], c["d"])
    return dict(block=block, params=list(block.parameters()), x=torch.randn(shape, generator=g, device=DEV).requires_grad_(True),
                dy=torch.randn(shape, generator=g, device=DEV), one=torch.ones((), device=DEV))


def _prepare_attn(c, g, seed):
    B, H, L, k, dt = c["batch"], c["heads"], c["seq"], c["topk"], DTYPES[c["dtype"]]
    s = dict(q=torch.randn(B, H, L, c["d_qk"], generator=g, device=DEV).to(dt),
             k=torch.randn(B, H, L, c["d_qk"], generator=g, device=DEV).to(dt),
             v=torch.randn(B, H, L, c["d_v"], generator=g, device=DEV).to(dt))
    # what an indexer hands over: per query the k best-scored positions, the causal ones first; a query with fewer than k
    # positions behind it gets later ones too, which the attention ignores
    later = torch.ones(L, L, dtype=torch.bool, device=DEV).triu(1)
    s["idx"] = torch.stack([torch.rand(L, L, generator=g, device=DEV).masked_fill(later, -1.0).topk(min(k, L), dim=-1).indices
                            for _ in range(B)])
    if c["kind"] == "attn_train":
        for n in "qkv":
            s[n].requires_grad_(True)
        s["dy"] = torch.randn(B, H, L, c["d_v"], generator=g, device=DEV).to(dt)
    return s


def _prepare_indexer(c, g, seed):
    B, L, H, d, dt = c["batch"], c["seq"], c["heads"], c["d"], DTYPES[c["dtype"]]
    return dict(q=torch.randn(B, L, H, d, generator=g, device=DEV).to(dt), k=torch.randn(B, L, d, generator=g, device=DEV).to(dt),
                w=torch.rand(B, L, H, generator=g, device=DEV).to(dt))


_PREPARE = dict(linear_fwd=_prepare_linear, linear_train=_prepare_linear, grouped_train=_prepare_grouped,
                moe_serve=_prepare_moe_serve, moe_train=_prepare_moe_train, attn_fwd=_prepare_attn, attn_train=_prepare_attn,
                indexer=_prepare_indexer)


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "linear_fwd":
        with torch.no_grad():
            return s["layer"](s["x"])
    if kind == "linear_train":
        y = s["layer"](s["x"])
        gx, gw = torch.autograd.grad(y, [s["x"], s["layer"].weight], s["dy"])
        return dict(y=y.detach(), grad_x=gx, grad_w=gw)
    if kind == "grouped_train":
        y = K.moe_grouped_gemm(s["x"], s["w"], s["starts"], s["ends"], dtype=torch.bfloat16)
        gx, gw = torch.autograd.grad(y, [s["x"], s["w"]], s["dy"])
        return dict(y=y.detach(), grad_x=gx, grad_w=gw)
    if kind == "moe_serve":
        with torch.no_grad():
            return s["layer"](s["x"])
    if kind == "moe_train":
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y, balance = s["block"](s["x"])
        grads = torch.autograd.grad([y, balance], [s["x"], *s["params"]], [s["dy"], s["one"]])
        return dict(y=y.detach(), balance=balance.detach(), grads=list(grads), bias=s["block"].expert_bias)
    if kind == "attn_fwd":
        with torch.no_grad():
            return K.sparse_attention(s["q"], s["k"], s["v"], s["idx"])
    if kind == "attn_train":
        out, attn = K.sparse_attention(s["q"], s["k"], s["v"], s["idx"])
        gq, gk, gv = torch.autograd.grad(out, [s["q"], s["k"], s["v"]], s["dy"])
        return dict(out=out.detach(), attn=attn, grad_q=gq, grad_k=gk, grad_v=gv)
    return K.lightning_indexer_fused(s["q"], s["k"], s["w"])


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far two correct implementations may be apart
# ---------------------------------------------------------------------------------------------------------------------
def _experts_hit(c):
    """Experts that receive at least one token: the router's distribution, sampled."""
    rng = np.random.default_rng(0)
    T, E = min(c["tokens"], 2048), c["experts"]
    score = 1.0 / (1.0 + np.exp(-rng.standard_normal((T, E)) * 0.02 * math.sqrt(c["d"])))
    score += rng.standard_normal(E) * c["bias_std"]
    return len(np.unique(np.argpartition(-score, c["top_k"] - 1, axis=1)[:, :c["top_k"]]))


def work(case):
    c, kind = case, case["kind"]
    if kind.startswith("linear"):
        M, Kd, N = c["tokens"], c["d_in"], c["d_out"]
        once = 2 * M * Kd + 4 * N * Kd + 2 * M * N
        return dict(bytes=once if kind == "linear_fwd" else 2 * once, flops=(2.0 if kind == "linear_fwd" else 6.0) * M * N * Kd)
    if kind == "grouped_train":
        R, Kd, N, E = c["rows"], c["d_in"], c["d_out"], c["experts"]
        # the expert weights are kept as one e4m3 byte per element; their gradient is fp32
        return dict(bytes=2 * (2 * R * Kd + 2 * R * N) + 5 * E * N * Kd, flops=6.0 * R * N * Kd)
    if kind == "moe_serve":
        T, d, inter = c["tokens"], c["d"], c["inter"]
        n = T * (c["top_k"] + 1)
        return dict(bytes=6 * T * d + 4 * c["experts"] * d + 3 * d * inter * (_experts_hit(c) + 1),
                    flops=6.0 * n * d * inter + 2.0 * T * d * c["experts"])
    if kind == "moe_train":
        T, d, h, E = c["batch"] * c["seq"], c["d"], c["hidden"], c["experts"]
        weights = E * 3 * d * (h // 2) + 3 * d * h + E * d
        return dict(bytes=16 * T * d + 8 * weights, flops=18.0 * T * d * (c["top_k"] * (h // 2) + h) + 6.0 * T * d * E)
    if kind.startswith("attn"):
        B, H, L, k, dq, dv, it = c["batch"], c["heads"], c["seq"], min(c["topk"], c["seq"]), c["d_qk"], c["d_v"], ITEM[c["dtype"]]
        valid = B * H * (k * (k + 1) / 2 + (L - k) * k)          # causal (query, key) pairs
        fwd = B * H * L * ((2 * dq + 2 * dv) * it + 4 * k) + 8 * B * L * k
        bwd = B * H * L * (4 * dq + 3 * dv) * it + 8 * B * L * k
        if kind == "attn_fwd":
            return dict(bytes=fwd, flops=2.0 * valid * (dq + dv))
        return dict(bytes=fwd + bwd, flops=2.0 * valid * (dq + dv) + 2.0 * valid * (3 * dq + 2 * dv))
    B, L, H, d, it = c["batch"], c["seq"], c["heads"], c["d"], ITEM[c["dtype"]]
    return dict(bytes=B * L * (H * d + d + H) * it + 2 * B * L * L, flops=2.0 * B * L * L * H * d)


def tolerance(case):
    kind = case["kind"]
    if kind in ("linear_fwd", "linear_train", "grouped_train"):
        return dict(rel=5e-3)                  # bf16 results of e4m3 products summed in fp32
    if kind in ("moe_serve", "moe_train"):
        return dict(rel=1e-2)                  # bf16 intermediates that are rounded to e4m3 again
    if kind == "indexer":
        return dict(rel=1e-3)                  # fp16 logits
    return dict(rel=1e-5 if case["dtype"] == "fp32" else 5e-3)
