"""The drop-in MoE block on the GPU: the combine pass's backward against autograd, the block against its own torch
path on the CPU (same weights; e4m3 noise only), and the expert-sharded block on 2 GPUs against the unsharded one
(forward, gradients, bias update)."""
import os
import socket
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def K():
    from cinnamon_b200 import kernels
    yield kernels
    assert kernels.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_combine_backward_matches_autograd(K, dtype):
    g = torch.Generator().manual_seed(4)
    T, k, d = 70, 3, 136
    rows = torch.randn(T * k + 5, d, generator=g).to(dtype).cuda().requires_grad_(True)
    perm = torch.randperm(T * k, generator=g)
    pos = perm.view(T, k).sort(dim=1).values.cuda()
    gates = torch.rand(T, k, generator=g).cuda().requires_grad_(True)
    addend = torch.randn(T, d, generator=g).bfloat16().cuda().requires_grad_(True)
    dy = torch.randn(T, d, generator=g).cuda()
    y = K.moe_combine_autograd(rows, pos, gates, addend)
    y.backward(dy)
    r2, g2, a2 = (t.detach().clone().requires_grad_(True) for t in (rows, gates, addend))
    y2 = (r2.float()[pos] * g2.unsqueeze(-1)).sum(1) + a2.float()
    y2.backward(dy)
    torch.testing.assert_close(y, y2, rtol=1e-5, atol=1e-5)
    tol = dict(rtol=1e-2, atol=1e-2) if dtype == torch.bfloat16 else dict(rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(rows.grad.float(), r2.grad.float(), **tol)
    torch.testing.assert_close(gates.grad, g2.grad, rtol=1e-4, atol=1e-4)
    torch.testing.assert_close(addend.grad.float(), a2.grad.float(), rtol=1e-2, atol=1e-2)
    assert torch.all(rows.grad[T * k:] == 0)                  # rows no pair names


def test_moe_block_on_gpu_against_its_cpu_path(K):
    from cinnamon_b200 import layers
    torch.manual_seed(7)
    E, k, d, h = 8, 2, 256, 512
    cpu = layers.MoE(E, 1, k, d, h, 2, 0.001, 0.01)
    gpu = layers.MoE(E, 1, k, d, h, 2, 0.001, 0.01)
    gpu.load_state_dict(cpu.state_dict())
    gpu = K.convert_to_fp8(gpu.cuda())
    assert isinstance(gpu.shared_experts[0].w1, K.FP8Linear)
    x = torch.randn(3, 40, d)
    xc, xg = x.clone().requires_grad_(True), x.clone().cuda().requires_grad_(True)
    cpu.train(), gpu.train()
    yc, bc = cpu(xc)
    (yc.pow(2).mean() + bc).backward()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        yg, bg = gpu(xg)
    (yg.float().pow(2).mean() + bg).backward()
    torch.cuda.synchronize()
    rel = lambda a, b: float((a.detach().cpu().float() - b).norm() / b.norm())                    # noqa: E731
    assert rel(yg, yc.detach()) < 0.08 and abs(float(bg) - float(bc)) < 2e-3
    assert torch.equal(gpu.expert_bias.cpu(), cpu.expert_bias)
    assert rel(xg.grad, xc.grad) < 0.2
    for (n, pc), (_, pg) in zip(cpu.named_parameters(), gpu.named_parameters()):
        assert pg.grad is not None and torch.isfinite(pg.grad).all(), n
        assert rel(pg.grad, pc.grad) < 0.25, (n, rel(pg.grad, pc.grad))


EP_WORKER = r'''
import os, sys, torch, torch.distributed as dist
sys.path.insert(0, sys.argv[1])
from cinnamon_b200 import kernels as K, layers
rank = int(os.environ["RANK"]); world = int(os.environ["WORLD_SIZE"])
torch.cuda.set_device(rank)
dist.init_process_group("nccl", device_id=torch.device("cuda", rank))
E, k, d, h = 8, 2, 256, 512
torch.manual_seed(3)
full = layers.MoE(E, 1, k, d, h, 2, 0.01, 0.02).cuda()
sharded = layers.MoE(E, 1, k, d, h, 2, 0.01, 0.02, group=dist.group.WORLD, exchange=sys.argv[3]).cuda()
el = E // world
with torch.no_grad():
    sharded.router.weight.copy_(full.router.weight)
    sharded.shared_experts.load_state_dict(full.shared_experts.state_dict())
    sharded.routed_experts.w12.copy_(full.routed_experts.w12[rank * el:(rank + 1) * el])
    sharded.routed_experts.w3.copy_(full.routed_experts.w3[rank * el:(rank + 1) * el])
xs = [torch.randn(2, 24 + 8 * r, d, generator=torch.Generator().manual_seed(40 + r)).cuda() for r in range(world)]
full.train(); sharded.train()
full.gamma = 0.0        # `full` is called once per rank's tokens: its bias must not move between the calls
x_full = [t.clone().requires_grad_(True) for t in xs]
outs = [full(t) for t in x_full]
sum(o.pow(2).sum() + b for o, b in outs).backward()
x = xs[rank].clone().requires_grad_(True)
y, bl = sharded(x)
(y.pow(2).sum() + bl).backward()
diffs = []
def close(a, b, tol=1e-3):
    err = float((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-30))
    diffs.append(round(err, 6))
    return err < tol
ok = [torch.equal(y, outs[rank][0].detach()), close(x.grad, x_full[rank].grad)]
for a, b in ((sharded.router.weight, full.router.weight), (sharded.shared_experts[0].w1.weight, full.shared_experts[0].w1.weight)):
    ga = a.grad.clone(); dist.all_reduce(ga)
    ok.append(close(ga, b.grad))
gz = lambda p: p.grad if p.grad is not None else torch.zeros_like(p)
# the experts' weight gradients quantise dY and x in tiles that run along the rows of an expert; sharded, an expert's
# rows are the two ranks' tokens in one list, unsharded they arrive in two calls: same mathematics, different e4m3 tiles
ok.append(close(gz(sharded.routed_experts.w12), full.routed_experts.w12.grad[rank * el:(rank + 1) * el], 0.1))
ok.append(close(gz(sharded.routed_experts.w3), full.routed_experts.w3.grad[rank * el:(rank + 1) * el], 0.1))
# a second step through the same block (the exchange buffers and their flags are reused)
x2 = (xs[rank] * 0.5).clone().requires_grad_(True)
y2, bl2 = sharded(x2)
(y2.pow(2).sum() + bl2).backward()
ok.append(bool(torch.isfinite(y2).all()) and bool(torch.isfinite(x2.grad).all()) and float(x2.grad.abs().sum()) > 0)
torch.cuda.synchronize()
with open(os.path.join(sys.argv[2], f"ok_{rank}"), "w") as f:
    f.write(repr([bool(v) for v in ok]) + f" status {K.device_status()}" + (" " + repr(diffs) if not all(ok) else ""))
dist.barrier(); dist.destroy_process_group()
'''


@pytest.mark.parametrize("exchange", ["nccl", "p2p"])
def test_sharded_moe_block_trains_like_the_unsharded_one_on_gpus(K, tmp_path, exchange):
    """Outputs and all gradients of the expert-sharded block on 2 GPUs against the unsharded block, with the rows
    exchanged by all-to-all collectives and by peer stores over NVLink (forward and backward)."""
    if torch.cuda.device_count() < 2:
        pytest.skip("needs 2 GPUs")
    script = tmp_path / "ep_train.py"
    script.write_text(EP_WORKER)
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        port = s.getsockname()[1]
    subprocess.check_call([sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2",
                           "--master-addr", "127.0.0.1", "--master-port", str(port), str(script), ROOT, str(tmp_path),
                           exchange],
                          timeout=600, env=dict(os.environ, NCCL_NVLS_ENABLE="0"))
    for rank in range(2):
        text = (tmp_path / f"ok_{rank}").read_text()
        assert text == "[True, True, True, True, True, True, True] status 0", f"rank {rank}: {text}"


@pytest.mark.parametrize("case", [(2, 40, 8, 2, 256, 512, 0.01), (1, 129, 33, 3, 256, 1024, 0.0), (3, 64, 300, 6, 512, 512, 0.02)])
@pytest.mark.parametrize("autocast", [True, False])
def test_native_block_matches_the_module_path(K, case, autocast):
    """The block as native autograd nodes against the same block run through its modules (a forward hook on an inner module
    selects that path): outputs, balance loss, bias update and every gradient.  The two differ where bf16 or e4m3 rounding
    meets sums in another order (x's gradient adds its parts before one rounding instead of after several)."""
    from cinnamon_b200 import layers
    B, L, E, k, d, h, alpha = case
    torch.manual_seed(E)
    with torch.device("cuda"):
        a = layers.MoE(E, 1, k, d, h, 2, 0.01, alpha)
        b = layers.MoE(E, 1, k, d, h, 2, 0.01, alpha)
    b.load_state_dict(a.state_dict())
    a, b = K.convert_to_fp8(a).train(), K.convert_to_fp8(b).train()
    for m in (b.shared_experts[0].w1, b.router):
        m.register_forward_hook(lambda *args: None)
    x = torch.randn(B, L, d, device="cuda")
    dy = torch.randn(B, L, d, device="cuda")
    got = []
    for block in (a, b):
        xi = x.clone().requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=autocast):
            y, bal = block(xi)
        ((y.float() * dy).sum() + (bal * 3.0 if bal is not None else 0.0)).backward()
        got.append((y, bal, xi.grad, dict(block.named_parameters()), block.expert_bias))
    (y0, b0, gx0, p0, eb0), (y1, b1, gx1, p1, eb1) = got
    rel = lambda u, v: float((u.float() - v.float()).norm() / v.float().norm())                   # noqa: E731
    assert rel(y0, y1) < 1e-3 and torch.equal(eb0, eb1) and (b0 is None) == (b1 is None)
    if b0 is not None:
        assert abs(float(b0) - float(b1)) < 1e-5 * abs(float(b1)) + 1e-9
    assert gx0.dtype == gx1.dtype and rel(gx0, gx1) < 1e-2
    for name, p in p0.items():
        assert p.grad.dtype == p1[name].grad.dtype and rel(p.grad, p1[name].grad) < 1e-2, name


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,d,hidden", [(48, 256, 512), (131, 384, 128)])
def test_native_swiglu_is_its_layers_bit_for_bit(K, dtype, tokens, d, hidden):
    """The shared expert as one node against the same three layers (a hook on one of them selects that path): every output
    and gradient is the same number, x's too, whose two parts are rounded by layer and added up in autograd's order.
    (Reductions of fewer than 20 blocks of 128 are never cut, so no sum is taken in another order.)"""
    from cinnamon_b200 import layers
    torch.manual_seed(tokens)
    with torch.device("cuda"):
        block = layers.SwiGLU(d, hidden)
    block = K.convert_to_fp8(block)
    x = torch.randn(tokens, d, device="cuda").to(dtype)
    dy = torch.randn(tokens, d, device="cuda").bfloat16()
    base = torch.randn(tokens, d, device="cuda").to(dtype)                     # a third gradient of x, from elsewhere
    got = []
    for _ in range(2):
        xi = x.clone().requires_grad_(True)
        y = block(xi)
        got.append([y, *torch.autograd.grad([y, xi * base], [xi, *block.parameters()], [dy, torch.ones_like(xi)])])
        block.w1.register_forward_hook(lambda *args: None)
    for a, b in zip(*got):
        assert a.dtype == b.dtype and torch.equal(a, b)


def test_native_routed_experts_compute_the_module_paths_silu(K):
    """Forward of the block on widely spread activations (two experts per token, whose gates both paths add up alike): the
    node quantises silu(h1) * h2 in the pass that computes it, the module path from a bf16 copy; the output is the same, bit
    for bit."""
    from cinnamon_b200 import layers
    torch.manual_seed(7)
    with torch.device("cuda"):
        block = layers.MoE(4, 1, 2, 256, 1024, 2, 0.0, 0.0)
    block = K.convert_to_fp8(block).eval()
    with torch.no_grad():
        block.routed_experts.w12.mul_(12.0)
    x = torch.randn(1, 8192, 256, device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        native, _ = block(x)
        block.router.register_forward_hook(lambda *args: None)
        modules, _ = block(x)
    assert torch.equal(native, modules)


@pytest.mark.parametrize("grad", [True, False])
def test_forward_mode_tangents_are_refused_not_dropped(K, grad):
    """Neither the FP8 linear nor the attention has a forward-mode derivative: a dual input raises, with frozen weights and
    without a gradient to record too, where the calls take a path without an autograd node."""
    import torch.autograd.forward_ad as fw
    from cinnamon_b200 import layers
    with torch.device("cuda"):
        lin = K.FP8Linear(256, 384).requires_grad_(False)
        swiglu = K.convert_to_fp8(torch.nn.Sequential(layers.SwiGLU(256, 512))).requires_grad_(False)
        x, tangent = torch.randn(2, 32, 256).unbind(0)
        q, k, v = torch.randn(3, 1, 2, 32, 64).unbind(0)
        idx = torch.zeros(1, 32, 4, dtype=torch.long)
    with torch.set_grad_enabled(grad), fw.dual_level():
        for call in (lambda: lin(fw.make_dual(x, tangent)), lambda: swiglu(fw.make_dual(x, tangent)),
                     lambda: K.sparse_attention(fw.make_dual(q, torch.ones_like(q)), k, v, idx),
                     lambda: K.sparse_attention(q, k, fw.make_dual(v, torch.ones_like(v)), idx)):
            with pytest.raises(RuntimeError, match="jvp"):
                call()


def test_swiglu_without_gradients_keeps_nothing_for_a_backward(K):
    """Evaluation: one launch quantises a layer's input and weight (no block copies, no transposed weight); same numbers."""
    from cinnamon_b200 import layers
    with torch.device("cuda"):
        block = K.convert_to_fp8(layers.SwiGLU(256, 512))
    x = torch.randn(3, 40, 256, device="cuda")
    want = block(x)
    n = K.launch_count
    with torch.no_grad():
        got = block(x)
    assert K.launch_count - n == 5                # quantise, multiply; silu; quantise, multiply
    assert torch.equal(got, want) and not got.requires_grad
    block.requires_grad_(False)
    assert torch.equal(block(x), want)


@pytest.mark.parametrize("hooked", [False, True])
def test_balance_loss_alone_leaves_the_experts_without_gradients(K, hooked):
    """Differentiating only the balance loss: the router and x get a gradient, no expert gets one (None, not zeros, which an
    optimiser with weight decay or momentum would act on)."""
    from cinnamon_b200 import layers
    with torch.device("cuda"):
        block = K.convert_to_fp8(layers.MoE(8, 1, 2, 256, 1024, 2, 0.01, 0.01))
    if hooked:
        block.shared_experts[0].w1.register_forward_hook(lambda *args: None)
    x = torch.randn(2, 40, 256, device="cuda", requires_grad=True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        _, balance = block(x)
    balance.backward()
    assert block.router.weight.grad is not None and x.grad is not None
    assert [n for n, p in block.named_parameters() if p.grad is not None] == ["router.weight"]


def test_moe_layers_refuse_a_bias_left_on_the_host(K):
    """The routing bias on the CPU and an input of another width raise before anything is launched."""
    from cinnamon_b200 import layers, moe
    with torch.device("cuda"):
        block = K.convert_to_fp8(layers.MoE(8, 1, 2, 256, 1024, 2, 0.01, 0.01))
        w = lambda *s: torch.randn(*s).bfloat16()                                             # noqa: E731
        serve = moe.ExpertParallelMoE(w(8, 256).float(), torch.zeros(8), w(8, 256, 256), w(8, 256, 128), 2,
                                      shared=moe.FP8SwiGLU(w(128, 256), w(128, 256), w(256, 128)))
        x = torch.randn(1, 40, 256)
        wide = torch.randn(40, 272).bfloat16()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        block(x), serve(x[0].bfloat16())
        torch.cuda.synchronize()
        with pytest.raises(AssertionError, match="widths"):
            serve(wide)
        block.expert_bias = block.expert_bias.cpu()
        serve.expert_bias = serve.expert_bias.cpu()
        with pytest.raises(AssertionError, match="CUDA"):
            block(x)
        n = K.launch_count
        with pytest.raises(AssertionError, match="CUDA"):
            serve(x[0].bfloat16())
        assert K.launch_count == n


def test_launch_count_is_what_the_profiler_sees(K):
    """``K.launch_count`` against the library's kernels in a profile: linears, routing with and without its scan, attention of
    every type through tiles and gathers, the serving layer, a training step of the block."""
    from torch.profiler import ProfilerActivity, profile
    from cinnamon_b200 import layers, moe
    with torch.device("cuda"):
        lin = K.FP8Linear(512, 384)
        block = K.convert_to_fp8(layers.MoE(8, 1, 2, 256, 1024, 2, 0.01, 0.01))
        w = lambda *s: torch.randn(*s).bfloat16()                                             # noqa: E731
        serve = moe.ExpertParallelMoE(w(8, 256).float(), torch.zeros(8), w(8, 256, 256), w(8, 256, 128), 2,
                                      shared=moe.FP8SwiGLU(w(128, 256), w(128, 256), w(256, 128)))
        x = torch.randn(2, 40, 256, requires_grad=True)
        bias = torch.zeros(8)

    def attention(dtype, d, mode):
        before = K._L.cinn_set_sparse_attn_dense(mode)
        q, k, v = (torch.randn(1, 2, 300, d, device="cuda", dtype=dtype, requires_grad=True) for _ in range(3))
        out, _ = K.sparse_attention(q, k, v, torch.randint(0, 300, (1, 300, 16), device="cuda"))
        out.sum().backward()
        K._L.cinn_set_sparse_attn_dense(before)
    calls = [lambda: lin(torch.randn(48, 512, device="cuda")).sum().backward(), lambda: block(x)[0].sum().backward(),
             lambda: serve(x[0].detach().bfloat16()), lambda: K.moe_route(torch.randn(200, 8, device="cuda"), bias, 2),
             lambda: K.moe_route(torch.randn(3000, 8, device="cuda"), bias, 2),
             lambda: K.fp8_matmul_dsv3(K.quantize_fp8_rowwise(torch.randn(64, 8192, device="cuda"))[0],               # cut along K
                                       K.quantize_fp8_blockwise(torch.randn(256, 8192, device="cuda"))[0].t(),
                                       torch.ones(64, 64, device="cuda"), torch.ones(64, 2, device="cuda"))]
    calls += [lambda dt=dt, d=d, mode=mode: attention(dt, d, mode) for dt in (torch.bfloat16, torch.float16, torch.float32)
              for d in (64, 20) for mode in (0, 1)]
    for i, call in enumerate(calls):
        call()
        torch.cuda.synchronize()
        n = K.launch_count
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
            call()
            torch.cuda.synchronize()
        seen = [e.name for e in prof.events() if e.device_type.name == "CUDA" and "cinn::" in e.name]
        assert K.launch_count - n == len(seen), (i, seen)


@pytest.mark.parametrize("T", [40, 3100])
def test_swiglu_in_training_under_capture(K, T):
    """A few tokens under capture take SwiGLU as passes of its own, many take it inside the quantisers: the numbers of the call outside."""
    from cinnamon_b200 import layers
    torch.manual_seed(T)
    with torch.device("cuda"):
        block = K.convert_to_fp8(layers.SwiGLU(256, 1024))
    x = torch.randn(T, 256, device="cuda").to(torch.bfloat16).requires_grad_(True)
    dy = torch.randn(T, 256, device="cuda").to(torch.bfloat16)

    def run():
        n = K.launch_count
        y = block(x)
        g = torch.autograd.grad(y, [x, *block.parameters()], dy)
        return [y.detach(), *g], K.launch_count - n

    (want, outside), _ = run(), torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got, inside = run()
    graph.replay()
    assert inside - outside == (2 if T == 40 else 0)          # SwiGLU by itself, forward and backward
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    del graph
