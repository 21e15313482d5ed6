"""Block-scaled FP8 GEMM parity: CUDA (through the C ABI) against the float64
dequantise -> matmul oracle.  Tolerance from the specification: relative
Frobenius error <= 1e-3 on the fp32 result; the bf16 result is compared with the
float64 result rounded to bf16."""
import numpy as np
import pytest
import torch

from _util import assert_bf16_close, bits_of, bytes_of, rel_fro
from oracle import fp8_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-3          # rel-Frobenius bound of the specification (fp32 output)


@pytest.fixture(scope="module")
def K():
    from cinnamon_b200 import kernels
    kernels.set_div_mode("rn")
    yield kernels
    assert kernels.device_status() == 0, "a kernel gave up on a bounded wait"
    kernels.set_div_mode("full")
    torch.cuda.empty_cache()            # (what is allocated next does not keep this module's large segments)


def _operands(M, N, Kd, seed):
    x, w, _ = O.make_linear_case(M, Kd, N, seed)
    xq, xs = O.quantize_rowwise(x, 128)
    wq, ws = O.quantize_blockwise(w.float(), 128, 128)
    return xq, xs, wq, ws


def _f8(t):
    return t.cuda().view(torch.float8_e4m3fn)


SHAPES = [(128, 256, 128), (256, 512, 512), (130, 576, 512), (130, 576, 640), (1, 128, 256), (300, 64, 1024),
          (4096, 2048, 512), (257, 1000, 144)]


@pytest.mark.parametrize("M,N,Kd", SHAPES)
def test_gemm_weight_layout_nk(K, M, N, Kd):
    """B given as the (N, K) weight seen through .t(): the forward layout."""
    xq, xs, wq, ws = _operands(M, N, Kd, seed=M + N + Kd)
    ref = O.fp8_matmul_f64(xq, wq.t(), xs, ws.t())
    out32 = K.fp8_matmul_dsv3(_f8(xq), _f8(wq).t(), xs.cuda(), ws.cuda().t(), out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert K.device_status() == 0
    err = rel_fro(out32, ref)
    maxabs = float((out32.cpu().double() - ref).abs().max())
    print(f"[{M}x{N}x{Kd}] fp32 rel-Fro {err:.3e} max-abs {maxabs:.3e}")
    assert err <= TOL
    assert err <= 2e-5          # e4m3 products are exact, only fp32 accumulation rounds
    out16 = K.fp8_matmul_dsv3(_f8(xq), _f8(wq).t(), xs.cuda(), ws.cuda().t())
    assert out16.dtype == torch.bfloat16
    assert_bf16_close(out16, ref, "bf16 output")
    assert (out16.cpu() != ref.to(torch.bfloat16)).float().mean().item() < 1e-2


@pytest.mark.parametrize("M,N,Kd", [(128, 256, 128), (256, 512, 512), (130, 576, 640), (300, 64, 1024), (4096, 2048, 512)])
def test_gemm_layout_kn(K, M, N, Kd):
    """B stored (K, N) as fp8_matmul_dsv3 documents (src/kernels.py:669)."""
    xq, xs, wq, ws = _operands(M, N, Kd, seed=7 + M + N + Kd)
    b = wq.t().contiguous()
    bs = ws.t().contiguous()
    ref = O.fp8_matmul_f64(xq, b, xs, bs)
    out32 = K.fp8_matmul_dsv3(_f8(xq), _f8(b), xs.cuda(), bs.cuda(), out_dtype=torch.float32)
    err = rel_fro(out32, ref)
    print(f"[KN {M}x{N}x{Kd}] fp32 rel-Fro {err:.3e}")
    assert err <= TOL and err <= 2e-5


@pytest.mark.parametrize("M,N,Kd", [(128, 256, 8192), (1, 64, 7168), (130, 333, 6032), (1024, 512, 8208), (300, 516, 8208), (257, 260, 12304)])
@pytest.mark.parametrize("kn", [False, True])
def test_gemm_cut_along_k(K, M, N, Kd, kn):
    """Few tiles, long reduction: partial sums over pieces of K (the last one short), added in a fixed order."""
    if kn and N % 16:
        pytest.skip("B stored (K, N) needs N % 16 == 0")
    assert K._L.cinn_fp8_gemm_workspace_bytes(M, N, Kd, int(kn)) > 0
    xq, xs, wq, ws = _operands(M, N, Kd, seed=M + N + Kd)
    ref = O.fp8_matmul_f64(xq, wq.t(), xs, ws.t())
    b = _f8(wq.t().contiguous()) if kn else _f8(wq).t()
    for dtype in (torch.float32, torch.bfloat16):
        out = K.fp8_matmul_dsv3(_f8(xq), b, xs.cuda(), ws.cuda().t(), out_dtype=dtype)
        if dtype == torch.float32:
            assert rel_fro(out, ref) <= 2e-5
        else:
            assert_bf16_close(out, ref, "bf16 output")
        assert torch.equal(out, K.fp8_matmul_dsv3(_f8(xq), b, xs.cuda(), ws.cuda().t(), out_dtype=dtype))


@pytest.mark.parametrize("N,Kd", [(1024, 512), (333, 144), (576, 2064), (40, 16), (4096, 7168)])
def test_few_rows_have_the_bits_of_many(K, N, Kd):
    """The kernel for few rows forms the sums of the others: every row of a small call equals that row of a large one, for one,
    a part of, all and more than a tile of rows, columns that end inside a block, reductions that end inside a K block."""
    M = 8192 if N * Kd < 1 << 20 else 4096
    xq, xs, wq, ws = _operands(M, N, Kd, seed=N + Kd)
    a, sa, b, sb = _f8(xq), xs.cuda(), _f8(wq), ws.cuda()
    for dtype in (torch.bfloat16, torch.float32, torch.float16):
        whole = K.fp8_matmul_dsv3(a, b.t(), sa, sb.t(), out_dtype=dtype)
        for m in (1, 63, 64, 65, 128, 129, 300):
            few = K.fp8_matmul_dsv3(a[:m].contiguous(), b.t(), sa[:m].contiguous(), sb.t(), out_dtype=dtype)
            if K._L.cinn_fp8_gemm_workspace_bytes(m, N, Kd, 0) == 0:       # (a cut reduction adds in another order)
                assert torch.equal(few, whole[:m]), (m, dtype)
    assert K.device_status() == 0


@pytest.mark.parametrize("N,Kd,rows", [(40, 16, 20000), (96, 272, 8192), (4096, 7168, 4096), (7168, 5136, 2048)])
def test_few_rows_without_a_cut(K, N, Kd, rows):
    """Calls that are never cut along K (the experts' and the shared expert's): the kernel for few rows, also over a long reduction, gives
    every row the bits of a call of many rows, which is too large for it, and both are the float64 oracle's."""
    xq, xs, wq, ws = _operands(rows, N, Kd, seed=N + Kd)
    a, sa, b, sb = _f8(xq), xs.cuda(), _f8(wq), ws.cuda()

    def run(m, dtype):
        return K._gemm(a[:m].contiguous(), sa[:m].contiguous(), b, 0, sb, 1, sb.stride(0), m, N, Kd, dtype, whole=True)
    for dtype in (torch.bfloat16, torch.float32, torch.float16):
        many = run(rows, dtype)
        for m in (1, 5, 16, 63, 64, 65, 100, 128):
            assert torch.equal(run(m, dtype), many[:m]), (m, dtype)
        if dtype == torch.float32:
            assert rel_fro(many[:128], O.fp8_matmul_f64(xq[:128], wq.t(), xs[:128], ws.t())) <= 2e-5
    assert K.device_status() == 0


PAIR_SCRIPT = r"""
import sys, torch
sys.path.insert(0, sys.argv[1])
from cinnamon_b200 import kernels as K
from oracle import fp8_oracle as O
M, N, Kd = 2304, 2560, 640          # 9 x 10 tiles of 256 x 256: enough for the two-SM kernel, ragged against nothing
xq, xs = O.quantize_rowwise(O.make_linear_case(M, Kd, N, 77)[0], 128)
w = O.make_linear_case(M, Kd, N, 77)[1]
wq, ws = O.quantize_blockwise(w.float(), 128, 128)
f8 = lambda t: t.cuda().view(torch.float8_e4m3fn)
nk = K.fp8_matmul_dsv3(f8(xq), f8(wq).t(), xs.cuda(), ws.cuda().t(), out_dtype=torch.float32)
b = wq.t().contiguous(); bs = ws.t().contiguous()
kn = K.fp8_matmul_dsv3(f8(xq), f8(b), xs.cuda(), bs.cuda(), out_dtype=torch.float32)
torch.cuda.synchronize()
assert K.device_status() == 0
torch.save({"nk": nk.cpu(), "kn": kn.cpu()}, sys.argv[2])
"""


def test_two_sm_and_one_sm_kernels_agree(K, tmp_path):
    """CINN_GEMM_PAIR=0 forces the one-SM kernel, =2 the two-SM (cta_group::2) kernel for both B layouts."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    script = tmp_path / "pair.py"
    script.write_text(PAIR_SCRIPT)
    outs = {}
    for mode in ("0", "2"):
        out = tmp_path / f"out{mode}.pt"
        subprocess.check_call([sys.executable, str(script), root, str(out)], env=dict(os.environ, CINN_GEMM_PAIR=mode),
                              timeout=300)
        outs[mode] = torch.load(out)
    M, N, Kd = 2304, 2560, 640
    x, w, _ = O.make_linear_case(M, Kd, N, 77)
    xq, xs = O.quantize_rowwise(x, 128)
    wq, ws = O.quantize_blockwise(w.float(), 128, 128)
    ref = O.fp8_matmul_f64(xq, wq.t(), xs, ws.t())
    for mode in ("0", "2"):
        for layout in ("nk", "kn"):
            err = rel_fro(outs[mode][layout], ref)
            assert err <= TOL and err <= 2e-5, (mode, layout, err)
    assert rel_fro(outs["2"]["nk"], outs["0"]["nk"].double()) < 1e-6
    assert rel_fro(outs["2"]["kn"], outs["0"]["kn"].double()) < 1e-6


def test_gemm_is_deterministic(K):
    xq, xs, wq, ws = _operands(512, 1024, 1024, seed=5)
    a = K.fp8_matmul_dsv3(_f8(xq), _f8(wq).t(), xs.cuda(), ws.cuda().t(), out_dtype=torch.float32)
    b = K.fp8_matmul_dsv3(_f8(xq), _f8(wq).t(), xs.cuda(), ws.cuda().t(), out_dtype=torch.float32)
    assert torch.equal(a, b)


@pytest.mark.parametrize("M,Kd,N,rs", [(256, 512, 384, False), (512, 256, 640, True), (4096, 512, 2048, False)])
def test_autograd_function_matches_oracle(K, M, Kd, N, rs):
    """FP8MatmulFunction forward / dgrad / wgrad (src/kernels.py:739-794)."""
    x, w, dy = O.make_linear_case(M, Kd, N, seed=11 + M)
    ref_out, saved = O.fp8_linear_forward(x, w, rs)
    ref_gx, ref_gw = O.fp8_linear_backward(dy, saved, rs)
    xg = x.cuda().requires_grad_(True)
    wg = w.float().cuda().requires_grad_(True)
    out = K.FP8MatmulFunction.apply(xg, wg, rs)
    out.backward(dy.cuda())
    assert out.dtype == torch.bfloat16 and xg.grad.shape == x.shape and wg.grad.shape == w.shape
    for name, got, ref in (("fwd", out, ref_out), ("dgrad", xg.grad, ref_gx), ("wgrad", wg.grad, ref_gw)):
        err = rel_fro(got.detach().float(), ref)
        print(f"{name}: rel-Fro(bf16 out) {err:.3e}")
        assert_bf16_close(got.detach().to(torch.bfloat16), ref, name)
        assert err < 4e-3, name          # bf16 rounding alone costs ~1.7e-3


def test_fp8_linear_weight_cache(K):
    """The optional e4m3 weight cache: same outputs and gradients, one quantiser launch fewer per call while the
    weight is unchanged, refreshed after an in-place update."""
    torch.manual_seed(5)
    a = K.FP8Linear(256, 384).cuda()
    b = K.FP8Linear(256, 384, cache_quantized_weight=True).cuda()
    b.load_state_dict(a.state_dict())
    x = torch.randn(64, 256, device="cuda")
    for step in range(3):
        ya, yb = a(x), b(x)
        assert torch.equal(ya, yb)
        ya.sum().backward()
        yb.sum().backward()
        assert torch.equal(a.weight.grad, b.weight.grad)
        if step == 1:                                              # an optimiser step: the cache must notice
            with torch.no_grad():
                a.weight.add_(0.01)
                b.weight.add_(0.01)
        a.weight.grad = b.weight.grad = None
    n0 = K.launch_count
    b(x)
    cached = K.launch_count - n0
    n0 = K.launch_count
    a(x)
    assert K.launch_count - n0 == cached + 1


def test_grouped_gemm_scattered_rows(K):
    """Output rows stored at per-row addresses (the expert-parallel way home): here a permutation inside a local
    buffer, with a dropped row (address 0) and ragged expert sizes; same bits as the plain grouped GEMM."""
    g = torch.Generator().manual_seed(41)
    E, d_in, d_out = 4, 256, 384
    counts = [130, 0, 77, 200]
    T = sum(counts)
    x = torch.randn(T, d_in, generator=g).bfloat16().cuda()
    w = (torch.randn(E, d_out, d_in, generator=g) * 0.05).bfloat16().cuda()
    ends = torch.tensor(counts).cumsum(0).cuda()
    starts = ends - torch.tensor(counts).cuda()
    xq, xs = K.quantize_fp8_rowwise(x)
    wq, ws = K.quantize_expert_weights(w)
    ref = K.fp8_grouped_gemm(xq, xs, wq, ws, starts, ends, out_dtype=torch.bfloat16)
    perm = torch.randperm(T, generator=g).cuda()
    out = torch.full((T + 3, d_out), 7.0, dtype=torch.bfloat16, device="cuda")
    table = out.data_ptr() + perm * (d_out * 2)
    table[5] = 0                                                            # this row has no destination
    K.fp8_grouped_gemm_scatter(xq, xs, wq, ws, starts, ends, table.contiguous(), out_dtype=torch.bfloat16)
    torch.cuda.synchronize()
    assert K.device_status() == 0
    keep = torch.ones(T, dtype=torch.bool, device="cuda")
    keep[5] = False
    assert torch.equal(out[perm[keep]], ref[keep])
    assert torch.all(out[perm[5]] == 7.0) and torch.all(out[T:] == 7.0)     # untouched


def test_fp8_linear_module(K):
    g = torch.Generator().manual_seed(3)
    lin = K.FP8Linear(256, 384, bias=True, round_scale=True).cuda()
    x = torch.randn(2, 65, 256, generator=g).cuda()
    y = lin(x)
    assert y.shape == (2, 65, 384)
    ref, _ = O.fp8_linear_forward(x.cpu().reshape(-1, 256), lin.weight.detach().cpu(), True)
    ref = ref.reshape(2, 65, 384) + lin.bias.detach().cpu().double()
    assert rel_fro(y.float(), ref) < 4e-3
    y.sum().backward()
    assert lin.weight.grad is not None and lin.weight.grad.dtype == torch.float32


@pytest.mark.parametrize("grad", [True, False])
def test_fp8_linear_refuses_operands_that_do_not_fit(K, grad):
    """A weight left on the host, a weight of another width and an input without rows raise before anything is launched."""
    with torch.device("cuda"):
        lin = K.FP8Linear(256, 384)
    x = torch.randn(32, 256, device="cuda", requires_grad=grad)
    lin(x)
    torch.cuda.synchronize()
    launched = K.launch_count
    with torch.set_grad_enabled(grad):
        with pytest.raises(AssertionError, match="CUDA"):
            K.FP8Linear(256, 384)(x)
        for width in (128, 272):
            with pytest.raises(AssertionError, match="wide"):
                lin(torch.randn(32, width, device="cuda", requires_grad=grad))
        with pytest.raises(RuntimeError, match="no rows"):
            lin(x[:0])
        w_q, w_s = K.quantize_fp8_blockwise(torch.randn(384, 128, device="cuda"))
        launched += 1
        with pytest.raises(AssertionError, match="quantised copy"):
            K._host.linear(x, lin.weight, False, True, K._DIV_MODE, w_q, w_s, None)
    assert K.launch_count == launched


def test_fp8_linear_converts_its_weight_before_the_quantisers(K):
    """A float64 weight in training: the same numbers as its fp32 copy.  The weight's quantiser starts beside the
    activations', so the conversion it reads has to be enqueued ahead of both: seen in the order of the launches."""
    from torch.profiler import ProfilerActivity, profile
    with torch.device("cuda"):
        lin = K.FP8Linear(512, 1024)
    wide = K.FP8Linear(512, 1024)
    wide.weight = torch.nn.Parameter(lin.weight.detach().double())
    got = []
    for layer in (lin, wide):
        x = torch.randn(256, 512, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).requires_grad_(True)
        layer(x)
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
            y = layer(x)
            torch.cuda.synchronize()
        names = [e.name for e in sorted((e for e in prof.events() if e.device_type.name == "CUDA"), key=lambda e: e.time_range.start)]
        got.append([y, *torch.autograd.grad(y, [x, layer.weight], torch.ones_like(y))])
    for a, b in zip(*got):
        assert torch.equal(a, b.to(a.dtype))
    quantisers = [i for i, n in enumerate(names) if "quant_" in n]
    assert len(quantisers) == 2 and quantisers[1] == quantisers[0] + 1, names          # nothing between the two


def test_weight_caches_and_updates_through_data(K):
    """The e4m3 copies follow every update that goes through the tensor (version counter); an update through
    ``.data`` leaves them stale until ``invalidate_weight_cache`` is called - the documented behaviour."""
    torch.manual_seed(6)
    E, d, h, T = 3, 256, 128, 96
    w = (torch.randn(E, h, d, device="cuda") * 0.02)
    x = torch.randn(T, d, device="cuda").bfloat16()
    starts = torch.tensor([0, 32, 64], device="cuda")
    ends = torch.tensor([32, 64, 96], device="cuda")
    y0 = K.moe_grouped_gemm(x, w, starts, ends)
    n0 = K.launch_count
    assert torch.equal(K.moe_grouped_gemm(x, w, starts, ends), y0)
    assert K.launch_count - n0 == 2                                 # token quantiser + GEMM: the weights came from the cache
    w.mul_(2.0)                                                     # in place through the tensor: noticed
    y1 = K.moe_grouped_gemm(x, w, starts, ends)
    torch.testing.assert_close(y1.float(), 2 * y0.float(), rtol=2e-2, atol=1e-3)
    w.data.mul_(0.5)                                                # behind autograd's back: not noticed ...
    assert torch.equal(K.moe_grouped_gemm(x, w, starts, ends), y1)
    K.invalidate_weight_cache()                                     # ... until the caches are dropped
    assert torch.equal(K.moe_grouped_gemm(x, w, starts, ends), y0)
    lin = K.FP8Linear(256, 128, cache_quantized_weight=True).cuda()
    z0 = lin(x)
    lin.weight.data.mul_(2.0)
    assert torch.equal(lin(x), z0)
    K.invalidate_weight_cache(lin)
    torch.testing.assert_close(lin(x).float(), 2 * z0.float(), rtol=2e-2, atol=1e-3)


def _grouped_case(E, d_in, d_out, counts, seed, gap=0):
    g = torch.Generator().manual_seed(seed)
    T = sum(counts) + gap
    x = torch.randn(T, d_in, generator=g).bfloat16()
    w = (torch.randn(E, d_out, d_in, generator=g) * 0.02).bfloat16()
    ends = torch.tensor(counts).cumsum(0)
    starts = ends - torch.tensor(counts)
    return x, w, starts, ends


GROUPED = {
    "equal_reference_case": (8, 512, 128, [32] * 8),                       # tests/test_kernels.py:131-155
    "ragged": (6, 256, 384, [5, 0, 130, 1, 257, 64]),
    "empty_first_last": (5, 384, 256, [0, 200, 0, 129, 0]),
    "one_owns_all": (4, 256, 512, [0, 0, 700, 0]),
    "single_tokens": (16, 128, 128, [1] * 16),
    "wide_k": (3, 1024, 320, [100, 300, 28]),
}


@pytest.mark.parametrize("name", list(GROUPED))
def test_grouped_gemm(K, name):
    E, d_in, d_out, counts = GROUPED[name]
    x, w, starts, ends = _grouped_case(E, d_in, d_out, counts, seed=len(name), gap=9)
    ref = O.grouped_gemm_fp8_f64(x, w, starts, ends)
    xq, xs = K.quantize_fp8_rowwise(x.cuda())
    wq, ws = K.quantize_expert_weights(w.cuda())
    T = x.shape[0]
    out = torch.full((T, d_out), 777.0, dtype=torch.float32, device="cuda")       # canary everywhere
    K.fp8_grouped_gemm(xq, xs, wq, ws, starts.cuda(), ends.cuda(), out=out)
    torch.cuda.synchronize()
    assert K.device_status() == 0
    used = int(ends[-1])
    assert torch.all(out[used:] == 777.0), "rows outside every expert's range were written"
    err = rel_fro(out[:used], ref[:used])
    print(f"{name}: rel-Fro {err:.3e}")
    assert err <= TOL and err <= 2e-5
    # the drop-in entry point: fp16 result like the reference, loose check like its own test
    out16 = K.moe_grouped_gemm(x.cuda(), w.cuda(), starts.cuda(), ends.cuda())
    assert out16.dtype == torch.float16 and out16.shape == (T, d_out)
    plain = O.grouped_gemm_f64(x, w, starts, ends)
    rel = ((plain[:used] - out16[:used].cpu().double()).abs() / (plain[:used].abs() + 1e-6))
    assert rel.median().item() < 0.08


@pytest.mark.parametrize("case", [(3, 384, 4096, [700, 0, 900]), (2, 256, 9480, [257, 511]), (2, 144, 4872, [1, 1280]), (1, 128, 5000, [1152])])
def test_grouped_gemm_on_sm_pairs(K, case):
    """Enough rows per expert for the two-SM kernel: tiles whose second half is empty, full or cut anywhere, an expert
    without rows, columns that are no multiple of a tile, every way out (TMA boxes, staged tails, 2- and 4-byte types)."""
    E, d_in, d_out, counts = case
    x, w, starts, ends = _grouped_case(E, d_in, d_out, counts, seed=d_out, gap=9)
    ref = O.grouped_gemm_fp8_f64(x, w, starts, ends)
    xq, xs = K.quantize_fp8_rowwise(x.cuda())
    wq, ws = K.quantize_expert_weights(w.cuda())
    T, used = x.shape[0], int(ends[-1])
    covered = torch.zeros(T, dtype=torch.bool)
    for s, e in zip(starts.tolist(), ends.tolist()):
        covered[s:e] = True
    for dtype in (torch.float32, torch.bfloat16, torch.float16):
        out = torch.full((T, d_out), 777.0, dtype=dtype, device="cuda")
        K.fp8_grouped_gemm(xq, xs, wq, ws, starts.cuda(), ends.cuda(), out=out)
        got = out.cpu()
        assert torch.all(got[~covered] == 777.0), "rows outside every expert's range were written"
        assert rel_fro(got[covered].float(), ref[covered]) <= {torch.float32: 2e-5, torch.bfloat16: 2e-3, torch.float16: 3e-4}[dtype]


@pytest.mark.parametrize("case", [(3, 4096, 384, [700, 0, 900]), (2, 9488, 272, [257, 511]), (2, 4880, 144, [1, 1280]), (1, 5008, 128, [1152])])
def test_grouped_input_gradient_on_sm_pairs(K, case):
    """The same edges for the input gradient, whose weight is read with the reduction axis outermost (a reduction that ends
    inside a block meets the next expert's rows under zeros)."""
    E, d_in, d_out, counts = case
    x, w, starts, ends = _grouped_case(E, d_in, d_out, counts, seed=d_in, gap=9)
    dy = torch.randn(x.shape[0], d_out, generator=torch.Generator().manual_seed(d_in)).bfloat16()
    ref, _ = O.grouped_gemm_fp8_backward_f64(x, w, starts, ends, dy)
    gq, gs = K.quantize_fp8_rowwise(dy.cuda())
    wq, ws = K.quantize_expert_weights(w.cuda())
    inside = torch.zeros(x.shape[0], dtype=torch.bool)
    for s, e in zip(starts.tolist(), ends.tolist()):
        inside[s:e] = True
    for dtype in (torch.float32, torch.bfloat16):
        got = K.fp8_grouped_gemm_dgrad(gq, gs, wq, ws, starts.cuda(), ends.cuda(), out_dtype=dtype).cpu()
        assert torch.all(got[~inside] == 0)
        assert rel_fro(got[inside].float(), ref[inside]) <= {torch.float32: 2e-5, torch.bfloat16: 2e-3}[dtype]
    assert K.device_status() == 0


def test_gemms_under_a_cap_of_one_sm(K):
    """Dense (also more than 128 rows), grouped (enough rows for pairs) and grouped weight gradient: the same bits as uncapped."""
    xq, xs, wq, ws = _operands(300, 320, 512, seed=1)
    x, w, starts, ends = _grouped_case(2, 256, 512, [300, 500], seed=2)

    def run():
        dense = K.fp8_matmul_dsv3(_f8(xq), _f8(wq).t(), xs.cuda(), ws.cuda().t())
        xg, wg = x.cuda().float().requires_grad_(True), w.cuda().float().requires_grad_(True)
        y = K.moe_grouped_gemm(xg, wg, starts.cuda(), ends.cuda(), dtype=torch.bfloat16)
        return dense, y, *torch.autograd.grad(y, [xg, wg], torch.ones_like(y))
    want = run()
    before = K.set_gemm_sm_limit(1)
    try:
        got = run()
    finally:
        K.set_gemm_sm_limit(before)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("M,N,Kd", [(20000, 512, 1168), (20000, 512, 400), (5000, 1024, 2064), (600, 2560, 4112), (9000, 4352, 320), (4500, 2048, 128)])
def test_kernels_agree_on_every_reduction(K, M, N, Kd):
    """Reductions of one to 33 blocks, with less in the last one, over several tiles per pair of SMs: the bits of a cap of one SM, which
    leaves the one-SM kernel only."""
    xq, xs, wq, ws = _operands(M, N, Kd, seed=M + N + Kd)
    a, sa, b, sb = _f8(xq), xs.cuda(), _f8(wq), ws.cuda()

    def run(dtype):
        return K._gemm(a, sa, b, 0, sb, 1, sb.stride(0), M, N, Kd, dtype, whole=True)
    for dtype in (torch.bfloat16, torch.float32):
        want = run(dtype)
        before = K.set_gemm_sm_limit(1)
        try:
            got = run(dtype)
        finally:
            K.set_gemm_sm_limit(before)
        assert torch.equal(got, want)
    rows = torch.arange(0, M, max(1, M // 64))
    assert rel_fro(want.cpu()[rows], O.fp8_matmul_f64(xq[rows], wq.t(), xs[rows], ws.t())) <= 2e-5
    assert K.device_status() == 0


@pytest.mark.parametrize("case", [(8, 2560, 640, 380), (32, 768, 512, 285), (4, 1536, 384, 1200), (16, 512, 1024, 600)])
def test_grouped_kernels_agree(K, case):
    """Both directions at shapes that run on pairs of SMs and at shapes that do not for their waves: the bits of a cap of one SM."""
    E, d_in, d_out, rows = case
    counts = [rows + 37 * ((e * 5) % 9 - 4) for e in range(E)]
    x, w, starts, ends = _grouped_case(E, d_in, d_out, counts, seed=E + rows, gap=3)
    xq, xs = K.quantize_fp8_rowwise(x.cuda())
    wq, ws = K.quantize_expert_weights(w.cuda())
    gq, gs = K.quantize_fp8_rowwise(torch.randn(x.shape[0], d_out, generator=torch.Generator().manual_seed(E)).bfloat16().cuda())
    range_ = (starts.cuda(), ends.cuda())

    def run():
        return (K.fp8_grouped_gemm_dgrad(gq, gs, wq, ws, *range_, out_dtype=torch.bfloat16),
                K.moe_grouped_gemm(x.cuda(), w.cuda(), *range_, dtype=torch.bfloat16))
    want = run()
    before = K.set_gemm_sm_limit(1)
    try:
        got = run()
    finally:
        K.set_gemm_sm_limit(before)
    for a, b in zip(got, want):
        assert torch.equal(a[:int(ends[-1])], b[:int(ends[-1])])
    assert K.device_status() == 0


@pytest.mark.parametrize("name", list(GROUPED))
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_grouped_gemm_16bit(K, name, dtype):
    """The grouped GEMM in the reference's precision (16-bit operands, fp32 accumulation on the tensor cores) against
    the float64 product of the same 16-bit operands; canary rows; then the drop-in in its "16bit" mode, forward and
    backward."""
    E, d_in, d_out, counts = GROUPED[name]
    x, w, starts, ends = _grouped_case(E, d_in, d_out, counts, seed=7 + len(name), gap=9)
    x, w = x.to(dtype), w.to(dtype)
    T, used = x.shape[0], int(ends[-1])
    ref = torch.zeros(T, d_out, dtype=torch.float64)
    for e in range(E):
        s, t = int(starts[e]), int(ends[e])
        ref[s:t] = x[s:t].double() @ w[e].double().t()
    out = torch.full((T, d_out), 777.0, dtype=torch.float32, device="cuda")
    K.grouped_gemm_16bit(x.cuda(), w.cuda(), starts.cuda(), ends.cuda(), out=out)
    torch.cuda.synchronize()
    assert K.device_status() == 0
    assert torch.all(out[used:] == 777.0), "rows outside every expert's range were written"
    err = rel_fro(out[:used], ref[:used])
    print(f"{name} {dtype}: rel-Fro {err:.3e}")
    assert err < 2e-6                                            # exact products, fp32 accumulation
    out16 = K.grouped_gemm_16bit(x.cuda(), w.cuda(), starts.cuda(), ends.cuda(), out_dtype=torch.float16)
    torch.testing.assert_close(out16[:used].float().cpu(), ref[:used].float(), rtol=2e-3, atol=2e-3)
    prev = K.set_moe_grouped_precision("16bit")
    try:
        xg = x.float().cuda().requires_grad_(True)               # fp32 rows, as the reference's MoE passes them
        wg = w.float().cuda().requires_grad_(True)
        y = K.moe_grouped_gemm(xg, wg, starts.cuda(), ends.cuda())
        assert y.dtype == torch.float16
        rel = ((ref[:used] - y[:used].detach().cpu().double()).abs() / (ref[:used].abs() + 1e-6)).mean().item()
        assert rel < 0.01, rel                                   # the reference's own bound (tests/test_kernels.py:155)
        y.float().pow(2).mean().backward()
        assert torch.isfinite(xg.grad).all() and torch.isfinite(wg.grad).all() and wg.grad.abs().sum() > 0
    finally:
        K.set_moe_grouped_precision(prev)


def test_config2_full_size_sampled(K):
    """16384 x 18432 x 7168 forward; rows sampled for the float64 check."""
    M, Kd, N = 16384, 7168, 18432
    g = torch.Generator().manual_seed(1002)
    x = torch.randn(M, Kd, generator=g).bfloat16().cuda()
    w = (torch.randn(N, Kd, generator=g) * 0.02).bfloat16().cuda()
    xq, xs = K.quantize_fp8_rowwise(x)
    wq, ws = K.quantize_fp8_blockwise(w)
    out = K.fp8_matmul_dsv3(xq, wq.t(), xs, ws.t(), out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert K.device_status() == 0
    rows = torch.tensor([0, 1, 127, 128, 5000, 8191, 12345, 16383])
    ref = O.fp8_matmul_f64(xq[rows.cuda()].view(torch.uint8).cpu(), wq.view(torch.uint8).cpu().t(),
                           xs[rows.cuda()].cpu(), ws.cpu().t())
    err = rel_fro(out[rows.cuda()], ref)
    print(f"C2 forward sampled rows: rel-Fro {err:.3e}")
    assert err <= TOL and err <= 2e-5
    # linearity in the activation scales: doubling sA doubles the result exactly
    out2 = K.fp8_matmul_dsv3(xq, wq.t(), xs * 2, ws.t(), out_dtype=torch.float32)
    assert torch.equal(out2, out * 2)


@pytest.mark.parametrize("k_in,n_out", [(7168, 1536), (7168, 576), (1536, 24576), (512, 16384)])
def test_mla_projection_shapes_sampled(K, k_in, n_out):
    """Tall-skinny / small-N / small-K GEMMs of the MLA projections at 16384 tokens (quantised on the GPU,
    float64 check on sampled rows)."""
    Mt = 16384
    g = torch.Generator().manual_seed(1003 + n_out)
    x = torch.randn(Mt, k_in, generator=g).bfloat16().cuda()
    w = (torch.randn(n_out, k_in, generator=g) * 0.02).bfloat16().cuda()
    xq, xs = K.quantize_fp8_rowwise(x)
    wq, ws = K.quantize_fp8_blockwise(w)
    out = K.fp8_matmul_dsv3(xq, wq.t(), xs, ws.t(), out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert K.device_status() == 0
    rows = torch.tensor([0, 127, 128, 4097, 9999, 16383])
    ref = O.fp8_matmul_f64(xq[rows.cuda()].view(torch.uint8).cpu(), wq.view(torch.uint8).cpu().t(),
                           xs[rows.cuda()].cpu(), ws.cpu().t())
    err = rel_fro(out[rows.cuda()], ref)
    print(f"MLA {k_in}->{n_out}: rel-Fro {err:.3e}")
    assert err <= TOL and err <= 2e-5
    out16 = K.fp8_matmul_dsv3(xq, wq.t(), xs, ws.t())
    assert_bf16_close(out16[rows.cuda()], ref, "bf16 output")


@pytest.mark.parametrize("name", ["ragged", "empty_first_last", "wide_k"])
def test_grouped_gemm_backward(K, name):
    """moe_grouped_gemm is differentiable here (it is not in the reference): grouped dgrad in one launch,
    weight gradient per expert, both with the arithmetic of the dense backward."""
    E, d_in, d_out, counts = GROUPED[name]
    x, w, starts, ends = _grouped_case(E, d_in, d_out, counts, seed=40 + len(name))
    g = torch.Generator().manual_seed(41)
    dy = torch.randn(x.shape[0], d_out, generator=g).bfloat16()
    ref_dx, ref_dw = O.grouped_gemm_fp8_backward_f64(x, w, starts, ends, dy)
    xg = x.cuda().requires_grad_(True)
    wg = w.float().cuda().requires_grad_(True)
    out = K.moe_grouped_gemm(xg, wg, starts.cuda(), ends.cuda(), dtype=torch.bfloat16)
    out.backward(dy.cuda())
    torch.cuda.synchronize()
    assert K.device_status() == 0
    assert xg.grad.dtype == torch.bfloat16 and wg.grad.dtype == torch.float32
    assert_bf16_close(xg.grad, ref_dx, "grouped dgrad")
    assert_bf16_close(wg.grad.to(torch.bfloat16), ref_dw, "grouped wgrad")
    for e, c in enumerate(counts):
        if c == 0:
            assert torch.all(wg.grad[e] == 0)


def test_config2_backward_full_size_sampled(K):
    """Forward + backward of FP8MatmulFunction at the FFN width (x [16384, 7168], W [18432, 7168], dy [16384, 18432]),
    i.e. the step the benchmark times, with the fused quantiser passes in the loop.  dgrad is checked on sampled token
    rows, wgrad on sampled weight rows (all 7168 columns each), both against the float64 product of operands the CPU
    oracle quantised (src/kernels.py:763-794: dy row-wise, dy^T row-wise, x row-wise then re-quantised in blocks)."""
    M, Kd, N = 16384, 7168, 18432
    g = torch.Generator().manual_seed(1002)
    x = torch.randn(M, Kd, generator=g).bfloat16()
    w = torch.randn(N, Kd, generator=g) * 0.02
    dy = torch.randn(M, N, generator=g).bfloat16()
    xg = x.cuda().requires_grad_(True)
    wg = w.cuda().requires_grad_(True)
    out = K.FP8MatmulFunction.apply(xg, wg, False)
    out.backward(dy.cuda())
    torch.cuda.synchronize()
    assert K.device_status() == 0
    assert xg.grad.shape == (M, Kd) and wg.grad.shape == (N, Kd) and wg.grad.dtype == torch.float32
    wq, ws = O.quantize_blockwise(w, 128, 128)
    # dgrad: sampled token rows
    rows = torch.tensor([0, 1, 127, 128, 4097, 8191, 12345, 16383])
    dq, ds = O.quantize_rowwise(dy[rows], 128)
    ref_dx = O.fp8_matmul_f64(dq, wq, ds, ws)
    assert_bf16_close(xg.grad[rows.cuda()], ref_dx, "C2 dgrad")
    err_dx = rel_fro(xg.grad[rows.cuda()].float(), ref_dx)
    # wgrad: sampled weight rows; the reduction runs over all 16384 tokens
    nrows = torch.tensor([0, 127, 128, 255, 9000, 18431])
    dtq, dts = O.quantize_rowwise(dy[:, nrows].t().contiguous(), 128)
    xq, xs = O.quantize_rowwise(x, 128)
    xbq, xbs = O.requantize_row_to_block(xq, xs)
    ref_dw = O.fp8_matmul_f64(dtq, xbq, dts, xbs)
    assert_bf16_close(wg.grad[nrows.cuda()].to(torch.bfloat16), ref_dw, "C2 wgrad")
    err_dw = rel_fro(wg.grad[nrows.cuda()], ref_dw)
    # forward once more on sampled rows (bf16 result of the autograd path)
    ref_out = O.fp8_matmul_f64(xq[rows], wq.t(), xs[rows], ws.t())
    assert_bf16_close(out[rows.cuda()], ref_out, "C2 forward")
    print(f"C2 backward sampled: dgrad rel-Fro {err_dx:.3e}, wgrad rel-Fro {err_dw:.3e} (bf16 results)")
    assert err_dx < 4e-3 and err_dw < 4e-3          # bf16 rounding alone is 1.7e-3


def test_config4_grouped_gemm_literal_routing_sampled(K):
    """Grouped GEMMs of the MoE configuration at full size: 256 experts, 32768 tokens, top-8 (262144 rows), d = 7168,
    up-projection 7168 -> 4096 and down-projection 2048 -> 7168, with the row ranges that the literal routing
    specification produces (sigmoid scores + bias ~ N(0, 1): about 30 experts receive rows, several receive every
    token).  Gaps of a few rows that belong to no expert are inserted between some experts and a canary is written
    everywhere first.  Sampled rows - the first and last row of several experts among them - are checked against
    the float64 product."""
    from cinnamon_b200 import moe
    E, d, I, T, k = 256, 7168, 2048, 32768, 8
    g = torch.Generator(device="cuda").manual_seed(1004)
    xt = torch.randn(T, d, generator=g, device="cuda").bfloat16()
    router = torch.randn(E, d, generator=g, device="cuda") * 0.02
    bias = torch.randn(E, generator=g, device="cuda")
    r = moe.route(xt, router, bias, k)
    counts = r.counts.cpu()
    active = [e for e in range(E) if counts[e] > 0]
    assert int(counts.sum()) == T * k and len(active) < 64 and int(counts.max()) > 0.9 * T, "the literal routing is heavily skewed"
    # ranges with a 5-row gap in front of every third active expert
    starts, ends, pos = torch.zeros(E, dtype=torch.int64), torch.zeros(E, dtype=torch.int64), 0
    for e in range(E):
        if counts[e] > 0 and active.index(e) % 3 == 1:
            pos += 5
        starts[e], ends[e] = pos, pos + int(counts[e])
        pos = int(ends[e])
    R = pos + 9
    src = torch.zeros(R, dtype=torch.int64)
    for e in active:
        seg = r.token_indices[int(counts[:e].sum()):int(counts[:e + 1].sum())].cpu()
        src[int(starts[e]):int(ends[e])] = seg
    xq_t, xs_t = K.quantize_fp8_rowwise(xt)
    xq, xs = K.gather_quantized_rows(xq_t, xs_t, src.cuda())
    del xt, xq_t, xs_t
    covered = torch.zeros(R, dtype=torch.bool)
    for e in active:
        covered[int(starts[e]):int(ends[e])] = True
    sample = []
    for e in active[:4] + active[-3:] + [int(counts.argmax())]:
        s, t = int(starts[e]), int(ends[e])
        sample += [(e, s), (e, t - 1), (e, s + (t - s) // 2)]
        if t - s > 300:
            sample += [(e, s + 127), (e, s + 128), (e, t - 129)]
    rows = torch.tensor([p for _, p in sample])
    for name, d_in, d_out in (("up", d, 2 * I), ("down", I, d)):
        gw = torch.Generator(device="cuda").manual_seed(2004 + d_in)
        wq = torch.empty(E, d_out, d_in, dtype=torch.float8_e4m3fn, device="cuda")
        wsc = torch.empty(E, d_out // 128, d_in // 128, device="cuda")
        for e0 in range(0, E, 32):                                   # 32 experts at a time: the bf16 masters are large
            wpart = (torch.randn(32, d_out, d_in, generator=gw, device="cuda") * 0.02).bfloat16()
            wq[e0:e0 + 32], wsc[e0:e0 + 32] = K.quantize_expert_weights(wpart)
        del wpart
        if name == "up":
            aq, asc = xq, xs
        else:
            h = torch.randn(R, I, generator=gw, device="cuda").bfloat16()
            aq, asc = K.quantize_fp8_rowwise(h)
            del h
        out = torch.full((R, d_out), 777.0, dtype=torch.bfloat16, device="cuda")
        K.fp8_grouped_gemm(aq, asc, wq, wsc, starts.cuda(), ends.cuda(), out=out)
        torch.cuda.synchronize()
        assert K.device_status() == 0
        untouched = (out[(~covered).cuda()] == 777.0).all()
        assert bool(untouched), f"{name}: rows that belong to no expert were written"
        got = out[rows.cuda()].float().cpu()
        worst = 0.0
        for i, (e, p) in enumerate(sample):
            ref = O.fp8_matmul_f64(aq[p:p + 1].view(torch.uint8).cpu(), wq[e].view(torch.uint8).cpu().t(),
                                   asc[p:p + 1].cpu(), wsc[e].cpu().t())
            assert_bf16_close(got[i:i + 1].to(torch.bfloat16), ref, f"{name} row {p} of expert {e}")
            worst = max(worst, rel_fro(got[i:i + 1], ref))
        print(f"C4 {name}-projection, {len(active)} active experts, {len(sample)} sampled rows: worst rel-Fro {worst:.3e} (bf16)")
        del wq, wsc, out


FUSED_WGRAD = {
    "ragged": (6, 512, 256, [5, 0, 130, 1, 257, 64]),
    "one_owns_all": (4, 256, 512, [0, 0, 700, 0]),
    "empty_first_last": (5, 256, 256, [0, 128, 0, 129, 0]),
    "many_small": (16, 256, 256, [1, 2, 3, 127, 128, 129, 0, 0, 255, 256, 257, 16, 17, 15, 64, 1]),
}


@pytest.mark.parametrize("counts", [[255, 256, 256, 128], [256, 256, 256, 129], [0, 1, 128, 129, 127, 0, 200], [130, 600, 0, 20], [1300, 700]])
def test_grouped_weight_gradients_of_short_and_long_experts(K, counts):
    """None, one, two and more K blocks per expert, on both sides of two on average, several tiles per pair of SMs: the bits of the per-expert
    loop in every type of the gradient."""
    E, d_in, d_out = len(counts), 1792, 1536
    x, w, starts, ends = _grouped_case(E, d_in, d_out, counts, seed=sum(counts), gap=5)
    dy = torch.randn(x.shape[0], d_out, generator=torch.Generator().manual_seed(E)).bfloat16()
    xq, xs = K.quantize_fp8_rowwise(x.cuda())
    args = (dy.cuda(), xq, xs, starts.cuda(), ends.cuda(), E, d_in, d_out)
    loop = K.fp8_grouped_wgrad(*args, w_dtype=torch.float32, fused=False)
    assert torch.equal(K.fp8_grouped_wgrad(*args, w_dtype=torch.float32, fused=True), loop)
    assert torch.equal(K.fp8_grouped_wgrad(*args, w_dtype=torch.bfloat16, fused=True), K.fp8_grouped_wgrad(*args, w_dtype=torch.bfloat16, fused=False))
    assert all(bool((loop[e] == 0).all()) == (c == 0) for e, c in enumerate(counts))
    assert K.device_status() == 0


def test_grouped_weight_gradient_of_a_thousand_experts(K):
    """The largest number of experts of one call, most of them empty."""
    E, d = 1024, 256
    counts = [(e % 7 == 0) * (e % 5) for e in range(E)]
    x, w, starts, ends = _grouped_case(E, d, d, counts, seed=3, gap=2)
    dy = torch.randn(x.shape[0], d, generator=torch.Generator().manual_seed(4)).bfloat16()
    xq, xs = K.quantize_fp8_rowwise(x.cuda())
    args = (dy.cuda(), xq, xs, starts.cuda(), ends.cuda(), E, d, d)
    for dtype in (torch.float32, torch.bfloat16):
        assert torch.equal(K.fp8_grouped_wgrad(*args, w_dtype=dtype, fused=True), K.fp8_grouped_wgrad(*args, w_dtype=dtype, fused=False))
    assert K.device_status() == 0


@pytest.mark.parametrize("name", list(FUSED_WGRAD))
def test_grouped_weight_gradient_in_one_gemm(K, name):
    """cinn_fp8_grouped_wgrad_fused (segments padded to tiles on the device, two quantiser launches, one grouped-K
    GEMM, no host read-back) against the float64 oracle and against the per-expert loop, whose bytes and sums it
    must reproduce exactly; a gap of rows that belong to no expert and canary values in dW."""
    E, d_in, d_out, counts = FUSED_WGRAD[name]
    x, w, starts, ends = _grouped_case(E, d_in, d_out, counts, seed=60 + len(name), gap=7)
    g = torch.Generator().manual_seed(61)
    dy = torch.randn(x.shape[0], d_out, generator=g).bfloat16()
    _, ref_dw = O.grouped_gemm_fp8_backward_f64(x, w, starts, ends, dy)
    xq, xs = K.quantize_fp8_rowwise(x.cuda())
    args = (dy.cuda(), xq, xs, starts.cuda(), ends.cuda(), E, d_in, d_out)
    fused = K.fp8_grouped_wgrad(*args, w_dtype=torch.float32, fused=True)
    loop = K.fp8_grouped_wgrad(*args, w_dtype=torch.float32, fused=False)
    torch.cuda.synchronize()
    assert K.device_status() == 0
    assert torch.equal(fused, loop), float((fused - loop).abs().max())
    assert_bf16_close(fused.to(torch.bfloat16), ref_dw, "grouped wgrad, one GEMM")
    for e, c in enumerate(counts):
        if c == 0:
            assert torch.all(fused[e] == 0)
    assert torch.equal(K.fp8_grouped_wgrad(*args, w_dtype=torch.bfloat16, fused=True), fused.to(torch.bfloat16))
    # the same call that also hands back the row-wise quantisation of dY (one pass over dY for both): same dW bits,
    # and inside the expert ranges the bytes and scales of the row-wise quantiser
    both, gq, gs = K.fp8_grouped_wgrad(*args, w_dtype=torch.float32, fused=True, with_row_quant=True)
    wq, ws = K.quantize_fp8_rowwise(dy.cuda())
    assert torch.equal(both, fused)
    inside = torch.zeros(x.shape[0], dtype=torch.bool)
    for a, b in zip(starts.tolist(), ends.tolist()):
        inside[a:b] = True
    assert inside.any() and not inside.all()
    ins = inside.numpy()
    assert np.array_equal(bytes_of(gq)[ins], bytes_of(wq)[ins]) and np.array_equal(bits_of(gs)[ins], bits_of(ws)[ins])
    for dt in (torch.float16, torch.float32):                     # fp32 gradients take the two-pass route
        both, gq, gs = K.fp8_grouped_wgrad(dy.cuda().to(dt), *args[1:], w_dtype=torch.float32, fused=True, with_row_quant=True)
        wq, ws = K.quantize_fp8_rowwise(dy.cuda().to(dt))
        assert torch.equal(both, fused)
        assert np.array_equal(bytes_of(gq)[ins], bytes_of(wq)[ins]) and np.array_equal(bits_of(gs)[ins], bits_of(ws)[ins])


def test_zero_rows_outside_ranges(K):
    """cinn_zero_rows_outside clears exactly the rows that no range covers (gaps, empty / reversed / overlapping /
    out-of-bounds ranges, a row size that is not a multiple of 16), and the grouped input gradient built on it
    gives zero rows where no expert has rows."""
    import ctypes
    from cinnamon_b200 import _lib
    dev = torch.device("cuda")
    for T, row_bytes in ((1000, 256), (517, 36), (128, 16)):
        buf = torch.full((T, row_bytes), 7, dtype=torch.uint8, device=dev)
        starts = torch.tensor([-5, 40, 300, 290, 700, 650, 990], dtype=torch.int64, device=dev)
        ends = torch.tensor([10, 40, 420, 310, 650, 660, 5000], dtype=torch.int64, device=dev)
        _lib.check(_lib.lib.cinn_zero_rows_outside(ctypes.c_void_p(buf.data_ptr()), T, row_bytes, ctypes.c_void_p(starts.data_ptr()),
                                                   ctypes.c_void_p(ends.data_ptr()), starts.numel(), None), "zero")
        covered = torch.zeros(T, dtype=torch.bool)
        for s, e in zip(starts.tolist(), ends.tolist()):
            covered[max(s, 0):max(min(e, T), 0)] = True
        want = torch.where(covered[:, None], torch.tensor(7, dtype=torch.uint8), torch.tensor(0, dtype=torch.uint8)).expand(T, row_bytes)
        assert torch.equal(buf.cpu(), want)
    g = torch.Generator(device=dev).manual_seed(5)
    E, d_in, d_out, T = 3, 256, 384, 700
    dy = torch.randn(T, d_out, generator=g, device=dev).to(torch.bfloat16)
    w = (torch.randn(E, d_out, d_in, generator=g, device=dev) * 0.05).to(torch.bfloat16)
    dq, dsc = K.quantize_fp8_rowwise(dy)
    wq, wsc = K.quantize_expert_weights(w)
    starts = torch.tensor([10, 300, 300], dtype=torch.int64, device=dev)
    ends = torch.tensor([200, 300, 650], dtype=torch.int64, device=dev)
    dx = K.fp8_grouped_gemm_dgrad(dq, dsc, wq, wsc, starts, ends)
    assert torch.count_nonzero(dx[:10]) == 0 and torch.count_nonzero(dx[200:300]) == 0 and torch.count_nonzero(dx[650:]) == 0
    assert torch.count_nonzero(dx[10:200]) > 0 and torch.isfinite(dx.float()).all()


@pytest.mark.parametrize("M,N,Kd", [(1, 128, 128), (1, 4, 16), (33, 200, 144), (97, 1000, 1040), (128, 1024, 512), (64, 130, 2048),
                                    (128, 8320, 256), (5, 19072, 384), (31, 8192, 1152)])
@pytest.mark.parametrize("dtype,rs,div", [(torch.bfloat16, False, "full"), (torch.float32, True, "full"), (torch.float16, False, "rn")])
def test_linear_on_few_rows_in_one_kernel(K, M, N, Kd, dtype, rs, div):
    """Quantising and multiplying in one kernel (one to eight CTAs per column tile) against the product of what the quantisers give,
    in 64 bits: fp32 sums over K blocks (2^-23 per addition of partial products) and one rounding to bf16."""
    g = torch.Generator(device="cuda").manual_seed(M + N + Kd)
    x = torch.randn(M, Kd, device="cuda", generator=g).mul_(3).to(dtype)
    w = torch.randn(N, Kd, device="cuda", generator=g).mul_(0.02)
    mode = K.get_div_mode()
    K.set_div_mode(div)
    try:
        out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        assert K._L.cinn_fp8_linear_few(K._ptr(x), K._DTYPE_TAG[dtype], Kd, int(rs), K._ptr(w), Kd, K._ptr(out), M, N, Kd, K._DIV_MODE, K._stream(x)) == 0
        xq, xs = K.quantize_fp8_rowwise(x, 128, rs)
        wq, ws = K.quantize_fp8_blockwise(w)
        whole = K._gemm(xq, xs, wq, 0, ws, ws.stride(1), ws.stride(0), M, N, Kd, torch.bfloat16, whole=True)
    finally:
        K.set_div_mode(mode)
    a = xq.double() * xs.double().repeat_interleave(128, 1)[:, :Kd]
    b = wq.double() * ws.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)[:, :Kd]
    ref, size = a @ b.t(), a.abs() @ b.abs().t()
    assert bool(((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + size * (Kd + 64) * 2.0 ** -23).all())
    if N > 16384 or Kd <= 128:                          # one CTA per column tile: the sums of the separate kernels, in their order
        assert torch.equal(out, whole)
    else:
        assert float((out.double() - whole.double()).norm() / whole.double().norm()) < 2.0 ** -9


@pytest.mark.parametrize("M,N,Kd", [(1, 128, 256), (128, 1024, 512), (82, 3776, 512), (4, 1344, 1024), (33, 200, 144), (17, 1000, 656)])
@pytest.mark.parametrize("dtype,rs", [(torch.bfloat16, True), (torch.float32, False)])
def test_linear_on_few_rows_has_the_bits_of_two_kernels(K, M, N, Kd, dtype, rs):
    """One K block per CTA: the cluster scales and adds the products in one step, in the order of the separate kernels."""
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N + Kd)
    layer = K.FP8Linear(Kd, N, round_scale=rs).cuda()
    x = torch.randn(M, Kd, device="cuda", generator=g).mul_(3).to(dtype)
    n = K.launch_count
    with torch.no_grad():
        out = layer(x)
    assert K.launch_count - n == 1
    xq, xs = K.quantize_fp8_rowwise(x, 128, rs)
    wq, ws = K.quantize_fp8_blockwise(layer.weight.detach())
    assert torch.equal(out, K._gemm(xq, xs, wq, 0, ws, ws.stride(1), ws.stride(0), M, N, Kd, torch.bfloat16, whole=True))


def test_linear_on_few_rows_any_alignment(K):
    """One launch for rows that fit, two for those that do not (rows off 16-byte boundaries, strides, a reduction too long for it to
    pay); the same result."""
    g = torch.Generator(device="cuda").manual_seed(5)
    lin = K.FP8Linear(272, 384).cuda()
    x = torch.randn(20, 272, device="cuda", generator=g, dtype=torch.float32).to(torch.bfloat16)
    with torch.no_grad():
        n = K.launch_count
        ref = lin(x)
        assert K.launch_count - n == 1
        odd = torch.empty(20 * 272 + 3, device="cuda", dtype=torch.bfloat16)[3:].view(20, 272).copy_(x)
        wide = torch.empty(20, 300, device="cuda", dtype=torch.bfloat16)[:, 4:276].copy_(x)
        turned = x.t().contiguous().t()
        for other, few in ((odd, 2), (wide, 2), (turned, 2), (x.view(4, 5, 272), 1)):
            n = K.launch_count
            y = lin(other).reshape(20, 384)
            assert K.launch_count - n >= 2 if few == 2 else K.launch_count - n == 1
            assert float((y.double() - ref.double()).norm() / ref.double().norm()) < 2.0 ** -9
        long = K.FP8Linear(7168, 2048).cuda()
        n = K.launch_count
        long(torch.randn(4, 7168, device="cuda"))
        assert K.launch_count - n >= 2


@pytest.mark.parametrize("M,Kd,kernels", [(8, 512, 1), (33, 512, 2), (128, 128, 1), (128, 512, 2)])
def test_linear_on_few_rows_under_capture(K, M, Kd, kernels):
    """Outside a capture one kernel; inside one, where a launch costs next to nothing, two for many rows with an exchange between CTAs: the
    same bits."""
    lin = K.FP8Linear(Kd, 1024).cuda()
    x = torch.randn(M, Kd, device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).to(torch.bfloat16)
    with torch.no_grad():
        n = K.launch_count
        ref = lin(x)
        assert K.launch_count - n == 1
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            n = K.launch_count
            out = lin(x)
            assert K.launch_count - n == kernels
        g.replay()
    assert torch.equal(out, ref)
    del g


@pytest.mark.parametrize("M", [1, 31, 32, 33, 64, 65, 97, 128])
@pytest.mark.parametrize("dtype,special", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, True)])
def test_linear_on_few_rows_in_passes_of_32(K, M, dtype, special):
    """One, two or four passes over the rows of x, also with NaN and infinity in x and in the weight: the bits of two kernels."""
    g = torch.Generator(device="cuda").manual_seed(M)
    lin = K.FP8Linear(400, 264).cuda()
    x = torch.randn(M, 400, device="cuda", generator=g).mul_(3)
    if special:
        x[0, 7], x[M // 2, 130], x[M - 1, 399] = float("nan"), float("inf"), -float("inf")
        with torch.no_grad():
            lin.weight[5, 9], lin.weight[200, 300], lin.weight[263, 399] = float("nan"), float("inf"), -float("inf")
    x = x.to(dtype)
    with torch.no_grad():
        n = K.launch_count
        out = lin(x)
    assert K.launch_count - n == 1
    xq, xs = K.quantize_fp8_rowwise(x, 128, lin.round_scale)
    wq, ws = K.quantize_fp8_blockwise(lin.weight.detach())
    ref = K._gemm(xq, xs, wq, 0, ws, ws.stride(1), ws.stride(0), M, 264, 400, torch.bfloat16, whole=True)
    assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out.nan_to_num(7.0), ref.nan_to_num(7.0))
    assert not special or (bool(ref.isnan().any()) and (M == 1 or bool(ref.isfinite().any())))       # (one row has them all)
