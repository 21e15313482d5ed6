"""Sparse attention: the float64 oracle against the reference's own outputs (golden vectors made by running its
Triton kernels in the CPU interpreter), and the CUDA kernels against both."""
import os

import numpy as np
import pytest
import torch

from oracle import sparse_attention_oracle as SO

HERE = os.path.dirname(os.path.abspath(__file__))
CASES = ["small", "ragged_dims", "causal_topk", "duplicates"]


@pytest.fixture(scope="module")
def vectors():
    return np.load(os.path.join(HERE, "golden", "sparse_attention_vectors.npz"))


def _case(vectors, name):
    t = {k: torch.from_numpy(vectors[f"{name}/{k}"]) for k in
         ("q", "k", "v", "idx", "out", "attn", "grad_out", "dq", "dk", "dv")}
    t["scale"] = float(vectors[f"{name}/scale"])
    return t


@pytest.mark.parametrize("name", CASES)
def test_oracle_matches_reference_vectors(vectors, name):
    c = _case(vectors, name)
    out, attn, _ = SO.forward(c["q"], c["k"], c["v"], c["idx"], c["scale"])
    torch.testing.assert_close(out.float(), c["out"], rtol=2e-5, atol=2e-6)
    torch.testing.assert_close(attn.float(), c["attn"], rtol=2e-5, atol=2e-7)
    dq, dk, dv = SO.backward(c["q"], c["k"], c["v"], c["idx"], c["scale"], c["grad_out"])
    torch.testing.assert_close(dq.float(), c["dq"], rtol=5e-5, atol=5e-6)
    torch.testing.assert_close(dk.float(), c["dk"], rtol=5e-5, atol=5e-6)
    torch.testing.assert_close(dv.float(), c["dv"], rtol=5e-5, atol=5e-6)


def test_oracle_backward_is_the_derivative():
    """The analytic backward against autograd through the float64 forward."""
    g = torch.Generator().manual_seed(9)
    q, k = (torch.randn(1, 2, 12, 8, generator=g, dtype=torch.float64).requires_grad_(True) for _ in range(2))
    v = torch.randn(1, 2, 12, 4, generator=g, dtype=torch.float64).requires_grad_(True)
    idx = torch.randint(0, 12, (1, 12, 5), generator=g)
    go = torch.randn(1, 2, 12, 4, generator=g, dtype=torch.float64)
    out, _, _ = SO.forward(q, k, v, idx, 0.3)
    ref = torch.autograd.grad(out, (q, k, v), go)
    got = SO.backward(q.detach(), k.detach(), v.detach(), idx, 0.3, go)
    for a, b in zip(got, ref):
        torch.testing.assert_close(a, b, rtol=1e-10, atol=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_kernels_match_reference_vectors(vectors, name):
    from cinnamon_b200 import kernels as K
    c = _case(vectors, name)
    q, k, v = (c[n].cuda().requires_grad_(True) for n in ("q", "k", "v"))
    out, attn = K.sparse_attention(q, k, v, c["idx"].cuda(), c["scale"])
    assert out.dtype == torch.float32 and attn.dtype == torch.float32
    torch.testing.assert_close(out.cpu(), c["out"], rtol=2e-5, atol=2e-6)
    torch.testing.assert_close(attn.cpu(), c["attn"], rtol=2e-5, atol=2e-7)
    out.backward(c["grad_out"].cuda())
    torch.testing.assert_close(q.grad.cpu(), c["dq"], rtol=5e-5, atol=5e-6)
    torch.testing.assert_close(k.grad.cpu(), c["dk"], rtol=5e-5, atol=5e-6)
    torch.testing.assert_close(v.grad.cpu(), c["dv"], rtol=5e-5, atol=5e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("shape", [(2, 4, 96, 32, 192, 64), (1, 3, 70, 128, 64, 64), (1, 2, 33, 7, 20, 6), (1, 1, 300, 40, 8, 136)])
def test_kernels_match_oracle(dtype, shape):
    """Model-like sizes (192-wide PoPE queries, 64-wide values), K larger than the sequence, odd sizes that take the
    scalar path; fp32 results against the float64 oracle on the same (already rounded) inputs."""
    from cinnamon_b200 import kernels as K
    B, H, L, Ks, Dqk, Dv = shape
    g = torch.Generator().manual_seed(sum(shape))
    q, k = (torch.randn(B, H, L, Dqk, generator=g).to(dtype) for _ in range(2))
    v = torch.randn(B, H, L, Dv, generator=g).to(dtype)
    idx = torch.randint(0, L, (B, L, Ks), generator=g)
    idx[:, :, 0] = torch.arange(L)                       # every query sees at least itself ...
    idx[0, 5, :] = L - 1                                 # ... except this one, which has no valid key at all
    go = torch.randn(B, H, L, Dv, generator=g).to(dtype)
    scale = Dqk ** -0.5
    ref_out, ref_attn, _ = SO.forward(q, k, v, idx, scale)
    qc, kc, vc = (t.cuda().requires_grad_(True) for t in (q, k, v))
    out, attn = K.sparse_attention(qc, kc, vc, idx.cuda(), scale)
    assert out.dtype == dtype and attn.shape == (B, H, L, Ks)
    tol = {torch.float32: 1e-5, torch.bfloat16: 8e-3, torch.float16: 1e-3}[dtype]       # rounding of the returned output
    torch.testing.assert_close(out.float().cpu().double(), ref_out, rtol=tol, atol=tol)
    torch.testing.assert_close(attn.cpu().double(), ref_attn, rtol=2e-5, atol=1e-7)
    assert torch.all(out[0, :, 5] == 0) and torch.all(attn[0, :, 5] == 0)
    out.backward(go.cuda())
    # the kernel differentiates with the fp32 output it saved; the oracle with its own float64 output
    ref = SO.backward(q, k, v, idx, scale, go)
    for name, got, want in zip(("dq", "dk", "dv"), (qc.grad, kc.grad, vc.grad), ref):
        assert got.dtype == dtype
        err = (got.float().cpu().double() - want).norm() / want.norm()
        assert err < {torch.float32: 2e-6, torch.bfloat16: 4e-3, torch.float16: 5e-4}[dtype], (name, float(err))


@pytest.mark.gpu
def test_edge_shapes():
    """No indices at all, indices outside the sequence, one query, a list much longer than the sequence."""
    from cinnamon_b200 import kernels as K
    g = torch.Generator().manual_seed(77)
    q, k, v = (torch.randn(1, 2, 9, 16, generator=g).cuda() for _ in range(3))
    out, attn = K.sparse_attention(q, k, v, torch.zeros(1, 9, 0, dtype=torch.int64, device="cuda"))
    assert attn.shape == (1, 2, 9, 0) and torch.all(out == 0)
    idx = torch.randint(-3, 14, (1, 9, 40), generator=g)                     # some below 0, some beyond L - 1
    ref_out, ref_attn, _ = SO.forward(q.cpu(), k.cpu(), v.cpu(), idx, 0.25)
    out, attn = K.sparse_attention(q, k, v, idx.cuda(), 0.25)
    torch.testing.assert_close(out.cpu().double(), ref_out, rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(attn.cpu().double(), ref_attn, rtol=2e-5, atol=1e-7)
    q1, k1, v1 = (t[:, :, :1].contiguous() for t in (q, k, v))
    out, attn = K.sparse_attention(q1, k1, v1, torch.zeros(1, 1, 3, dtype=torch.int64, device="cuda"))
    torch.testing.assert_close(out, v1.expand_as(out))                       # the only key, listed three times
    torch.testing.assert_close(attn, torch.full_like(attn, 1.0 / 3.0))


@pytest.mark.gpu
def test_argument_checks():
    from cinnamon_b200 import kernels as K
    q = torch.randn(1, 1, 4, 8)
    with pytest.raises(AssertionError):
        K.sparse_attention(q, q, q, torch.zeros(1, 4, 2, dtype=torch.int64))


@pytest.mark.gpu
def test_backward_with_gradient_buffers_at_odd_addresses():
    """A C caller may hand in gradient buffers that start on a 4-byte boundary only (a slice of an arena): the
    kernel then must not use its 16- or 8-byte atomics.  Same result as with aligned buffers."""
    import ctypes
    from cinnamon_b200 import kernels as K
    lib = K._lib.lib
    g = torch.Generator().manual_seed(31)
    B, H, L, Kk, dqk, dv = 1, 2, 24, 6, 16, 8
    q, k = (torch.randn(B, H, L, dqk, generator=g).cuda() for _ in range(2))
    v = torch.randn(B, H, L, dv, generator=g).cuda()
    idx = (torch.rand(B, L, Kk, generator=g) * (torch.arange(L).view(1, L, 1) + 1)).long().cuda()
    go = torch.randn(B, H, L, dv, generator=g).cuda()
    out = torch.empty(B, H, L, dv, device="cuda")
    lse = torch.empty(B, H, L, device="cuda")
    attn = torch.empty(B, H, L, Kk, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())                                        # noqa: E731
    K._lib.check(lib.cinn_sparse_attn_fwd(p(q), p(k), p(v), 1, p(idx), p(out), p(lse), p(attn), B, H, L, Kk, dqk, dv, 0.25, st), "fwd")
    grads = []
    for shift in (0, 1):                                                                # 0: 16-byte aligned, 1: +4 bytes
        arena = torch.zeros(3 * B * H * L * dqk + 8, device="cuda")
        n_qk, n_v = B * H * L * dqk, B * H * L * dv
        gq, gk, gv = arena[shift:shift + n_qk], arena[shift + n_qk:shift + 2 * n_qk], arena[shift + 2 * n_qk:shift + 2 * n_qk + n_v]
        assert (gq.data_ptr() % 16 == 0) == (shift == 0)
        K._lib.check(lib.cinn_sparse_attn_bwd(p(go), 1, p(out), p(lse), p(q), p(k), p(v), 1, p(idx), p(gq), p(gk), p(gv), B, H, L,
                                              Kk, dqk, dv, 0.25, st), "bwd")
        torch.cuda.synchronize()
        grads.append([t.clone() for t in (gq, gk, gv)])
    for a, b in zip(*grads):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-6)
    assert K.device_status() == 0


@pytest.fixture(params=["dense", "gather"])
def attention_path(request):
    """Every shape the tiles can take through the tiles, and through the gathers."""
    from cinnamon_b200 import kernels as K
    before = K._L.cinn_set_sparse_attn_dense(1 if request.param == "dense" else 0)
    yield request.param
    K._L.cinn_set_sparse_attn_dense(before)
    assert K.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("shape", [(1, 2, 1, 1, 64, 64), (1, 2, 127, 33, 64, 64), (2, 1, 129, 32, 192, 64), (1, 2, 300, 40, 72, 100),
                                   (1, 1, 385, 70, 128, 128), (1, 1, 260, 7, 20, 6)])
def test_tiles_and_gathers(dtype, shape, attention_path):
    """Partial tiles, one to four key tiles, padded and split widths, duplicates, queries without a valid key, indices
    outside the sequence.  The same bounds for both paths: fp32 arithmetic on the given inputs."""
    from cinnamon_b200 import kernels as K
    B, H, L, Ks, Dqk, Dv = shape
    g = torch.Generator().manual_seed(sum(shape))
    q, k, go = (torch.randn(B, H, L, d, generator=g).to(dtype) for d in (Dqk, Dqk, Dv))
    v = torch.randn(B, H, L, Dv, generator=g).to(dtype)
    idx = torch.randint(-2, L + 2, (B, L, Ks), generator=g)
    idx[:, L // 2] = L + 1                                # a query without any valid key
    scale = Dqk ** -0.5
    ref_out, ref_attn, _ = SO.forward(q, k, v, idx, scale)
    qc, kc, vc = (t.cuda().requires_grad_(True) for t in (q, k, v))
    out, attn = K.sparse_attention(qc, kc, vc, idx.cuda(), scale)
    tol = {torch.float32: 1e-5, torch.bfloat16: 8e-3, torch.float16: 1e-3}[dtype]       # rounding of the returned output
    torch.testing.assert_close(out.float().cpu().double(), ref_out, rtol=tol, atol=tol)
    torch.testing.assert_close(attn.cpu().double(), ref_attn, rtol=2e-5, atol=1e-7)
    out.backward(go.cuda())
    for name, got, want in zip(("dq", "dk", "dv"), (qc.grad, kc.grad, vc.grad), SO.backward(q, k, v, idx, scale, go)):
        assert got.dtype == dtype
        err = (got.float().cpu().double() - want).norm() / want.norm().clamp(min=1e-30)
        assert err < {torch.float32: 2e-6, torch.bfloat16: 4e-3, torch.float16: 5e-4}[dtype], (name, float(err))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(1, 2, 513, 64, 72, 64), (1, 2, 400, 24, 64, 100), (2, 40, 257, 32, 64, 64), (1, 75, 385, 512, 64, 40)])
def test_tiles_with_wide_scores(dtype, shape):
    """Scores of up to some 50, larger for later keys, so that the exponentials' reference point moves in late key tiles; with a
    block per SM and with two, lists of a power of two of slots (permuted four at a time) and others.  A score of 50 is known
    to 2^-22 of itself, its exponential to 50 x 2^-22 = 1.2e-5: the bound is three times that."""
    from cinnamon_b200 import kernels as K
    B, H, L, Ks, Dqk, Dv = shape
    g = torch.Generator().manual_seed(sum(shape))
    q, k = torch.randn(B, H, L, Dqk, generator=g), torch.randn(B, H, L, Dqk, generator=g)
    q, k = (q * 1.2).to(dtype), (k * (0.2 + torch.arange(L).view(1, 1, L, 1) / L)).to(dtype)
    v = torch.randn(B, H, L, Dv, generator=g).to(dtype)
    idx = torch.randint(0, L, (B, L, Ks), generator=g)
    before = K._L.cinn_set_sparse_attn_dense(1)
    try:
        out, attn = K.sparse_attention(q.cuda(), k.cuda(), v.cuda(), idx.cuda(), 1.0)
    finally:
        K._L.cinn_set_sparse_attn_dense(before)
    heads = sorted({0, 1, H // 2, H - 1})
    ref_out, ref_attn, _ = SO.forward(q[:, heads], k[:, heads], v[:, heads], idx, 1.0)
    tol = {torch.float32: 4e-5, torch.bfloat16: 8e-3}[dtype]                            # bf16: rounding of the returned output
    torch.testing.assert_close(out[:, heads].float().cpu().double(), ref_out, rtol=tol, atol=tol)
    torch.testing.assert_close(attn[:, heads].cpu().double(), ref_attn, rtol=4e-5, atol=1e-7)
    assert K.device_status() == 0


@pytest.fixture
def released():
    """Gives the test's memory back: a later test counts what the allocator holds."""
    yield
    torch.cuda.empty_cache()


@pytest.mark.gpu
@pytest.mark.usefixtures("released")
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H", [3, 80])                    # a block per SM, two of them
@pytest.mark.parametrize("Ks", [4, 64, 24])
def test_tiles_with_probabilities_at_odd_addresses(dtype, H, Ks):
    """A C caller's probabilities may start on a 4-byte boundary only (a slice of an arena): still the tiles, without their
    16-byte stores.  The output has the same bits; the probabilities differ by whether score x scale is rounded before
    the sum of exponentials is taken off it: 2^-24 of a score below 16, so 1e-6 of the probability, and as much for the exponent."""
    import ctypes
    from cinnamon_b200 import kernels as K
    lib = K._lib.lib
    g = torch.Generator().manual_seed(H + Ks)
    B, L, dqk, dv = 1, 257, 64, 64
    tag = {torch.bfloat16: 0, torch.float32: 1}[dtype]
    q, k = (torch.randn(B, H, L, dqk, generator=g).to(dtype).cuda() for _ in range(2))
    v = torch.randn(B, H, L, dv, generator=g).to(dtype).cuda()
    idx = torch.randint(0, L, (B, L, Ks), generator=g).cuda()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())                                        # noqa: E731
    before = K._L.cinn_set_sparse_attn_dense(1)
    try:
        need = lib.cinn_sparse_attn_workspace_bytes(B, H, L, Ks, dqk, dv, tag, 0)
        assert need > 0
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")
        results = []
        for shift in (0, 1, 2, 3):
            n = B * H * L * Ks
            arena = torch.full((n + 8,), 7.0, device="cuda")
            attn = arena[shift:shift + n]
            assert attn.data_ptr() % 16 == 4 * shift
            out, lse = torch.empty(B, H, L, dv, device="cuda"), torch.empty(B, H, L, device="cuda")
            K._lib.check(lib.cinn_sparse_attn_fwd_ws(p(q), p(k), p(v), tag, p(idx), p(out), None, p(lse), p(attn), B, H, L, Ks, dqk, dv,
                                                     0.125, p(ws), need, st), "fwd")
            assert torch.all(arena[:shift] == 7) and torch.all(arena[shift + n:] == 7)
            results.append((out, lse, attn))
    finally:
        K._L.cinn_set_sparse_attn_dense(before)
    for out, lse, attn in results[1:]:
        assert torch.equal(out, results[0][0]) and torch.equal(lse, results[0][1])
        torch.testing.assert_close(attn, results[0][2], rtol=3e-6, atol=1e-9)
    assert K.device_status() == 0


@pytest.mark.gpu
@pytest.mark.usefixtures("released")
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H", [2, 160])                   # a block per SM, two of them
@pytest.mark.parametrize("keys,Ks", [(1, 200), (23, 33), (140, 120), (300, 512)])
def test_tiles_weigh_repeated_picks(dtype, H, keys, Ks):
    """Keys picked up to 200 times by a query: one key, a row of consecutive ones (sixteen counts a chunk), some of many; lists whose
    counts start on every byte of a word, the last query's among them."""
    from cinnamon_b200 import kernels as K
    B, L, Dqk, Dv = 1, 300, 64, 64
    g = torch.Generator().manual_seed(H + Ks)
    q, k = (torch.randn(B, H, L, Dqk, generator=g).to(dtype) for _ in range(2))
    v = torch.randn(B, H, L, Dv, generator=g).to(dtype)
    idx = torch.randint(0, keys, (B, L, Ks), generator=g)
    idx[0, ::3] += (torch.arange(0, L, 3) - keys).clamp(min=0)[:, None]                # the last keys before a query
    before = K._L.cinn_set_sparse_attn_dense(1)
    try:
        out, attn = K.sparse_attention(q.cuda(), k.cuda(), v.cuda(), idx.cuda())
    finally:
        K._L.cinn_set_sparse_attn_dense(before)
    heads = sorted({0, H // 2, H - 1})
    ref_out, ref_attn, _ = SO.forward(q[:, heads], k[:, heads], v[:, heads], idx, Dqk ** -0.5)
    tol = {torch.float32: 1e-5, torch.bfloat16: 8e-3}[dtype]                            # bf16: rounding of the returned output
    torch.testing.assert_close(out[:, heads].float().cpu().double(), ref_out, rtol=tol, atol=tol)
    torch.testing.assert_close(attn[:, heads].cpu().double(), ref_attn, rtol=2e-5, atol=1e-7)
    assert K.device_status() == 0


@pytest.mark.gpu
@pytest.mark.usefixtures("released")
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(1, 160, 300, 40, 192, 64), (2, 76, 257, 33, 128, 64), (1, 150, 385, 64, 192, 128), (1, 230, 250, 24, 128, 100),
                                   (4, 37, 400, 16, 64, 128), (1, 45, 2048, 128, 192, 64), (1, 60, 130, 100, 192, 64), (1, 80, 256, 512, 72, 72),
                                   (1, 37, 1500, 32, 192, 64)])
def test_tiles_of_many_heads(dtype, shape):
    """More blocks than SMs: every width of queries and values with one pair of warpgroups per CTA and two CTAs per SM, lists of a power
    of two of slots and others, heads in one and in several groups, the last of them smaller; and the shapes that keep two pairs."""
    from cinnamon_b200 import kernels as K
    B, H, L, Ks, Dqk, Dv = shape
    g = torch.Generator().manual_seed(sum(shape))
    q, k = (torch.randn(B, H, L, Dqk, generator=g).to(dtype) for _ in range(2))
    v = torch.randn(B, H, L, Dv, generator=g).to(dtype)
    idx = torch.randint(-2, L + 2, (B, L, Ks), generator=g)
    idx[:, L // 2] = L + 1                                # a query without any valid key
    before = K._L.cinn_set_sparse_attn_dense(1)
    try:
        out, attn = K.sparse_attention(q.cuda(), k.cuda(), v.cuda(), idx.cuda())
    finally:
        K._L.cinn_set_sparse_attn_dense(before)
    heads = sorted({0, H // 2, H - 2, H - 1})
    ref_out, ref_attn, _ = SO.forward(q[:, heads], k[:, heads], v[:, heads], idx, Dqk ** -0.5)
    tol = {torch.bfloat16: 8e-3, torch.float16: 1e-3}[dtype]                            # rounding of the returned output
    torch.testing.assert_close(out[:, heads].float().cpu().double(), ref_out, rtol=tol, atol=tol)
    torch.testing.assert_close(attn[:, heads].cpu().double(), ref_attn, rtol=2e-5, atol=1e-7)
    assert K.device_status() == 0


@pytest.mark.gpu
@pytest.mark.usefixtures("released")
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H", [2, 160])
def test_tiles_of_many_heads_fall_back(dtype, H):
    """A NaN key that some queries picked, a key picked more than 255 times: with a block per SM and with two, the numbers and the NaNs
    of the gathers."""
    from cinnamon_b200 import kernels as K
    g = torch.Generator().manual_seed(H)
    q, k, v = (torch.randn(1, H, 384, 64, generator=g).to(dtype).cuda() for _ in range(3))
    idx = torch.randint(0, 100, (1, 384, 264), generator=g).cuda()
    idx[idx == 17] = 18
    for nan in (True, False):
        if nan:
            k[0, H // 2, 300, 3] = float("nan")
            idx[0, 301:340, 5] = 300
        else:
            k.nan_to_num_(0.0)
            idx[0, 200, :] = 7
        got = []
        for mode in (1, 0):
            before = K._L.cinn_set_sparse_attn_dense(mode)
            try:
                got.append(K.sparse_attention(q, k, v, idx))
            finally:
                K._L.cinn_set_sparse_attn_dense(before)
        assert bool(torch.isnan(got[0][0][0, H // 2, 301:340]).all()) == nan and not torch.isnan(got[0][0][0, 0]).any()
        for a, b in zip(*got):
            torch.testing.assert_close(a, b, rtol=1e-5 if dtype == torch.float32 else 8e-3, atol=1e-6, equal_nan=True)
    assert K.device_status() == 0


@pytest.mark.gpu
def test_tiles_fall_back_on_the_device(attention_path):
    """What the tiles cannot express: a key picked more than 255 times, and rows nobody picked that hold NaN or infinity."""
    from cinnamon_b200 import kernels as K
    g = torch.Generator().manual_seed(3)
    q, k, v = (torch.randn(1, 1, 140, 64, generator=g) for _ in range(3))
    idx = torch.randint(0, 140, (1, 140, 300), generator=g)
    idx[idx == 17] = 18
    idx[0, 100] = 5
    ref_out, ref_attn, _ = SO.forward(q, k, v, idx, 0.2)
    go = torch.randn(1, 1, 140, 64, generator=g)
    ref = SO.backward(q, k, v, idx, 0.2, go)
    k[0, 0, 17], v[0, 0, 17] = float("nan"), float("inf")
    for _ in range(2):
        qc, kc, vc = (t.cuda().requires_grad_(True) for t in (q, k, v))
        out, attn = K.sparse_attention(qc, kc, vc, idx.cuda(), 0.2)
        out.backward(go.cuda())
        for got, want in zip((qc.grad, kc.grad, vc.grad), ref):
            assert float((got.cpu().double() - want).norm() / want.norm()) < 2e-6
        torch.testing.assert_close(out.cpu().double(), ref_out, rtol=1e-5, atol=1e-6)
        torch.testing.assert_close(attn.cpu().double(), ref_attn, rtol=2e-5, atol=1e-7)
        idx[0, 100, ::2] = 6                              # now only the rows that nobody picked
        clean = (q, torch.nan_to_num(k), torch.nan_to_num(v, posinf=0.0), idx, 0.2)
        (ref_out, ref_attn, _), ref = SO.forward(*clean), SO.backward(*clean, go)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("key", [17, 200, 300])
def test_a_nan_key_reaches_the_queries_that_picked_it(dtype, key):
    """A picked key that holds NaN, in the first, second or third key tile, the only one picked there: tiles and gathers give
    the same numbers and the same NaNs."""
    from cinnamon_b200 import kernels as K
    g = torch.Generator().manual_seed(key)
    q, k, v = (torch.randn(1, 2, 400, 64, generator=g).to(dtype) for _ in range(3))
    idx = torch.randint(0, 100, (1, 400, 24), generator=g)
    idx[idx == 17] = 18
    idx[0, 301:340, 5] = key
    k[0, 0, key, 3] = float("nan")
    got = []
    for mode in (1, 0):
        before = K._L.cinn_set_sparse_attn_dense(mode)
        try:
            out, attn = K.sparse_attention(q.cuda(), k.cuda(), v.cuda(), idx.cuda())
            got.append((out.cpu(), attn.cpu()))
        finally:
            K._L.cinn_set_sparse_attn_dense(before)
    assert torch.isnan(got[0][0][0, 0, 301:340]).all() and not torch.isnan(got[0][0][0, 1]).any()
    for a, b in zip(*got):
        torch.testing.assert_close(a, b, rtol=1e-5 if dtype == torch.float32 else 8e-3, atol=1e-6, equal_nan=True)
    assert K.device_status() == 0


def test_scratch_of_the_tiles_is_bounded():
    """No shape asks for more than 16 GiB, and the listed training shape for what its documentation says."""
    from cinnamon_b200 import _lib
    need = _lib.lib.cinn_sparse_attn_workspace_bytes
    assert 0 < need(32, 8, 1024, 128, 192, 64, _lib.F32, 0) < 0.8e9 and 0 < need(32, 8, 1024, 128, 192, 64, _lib.F32, 1) < 1.2e9
    for B, H, L, K in ((512, 8, 1024, 512), (64, 64, 4096, 512), (16, 64, 12000, 512), (4096, 16, 512, 256)):
        for dtype in (_lib.F32, _lib.BF16, _lib.F16):
            for backward in (0, 1):
                assert 0 <= need(B, H, L, K, 192, 128, dtype, backward) <= 16 << 30


@pytest.mark.gpu
def test_without_room_for_the_scratch_the_gathers_compute_the_call():
    """Memory for the tensors but not for the tiles' scratch: the call succeeds, with the gathers' numbers."""
    from cinnamon_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(9)
    B, H, L, k, dq, dv = 4, 8, 1024, 128, 192, 64
    q, kk, v = (torch.randn(B, H, L, d, generator=g, device="cuda").requires_grad_(True) for d in (dq, dq, dv))
    idx = torch.randint(0, L, (B, L, k), generator=g, device="cuda")
    need = K._L.cinn_sparse_attn_workspace_bytes(B, H, L, k, dq, dv, 1, 0)
    outputs = 4 * B * H * L * (dv + 1 + k)
    assert need > 1.3 * outputs
    before = K._L.cinn_set_sparse_attn_dense(0)
    want = [t.detach().clone() for t in K.sparse_attention(q, kk, v, idx)]
    K._L.cinn_set_sparse_attn_dense(before)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    limit = torch.cuda.memory_reserved() + int(1.1 * outputs) + (24 << 20)
    try:
        torch.cuda.set_per_process_memory_fraction(limit / torch.cuda.get_device_properties(0).total_memory)
        out, attn = K.sparse_attention(q, kk, v, idx)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(out, want[0]) and torch.equal(attn, want[1])
    tiles, _ = K.sparse_attention(q, kk, v, idx)
    assert not torch.equal(tiles, out)                            # (with room it is the tiles that compute it)
    torch.testing.assert_close(tiles, out, rtol=1e-5, atol=1e-5)
