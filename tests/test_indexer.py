"""Lightning indexer: oracle against the reference kernel's outputs (Triton interpreter), CUDA kernel against both."""
import os

import numpy as np
import pytest
import torch

from oracle import sparse_attention_oracle as SO

HERE = os.path.dirname(os.path.abspath(__file__))
CASES = ["model_like", "wide_head", "bf16_inputs", "narrow"]


@pytest.fixture(scope="module")
def vectors():
    return np.load(os.path.join(HERE, "golden", "indexer_vectors.npz"))


def _case(vectors, name):
    dt = torch.bfloat16 if int(vectors[f"{name}/bf16"]) else torch.float32
    q, k, w = (torch.from_numpy(vectors[f"{name}/{n}"]).to(dt) for n in ("q", "k", "w"))
    return q, k, w, torch.from_numpy(vectors[f"{name}/out"])


def _close_fp16(got, want64):
    """Within one fp16 rounding step of the float64 value (plus the fp32 accumulation noise near a tie)."""
    want = want64.float()
    tol = want.abs() * 2.0 ** -10 + 1e-4
    assert torch.all((got.float() - want).abs() <= tol), float(((got.float() - want).abs() - tol).max())


@pytest.mark.parametrize("name", CASES)
def test_oracle_matches_reference_vectors(vectors, name):
    q, k, w, out = _case(vectors, name)
    _close_fp16(out, SO.lightning_indexer(q, k, w))


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_kernel_matches_reference_vectors(vectors, name):
    from cinnamon_b200 import kernels as K
    q, k, w, out = _case(vectors, name)
    got = K.lightning_indexer_fused(q.cuda(), k.cuda(), w.cuda())
    assert got.dtype == torch.float16 and got.shape == out.shape
    # same fp16-rounded operands, fp32 sums in another order: at most one fp16 step apart, nearly always equal
    assert torch.all((got.cpu().float() - out.float()).abs() <= out.float().abs() * 2.0 ** -10 + 1e-4)
    assert float((got.cpu() != out).float().mean()) < 0.02
    _close_fp16(got.cpu(), SO.lightning_indexer(q, k, w))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_kernel_views_and_sizes(dtype):
    """The model's call shape (B, L, 4 heads of 64) plus a strided view of the keys."""
    from cinnamon_b200 import kernels as K
    g = torch.Generator().manual_seed(12)
    q = torch.randn(2, 257, 4, 64, generator=g).to(dtype)
    kfull = torch.randn(2, 300, 128, generator=g).to(dtype)
    w = torch.rand(2, 257, 4, generator=g).to(dtype)
    k = kfull[:, :, 64:]                                                     # pitched rows
    got = K.lightning_indexer_fused(q.cuda(), kfull.cuda()[:, :, 64:], w.cuda())
    _close_fp16(got.cpu(), SO.lightning_indexer(q, k, w))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 1), (2, 127, 129, 3, 20), (1, 128, 128, 4, 64), (1, 130, 257, 5, 72), (1, 40, 131, 3, 128),
                                   (1, 17, 70, 2, 136)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_tile_edges(shape, dtype):
    """Partial query and key tiles, padded widths, more heads than fit at once, and a row too wide for the tensor cores."""
    from cinnamon_b200 import kernels as K
    B, Lq, Lk, H, d = shape
    g = torch.Generator().manual_seed(sum(shape))
    q, k = torch.randn(B, Lq, H, d, generator=g).to(dtype), torch.randn(B, Lk, d, generator=g).to(dtype)
    w = torch.rand(B, Lq, H, generator=g).to(dtype)
    got = K.lightning_indexer_fused(q.cuda(), k.cuda(), w.cuda())
    _close_fp16(got.cpu(), SO.lightning_indexer(q, k, w))
    assert K.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 8), (2, 300, 517, 9, 64), (3, 129, 1000, 4, 128), (20, 260, 391, 2, 64), (1, 2000, 1537, 3, 72),
                                   (4, 200, 136, 10, 64)])
def test_runs_of_tiles(shape, dtype):
    """CTAs with several tiles: runs that cross query tiles, rings that go round, odd and even rows, one head more than the ring has room
    for; values past fp16's range turn into infinities as the reference's do."""
    from cinnamon_b200 import kernels as K
    B, Lq, Lk, H, d = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    q, k = torch.randn(B, Lq, H, d, device="cuda", generator=g).to(dtype), torch.randn(B, Lk, d, device="cuda", generator=g).to(dtype)
    w = torch.rand(B, Lq, H, device="cuda", generator=g).to(dtype)
    for _ in range(2):
        got = K.lightning_indexer_fused(q, k, w)
    want = torch.zeros(B, Lq, Lk, device="cuda", dtype=torch.float64)
    for h in range(H):
        want += (q[:, :, h].half().double() @ k.half().double().transpose(1, 2)).clamp_min(0) * w[:, :, h, None].double()
    _close_fp16(got, want)
    if dtype == torch.bfloat16:
        q[0, 0], k[0, 0] = 0, 0
        q[0, 0, :, 0], k[0, 0, 0], w[0, 0] = 1e5, 2.0, 1.0
        got = K.lightning_indexer_fused(q, k, w)
        assert float(got[0, 0, 0]) == float("inf")
    assert K.device_status() == 0


@pytest.mark.gpu
def test_strided_queries_and_one_of_a_dimension():
    """Views that TMA reads (heads innermost but one, batch and rows of one) and one it does not (an expanded batch)."""
    from cinnamon_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()                     # noqa: E731
    for q, k in ((r(2, 4, 150, 64).transpose(1, 2), r(2, 150, 128)[:, :, 64:]), (r(1, 1, 1, 64), r(1, 1, 64)),
                 (r(150, 3, 2, 64).permute(2, 0, 1, 3), r(200, 2, 64).transpose(0, 1)), (r(1, 150, 4, 64).expand(2, -1, -1, -1), r(2, 33, 64))):
        w = torch.rand(q.shape[:3], device="cuda", generator=g).bfloat16()
        want = torch.einsum("bqhd,bkd->bqhk", q.double(), k.double()).clamp_min(0).mul(w.double()[..., None]).sum(2)
        _close_fp16(K.lightning_indexer_fused(q, k, w), want)
