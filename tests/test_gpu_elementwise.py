"""The elementwise kernels of a Qwen3 block at the edges of their vector paths, against the reference modules."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ulps(got, want, dtype):
    """Largest difference in units of the 16-bit type at the largest value: a rounding may fall to either side where the
    sums behind it were added in another order, and the second rounding doubles that."""
    eps = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
    return float((got.float() - want.float()).abs().max()) / (eps * max(1.0, float(want.float().abs().max())))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,H", [(1, 8), (3, 264), (2, 1000), (5, 1024), (2, 4096), (3, 4104), (2, 8200), (2, 12288), (2, 100), (2, 4097)])
@torch.no_grad()
def test_add_rmsnorm(T, H, dtype):
    from nanoquantization_b200.layers import fused
    from nanoquantization_b200.models import RMSNorm
    g = torch.Generator(device=DEV).manual_seed(H)
    x, r = (torch.randn(T, H, generator=g, device=DEV).to(dtype) for _ in range(2))
    norm = RMSNorm(H, 1e-6).to(DEV)
    norm.weight.data = (torch.rand(H, generator=g, device=DEV) + 0.5).to(dtype)
    out, res = fused.add_rmsnorm(x, r.clone(), norm.weight, 1e-6)
    assert torch.equal(res, x + r) and _ulps(out, norm(x + r), dtype) <= 2
    out, res = fused.add_rmsnorm(x, None, norm.weight, 1e-6)
    assert res is x and _ulps(out, norm(x), dtype) <= 2


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,width", [(1, 8), (3, 100), (2, 4096), (2, 4104), (70000, 8),
                                     (3, 6), (3, 7), (20, 16004), (600, 4004), (600, 4010), (801, 15000), (1501, 8008)])
@torch.no_grad()
def test_silu_mul(T, width, dtype):
    from nanoquantization_b200.layers import fused
    g = torch.Generator(device=DEV).manual_seed(width)
    gu = (3 * torch.randn(T, 2 * width, generator=g, device=DEV)).to(dtype)
    gu.view(-1)[:4] = torch.tensor([-100.0, 100.0, -20.0, 0.0], device=DEV)
    assert _ulps(fused.silu_mul(gu), torch.nn.functional.silu(gu[:, :width]) * gu[:, width:], dtype) <= 2


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,heads,kv_heads,offset", [(1, 4, 1, 0), (3, 5, 2, 0), (3, 5, 2, 1), (17, 32, 8, 0), (17, 32, 8, 2), (40, 7, 1, 0),
                                                        (1366, 1, 1, 0), (1365, 1, 1, 0), (460, 5, 2, 0), (460, 5, 2, 1)])
@torch.no_grad()
def test_qknorm_rope(T, heads, kv_heads, offset, dtype):
    """Odd numbers of heads (half of a warp idle), weights that start off the 8-byte boundaries, and both sides of the 4096 heads
    from which two heads share a warp."""
    from nanoquantization_b200.layers import fused
    from nanoquantization_b200.models import RMSNorm, RotaryCache
    g = torch.Generator(device=DEV).manual_seed(heads)
    D = 128
    qkv = torch.randn(T, (heads + 2 * kv_heads) * D, generator=g, device=DEV).to(dtype)
    w = (torch.rand(2, D + 8, generator=g, device=DEV) + 0.5).to(dtype)
    qn, kn = RMSNorm(D, 1e-6).to(DEV), RMSNorm(D, 1e-6).to(DEV)
    qn.weight.data, kn.weight.data = w[0, offset:offset + D], w[1, offset:offset + D]
    rope = RotaryCache(D, 4096, 1e6).to(DEV)
    pos = torch.randint(0, 4096, (T,), generator=g, device=DEV)
    q, k, v = qkv.split([heads * D, kv_heads * D, kv_heads * D], dim=1)
    want_q, want_k = rope(qn(q.reshape(T, heads, D)), kn(k.reshape(T, kv_heads, D)), pos)
    want_v = v.clone()
    slots = torch.randperm(max(64, T), generator=g, device=DEV)[:T]
    kc, vc = (torch.full((max(64, T), kv_heads, D), 7.0, dtype=dtype, device=DEV) for _ in range(2))
    fused.qknorm_rope_(qkv, qn.weight, kn.weight, rope.cos_sin_cache, pos, heads, kv_heads, D, 1e-6, (kc, vc, slots))
    got_k = qkv[:, heads * D:(heads + kv_heads) * D].reshape(T, kv_heads, D)
    assert _ulps(qkv[:, :heads * D].reshape(T, heads, D), want_q, dtype) <= 2 and _ulps(got_k, want_k, dtype) <= 2
    assert torch.equal(kc[slots], got_k) and torch.equal(vc[slots], want_v.reshape(T, kv_heads, D))
    assert int((kc == 7.0).all(-1).all(-1).sum()) >= max(64, T) - T
