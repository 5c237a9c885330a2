"""Rotary embedding, stream addition and norm + convolution at the sizes where their vector paths begin and end, against
float64."""
import pytest
import torch

from nanoquantization_b200 import _lib
from nanoquantization_b200.engine.batch import StepBatch
from nanoquantization_b200.layers import mixers as ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _step(lens, starts, block_size=16):
    need = [(s + n - 1) // block_size + 1 for n, s in zip(lens, starts)]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(1)).tolist()
    blocks = [[order.pop() for _ in range(n)] for n in need]
    return StepBatch.host([[0] * n for n in lens], starts, blocks, list(range(len(lens))), max(need), block_size).to(DEV), sum(need)


@pytest.mark.parametrize("cached,normed", [(True, True), (True, False), (False, False)])
@pytest.mark.parametrize("neighbours", [False, True])
@pytest.mark.parametrize("dim,rot", [(64, 64), (128, 128), (256, 256), (128, 64), (96, 96)])
@pytest.mark.parametrize("lens,heads,kv_heads", [((1,), 1, 1), ((3, 2), 5, 2), ((595, 30), 3, 1), ((3, 1), 13, 4), ((595, 30), 12, 5), ((593,), 4, 1)], ids=str)
@torch.no_grad()
def test_rotation(lens, heads, kv_heads, dim, rot, neighbours, cached, normed):
    """One token, a few, and enough for four tokens per block with a remainder; whole heads that turn and parts of them."""
    step, nblocks = _step(lens, [7] * len(lens))
    T = sum(lens)
    proj = torch.randn(T, (heads + 2 * kv_heads) * dim + 8, device=DEV).bfloat16()
    want = proj.double()
    inv = (70.0 ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot)).float().to(DEV)
    norms = [1 + 0.2 * torch.randn(dim, device=DEV) for _ in range(2)] if normed else None
    kc, vc = (torch.full((nblocks, 16, kv_heads, dim), 5.0, device=DEV).bfloat16() for _ in range(2)) if cached else (None, None)
    desc = _lib.RopeDesc(heads, kv_heads, dim, dim, rot, int(neighbours), inv.data_ptr(), norms[0].data_ptr() if normed else None,
                         norms[1].data_ptr() if normed else None, 1e-6)
    q_off, k_off, v_off = 8, 8 + heads * dim, 8 + (heads + kv_heads) * dim
    ops.norm_rope(proj, kc, vc, desc, step, q_off, k_off, v_off)
    a = step.positions.double()[:, None, None] * inv.double()

    def turned(off, n, norm):
        x = want[:, off:off + n * dim].view(T, n, dim)
        if normed:
            x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * norm.double()
        i, j = (slice(0, rot, 2), slice(1, rot, 2)) if neighbours else (slice(0, rot // 2), slice(rot // 2, rot))
        y = x.clone()
        y[..., i], y[..., j] = x[..., i] * a.cos() - x[..., j] * a.sin(), x[..., j] * a.cos() + x[..., i] * a.sin()
        return y
    q, k = turned(q_off, heads, norms and norms[0]), turned(k_off, kv_heads, norms and norms[1])

    def close(got, want):   # one rounding to bfloat16; angles of up to 600 in float, 600 * 2^-24 apart
        assert float((got.double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max()) * 1.05
    close(proj[:, q_off:k_off].view(T, heads, dim), q)
    assert torch.equal(proj[:, :q_off].double(), want[:, :q_off]) and torch.equal(proj[:, v_off:].double(), want[:, v_off:])
    if cached:
        close(kc.view(-1, kv_heads, dim)[step.rows], k)
        assert torch.equal(vc.view(-1, kv_heads, dim)[step.rows].double(), want[:, v_off:v_off + kv_heads * dim].view(T, kv_heads, dim))
        assert int((kc == 5.0).flatten(2).all(-1).sum()) >= nblocks * 16 - T
    else:
        close(proj[:, k_off:v_off].view(T, kv_heads, dim), k)


@pytest.mark.parametrize("call", ["rope_store", "norm_rope", "norm_rope neighbours", "mixer_decode"])
@pytest.mark.parametrize("rot", [0, 64])
@torch.no_grad()
def test_dimensions_that_do_not_turn_pass_unchanged(rot, call):
    """Infinities and signed zeros beyond the rotated dimensions reach the cache bit for bit (infinity * 0 is not a number)."""
    T, heads, kv_heads, dim = 3, 4, 2, 128
    step, nblocks = _step([1] * T, [5, 0, 40])
    proj = torch.randn(T, (heads + 2 * kv_heads) * dim, device=DEV).bfloat16()
    k = proj[:, heads * dim:(heads + kv_heads) * dim].view(T, kv_heads, dim)
    k[:, :, rot::3], k[:, 0, rot + 1::3], k[:, 1, rot + 1::3] = float("inf"), float("-inf"), -0.0
    want = k.clone()
    inv = (70.0 ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / max(rot, 1))).float().to(DEV)
    kc, vc = (torch.zeros(nblocks, 16, kv_heads, dim, device=DEV).bfloat16() for _ in range(2))
    offs = (0, heads * dim, (heads + kv_heads) * dim)
    rope = _lib.RopeDesc(heads, kv_heads, dim, dim, rot, int(call.endswith("neighbours")), inv.data_ptr() if rot else None, None, None, 1e-6)
    if call == "rope_store":
        ops.rope_store(proj, kc, vc, inv, step, *offs, heads)
    elif call.startswith("norm_rope"):
        ops.norm_rope(proj, kc, vc, rope, step, *offs)
    else:
        att = _lib.AttentionDesc(heads, kv_heads, dim, dim, 0, 0.1, 0.0, None, 1.0, None, None, 0)
        ops.mixer_decode(proj, torch.empty(T, heads * dim, device=DEV).bfloat16(), (att, rope, 0, offs[2], 0, kc, vc), None, step)
    got = kc.view(-1, kv_heads, dim)[step.rows]
    assert torch.equal(got[..., rot:].view(torch.int16), want[..., rot:].view(torch.int16))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [4, 100, 4096, 5000, 8200, 37])
@torch.no_grad()
def test_stream_add(width, dtype):
    e, ids, v = torch.randn(9, width, device=DEV).to(dtype), torch.tensor([8, 0, 3, 3], device=DEV), torch.randn(width, device=DEV)
    x = torch.full((4, width), float("nan"), device=DEV)
    ops.stream_add(x, ids, e, None, False)
    assert torch.equal(x, e.float()[ids])
    ops.stream_add(x, ids, e, v, True)
    assert torch.equal(x, e.float()[ids] + e.float()[ids] + v)


@pytest.mark.parametrize("width", [4, 1020, 1028, 4096])
@torch.no_grad()
def test_norm_and_convolution_of_prompts(width):
    lens = (33, 17, 2)
    step, _ = _step(lens, [0] * 3)
    x, w, cw = torch.randn(sum(lens), width, device=DEV), 1 + 0.2 * torch.randn(width, device=DEV), torch.randn(4, width, device=DEV)
    state = torch.full((4, 3, width), 9.0, device=DEV)
    got = ops.rmsnorm_conv(x, w, cw, state, step, 1e-6, torch.float32)
    o = 0
    for b, n in enumerate(lens):
        h = x[o:o + n].double()
        h = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * w.double()
        full = torch.cat([torch.zeros(3, width, dtype=torch.float64, device=DEV), h])
        want = h + sum(cw.double()[j] * full[j:j + n] for j in range(4))
        # float sums of a few terms of the size of the largest
        assert float((got[o:o + n].double() - want).abs().max()) <= 1e-5 * float(want.abs().max())
        assert float((state[b].double() - full[-3:]).abs().max()) <= 1e-5 * float(full.abs().max())
        o += n


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps", [2, 3, 4, 5])
@pytest.mark.parametrize("lens,width", [((33, 17, 1), 132), ((16,), 1024), ((4801,), 36), ((4736, 3), 36)], ids=str)
@torch.no_grad()
def test_convolutions_of_prompts_by_taps_and_type(lens, width, taps, dtype):
    """Every number of taps in both types, on both sides of the number of tiles from which more rows are under way."""
    step, _ = _step(lens, [0] * len(lens))
    x, w, cw = torch.randn(sum(lens), width, device=DEV), 1 + 0.2 * torch.randn(width, device=DEV), torch.randn(taps, width, device=DEV)
    state = torch.full((len(lens), taps - 1, width), 9.0, device=DEV)
    got = ops.rmsnorm_conv(x, w, cw, state, step, 1e-6, dtype)
    o = 0
    for b, n in enumerate(lens):
        h = x[o:o + n].double()
        h = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * w.double()
        full = torch.cat([torch.zeros(taps - 1, width, dtype=torch.float64, device=DEV), h])
        want = h + sum(cw.double()[j] * full[j:j + n] for j in range(taps))
        # float sums of a few terms of the size of the largest; one rounding to bfloat16
        limit = 1e-5 if dtype == torch.float32 else 2.0 ** -8
        assert float((got[o:o + n].double() - want).abs().max()) <= limit * float(want.abs().max())
        assert float((state[b].double() - full[len(full) - taps + 1:]).abs().max()) <= 1e-5 * float(full.abs().max())
        o += n


@pytest.mark.parametrize("taps", [2, 4, 5])
@pytest.mark.parametrize("width", [4, 1020, 4096, 4100])
@torch.no_grad()
def test_norm_and_convolution_of_single_tokens(width, taps):
    """Six single tokens per sequence, one of which starts only at the third step."""
    w, cw = 1 + 0.2 * torch.randn(width, device=DEV), torch.randn(taps, width, device=DEV)
    x = torch.randn(6, 2, width, device=DEV)
    state, got = torch.full((3, taps - 1, width), 9.0, device=DEV), []
    for t in range(6):
        step, _ = _step((1, 1) if t >= 2 else (1,), [t, t - 2] if t >= 2 else [t])
        got.append(ops.rmsnorm_conv(x[t, :step.batch].contiguous(), w, cw, state, step, 1e-6, torch.float32))
    for b, first in ((0, 0), (1, 2)):
        h = x[first:, b].double()
        h = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * w.double()
        full = torch.cat([torch.zeros(taps - 1, width, dtype=torch.float64, device=DEV), h])
        want = h + sum(cw.double()[j] * full[j:j + len(h)] for j in range(taps))
        have = torch.stack([got[t][b] for t in range(first, 6)])
        assert float((have.double() - want).abs().max()) <= 1e-5 * float(want.abs().max())
        assert float((state[b].double() - full[len(full) - taps + 1:]).abs().max()) <= 1e-5 * float(full.abs().max())
