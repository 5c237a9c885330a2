"""Attention of a decode step over paged caches, heads of 128: against float64 over the same pages, at the edges of tiles (16
keys), of warps and of clusters, for every way of weighing, grouping and rotating.

Tolerance: queries, the new key and the weights are rounded to 16 bits once each, the result once: four roundings of half a
unit (2^-8 bfloat16, 2^-11 float16) relative to the result's scale, in the 2-norm; scores of a few units turn a query's
rounding into an error of the weight of the same size times the score."""
import pytest
import torch

from nanoquantization_b200.engine.batch import StepBatch

pytestmark = pytest.mark.gpu
DEV, D = "cuda", 128


def _setup(ctx, kv_heads, heads, block_size, dtype, seed=0):
    """Pages in shuffled order, rows of projections; what no sequence has written yet holds large numbers."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    need = [-(-n // block_size) for n in ctx]
    order = torch.randperm(sum(need) + 2, generator=torch.Generator().manual_seed(seed)).tolist()
    blocks = [[order.pop() for _ in range(n)] for n in need]
    kc, vc = (torch.full((sum(need) + 2, block_size, kv_heads, D), 30.0, device=DEV).to(dtype) for _ in range(2))
    for b, n in zip(blocks, ctx):
        for c in (kc, vc):
            flat = c[b].flatten(0, 1)
            flat[:n - 1] = torch.randn(n - 1, kv_heads, D, generator=g, device=DEV).to(dtype)
            c[b] = flat.view(len(b), block_size, kv_heads, D)
    step = StepBatch.host([[0]] * len(ctx), [n - 1 for n in ctx], blocks, list(range(len(ctx))), max(need) + 1, block_size).to(DEV)
    proj = torch.randn(len(ctx), (heads + 2 * kv_heads) * D + 8, generator=g, device=DEV).to(dtype)
    return step, blocks, kc, vc, proj


def _rotate(x, pos, rot, base, neighbours=False):
    f = base ** (-2.0 * torch.arange(rot // 2, device=DEV, dtype=torch.float64) / max(rot, 1))
    a = pos * f
    i, j = (slice(0, rot, 2), slice(1, rot, 2)) if neighbours else (slice(0, rot // 2), slice(rot // 2, rot))
    y = x.clone()
    y[..., i], y[..., j] = x[..., i] * a.cos() - x[..., j] * a.sin(), x[..., j] * a.cos() + x[..., i] * a.sin()
    return y


def _rms(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double()


def _close(got, want, dtype):
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    err = float((got.double() - want).norm() / want.norm())
    assert err <= 4 * eps, err


# edges of tiles and warps; rings that wrap many times with remainders, for each length of ring: four tiles (few CTAs), three (16 of
# about 1900 keys over clusters of two), two (48 of 1100 to 1500, one CTA a sequence and head; 50 of about 600 over clusters of eight)
SHAPES = [((1,), 1, 1, 16), ((2, 16, 17, 64, 65), 2, 8, 16), ((5, 500, 1025), 2, 2, 256), ((129, 3), 3, 48, 24), ((33,) * 70, 8, 32, 256), ((2048,), 8, 16, 256),
          ((4321,), 1, 4, 256), (tuple(1900 - 31 * i for i in range(16)), 8, 16, 256), (tuple(1500 - 8 * i for i in range(48)), 8, 8, 16),
          (tuple(600 - 3 * i for i in range(50)), 1, 2, 32)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("ctx,kv_heads,heads,block_size", SHAPES, ids=str)
@torch.no_grad()
def test_qwen3_step(ctx, kv_heads, heads, block_size, dtype):
    from nanoquantization_b200.layers import fused
    from nanoquantization_b200.models import RotaryCache
    step, blocks, kc, vc, proj = _setup(ctx, kv_heads, heads, block_size, dtype)
    proj = proj[:, :-8].contiguous()
    qw, kw = ((torch.rand(D, device=DEV) + 0.5).to(dtype) for _ in range(2))
    rope = RotaryCache(D, 8192, 1e6).to(DEV)
    before = [kc.clone(), vc.clone(), proj.clone()]
    got = fused.decode_attention(proj, qw, kw, rope.cos_sin_cache, step.positions, heads, kv_heads, D, 1e-6, kc, vc, step)
    # the caches as the launch of its own leaves them
    fused.qknorm_rope_(before[2], qw, kw, rope.cos_sin_cache, step.positions, heads, kv_heads, D, 1e-6, (before[0], before[1], step.rows))
    assert torch.equal(vc, before[1]) and float((kc.float() - before[0].float()).abs().max()) <= 2.0 ** (-6 if dtype == torch.bfloat16 else -9) * 4
    for b, n in enumerate(ctx):
        q = _rotate(_rms(proj[b, :heads * D].double().view(heads, D), qw), n - 1, D, 1e6)
        k, v = (c[blocks[b]].flatten(0, 1)[:n].double().repeat_interleave(heads // kv_heads, 1) for c in (kc, vc))
        w = torch.softmax(torch.einsum("hd,nhd->hn", q, k) * D ** -0.5, -1)
        _close(got[b], torch.einsum("hn,nhd->hd", w, v).flatten(), dtype)


@pytest.mark.parametrize("ctx,kv_heads,heads", [((9000,), 1, 8), ((16384, 5000), 2, 4), ((20000, 0, 8193), 1, 17), ((40000,), 8, 8)], ids=str)
@torch.no_grad()
def test_long_sequences_over_several_clusters(ctx, kv_heads, heads):
    """Sequences whose clusters' shares a second launch adds, long ones beside short and missing ones."""
    from nanoquantization_b200 import _lib
    from nanoquantization_b200.layers import fused
    from nanoquantization_b200.models import RotaryCache
    dtype = torch.bfloat16
    step, blocks, kc, vc, proj = _setup([n or 1 for n in ctx], kv_heads, heads, 256, dtype)
    assert _lib.load().nqb200_decode_attention_scratch_bytes(step.width, 256, len(ctx), heads, kv_heads) > 0
    proj = proj[:, :-8].contiguous()
    w = torch.ones(D, device=DEV, dtype=dtype)
    rope = RotaryCache(D, 1 << 16, 1e6).to(DEV)
    step.ctx.copy_(torch.tensor(ctx))
    got = fused.decode_attention(proj, w, w, rope.cos_sin_cache, step.positions, heads, kv_heads, D, 1e-6, kc, vc, step)
    for b, n in enumerate(ctx):
        if not n:
            assert not got[b].any()
            continue
        q = _rotate(_rms(proj[b, :heads * D].double().view(heads, D), w), n - 1, D, 1e6)
        k, v = (c[blocks[b]].flatten(0, 1)[:n].double().repeat_interleave(heads // kv_heads, 1) for c in (kc, vc))
        _close(got[b], torch.einsum("hn,nhd->hd", torch.softmax(torch.einsum("hd,nhd->hn", q, k) * D ** -0.5, -1), v).flatten(), dtype)


@pytest.mark.parametrize("ctx", [(0,), (0, 17, 0, 300, 0), (0,) * 3 + (5000,)], ids=str)
@torch.no_grad()
def test_rows_without_a_sequence(ctx):
    """A context of 0 (what paged interfaces pad a batch with): zeros, caches untouched, and the other rows as without them."""
    from nanoquantization_b200.layers import fused
    from nanoquantization_b200.models import RotaryCache
    heads, kv_heads, dtype = 8, 2, torch.bfloat16
    live = [i for i, n in enumerate(ctx) if n]
    step, _, kc, vc, proj = _setup([n or 1 for n in ctx], kv_heads, heads, 16, dtype)
    proj = proj[:, :-8].contiguous()
    w = torch.ones(D, device=DEV, dtype=dtype)
    rope = RotaryCache(D, 8192, 1e6).to(DEV)
    for i, n in enumerate(ctx):
        if not n:
            step.ctx[i], step.positions[i], step.rows[i] = 0, -1, -1
            step.table[i] = -1
    before = kc.clone(), vc.clone()
    got = fused.decode_attention(proj, w, w, rope.cos_sin_cache, step.positions, heads, kv_heads, D, 1e-6, kc, vc, step)
    assert not got[[i for i, n in enumerate(ctx) if not n]].any()
    changed = (kc != before[0]).flatten(2).any(-1).flatten().nonzero().flatten()
    assert sorted(changed.tolist()) == sorted(step.rows[live].tolist())
    if live:
        i64 = torch.cat([step.tokens[live], step.positions[live], step.rows[live]])
        i32 = torch.cat([torch.arange(len(live) + 1, device=DEV), step.pos0[live], step.ctx[live], step.slot[live], step.table[live].flatten()]).int()
        alone = StepBatch(i64, i32, [1] * len(live), [ctx[i] - 1 for i in live], step.width, step.block_size)
        kc, vc = before
        want = fused.decode_attention(proj[live].contiguous(), w, w, rope.cos_sin_cache, alone.positions, heads, kv_heads, D, 1e-6, kc, vc, alone)
        _close(got[live], want.double(), dtype)


@pytest.mark.parametrize("kind,chunk,rot", [("capped", 0, 128), ("capped", 40, 64), ("capped", 256, 0), ("sigmoid", 0, 128), ("sigmoid", 0, 64), ("sigmoid", 0, 0)])
@pytest.mark.parametrize("ctx,kv_heads,heads,block_size", SHAPES, ids=str)
@torch.no_grad()
def test_mixers_step(ctx, kv_heads, heads, block_size, chunk, rot, kind):
    from nanoquantization_b200.layers import mixers as ops
    from nanoquantization_b200.layers.sequence_mixers import AttentionMixer, SigmoidAttentionMixer
    dtype = torch.bfloat16
    step, blocks, kc, vc, proj = _setup(ctx, kv_heads, heads, block_size, dtype)
    off = 8
    if kind == "capped":
        m = AttentionMixer(heads=heads, kv_heads=kv_heads, dim=D, vdim=D, chunk=chunk or 1 << 20, rot_base=70.0, rot_dims=rot, scale=0.3, softcap=4.0,
                           out_scale=1.7, device=DEV)
        m.sink.copy_(torch.randn(heads))
    else:
        m = SigmoidAttentionMixer(heads=heads, kv_heads=kv_heads, dim=D, rot_base=70.0, rot_dims=rot, interleaved=True, scale=0.1, eps=1e-6, device=DEV)
        for t, mean in ((m.q_norm, 1.0), (m.k_norm, 1.0), (m.temp, 1.0), (m.bias, -3.0)):
            t.copy_(mean + 0.2 * torch.randn(t.shape))
    act = torch.full((len(ctx), heads * D + 5), 7.0, dtype=dtype, device=DEV)
    ops.mixer_decode(proj, act, (m.desc(), m.rope_desc(), off, m.value_column(off), 2, kc, vc), None, step)
    assert (act[:, :2] == 7).all() and (act[:, -3:] == 7).all()
    for b, n in enumerate(ctx):
        lo = (n - 1) // chunk * chunk if chunk else 0
        q = proj[b, off:off + heads * D].double().view(heads, D)
        if kind == "sigmoid":
            q = _rms(q, m.q_norm)
        q = _rotate(q, n - 1, rot, 70.0, kind == "sigmoid")
        k, v = (c[blocks[b]].flatten(0, 1)[lo:n].double().repeat_interleave(heads // kv_heads, 1) for c in (kc, vc))
        new = proj[b, off + heads * D:off + (heads + kv_heads) * D].double().view(kv_heads, D)
        new = _rotate(_rms(new, m.k_norm) if kind == "sigmoid" else new, n - 1, rot, 70.0, kind == "sigmoid")
        assert float((k[-1, ::heads // kv_heads] - new).abs().max()) <= 2.0 ** -8 * 8
        col = m.value_column(off)
        assert torch.equal(v[-1, ::heads // kv_heads], proj[b, col:col + kv_heads * D].double().view(kv_heads, D))
        s = torch.einsum("hd,nhd->hn", q, k) * m.scale
        if kind == "sigmoid":
            want = torch.einsum("hn,nhd->hd", torch.sigmoid(s * m.temp.double()[:, None] + m.bias.double()[:, None]), v)
        else:
            s = torch.cat([4.0 * torch.tanh(s / 4.0), m.sink.double()[:, None]], 1)
            want = 1.7 * torch.einsum("hn,nhd->hd", torch.softmax(s, -1)[:, :-1], v)
        _close(act[b, 2:-3], want.flatten(), dtype)
