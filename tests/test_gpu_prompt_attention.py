"""Attention of prompts on the tcgen05 kernel, against float64: each way it takes a score (no cap, the cap's short and long series,
the fraction, the exponential), with and without a running maximum, at the edges of its tiles and of chunks."""
import math

import pytest
import torch

from nanoquantization_b200 import _lib
from nanoquantization_b200.engine.batch import StepBatch
from nanoquantization_b200.layers import mixers as ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
H, G, BS = 4, 2, 128


@pytest.mark.parametrize("D,V,chunk", [(128, 128, 0), (64, 128, 512), (128, 64, 700)])
@pytest.mark.parametrize("softcap,spread,sink", [
    (50.0, 1.0, None),          # scores a tenth of the cap at most: the short series; the cap bounds them, no running maximum
    (50.0, 4.0, -3.0),          # the series
    (50.0, 20.0, 0.5),          # the fraction
    (20.0, 40.0, 45.0),         # beyond; a sink above every score
    (50.0, 1.0, 100.0),         # a sink so far above that hardly anything is left
    (120.0, 1.0, None),         # a cap too far for a fixed reference
    (120.0, 60.0, 3.0),
    (0.0, 1.0, None),           # no cap
    (0.0, 30.0, 2.0),           # no cap and a maximum that moves
    (400.0, 1.0, None),         # a cap so wide that its series' coefficients are not taken (some would leave the range of float)
])
def test_scores_of_every_range(D, V, chunk, softcap, spread, sink):
    g = torch.Generator(device=DEV).manual_seed(D + V + chunk + int(softcap + spread))
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)  # noqa: E731
    lengths, starts = [1000, 129, 257], [0, 640, 0]
    total = [n + s for n, s in zip(lengths, starts)]
    blocks = [-(-t // BS) for t in total]
    first = [sum(blocks[:i]) + 1 for i in range(3)]
    step = StepBatch.host([[0] * n for n in lengths], starts, [list(range(f, f + b)) for f, b in zip(first, blocks)], [0, 1, 2], max(blocks), BS).to(DEV)
    kc, vc = rnd(sum(blocks) + 1, BS, G, D), rnd(sum(blocks) + 1, BS, G, V)
    q = (rnd(sum(lengths), H * D).float() * spread).to(torch.bfloat16)
    sinks = None if sink is None else torch.full((H,), sink, device=DEV)
    desc = _lib.AttentionDesc(H, G, D, V, chunk, D ** -0.5, softcap, None if sinks is None else sinks.data_ptr(), 1.5)
    out = torch.full((sum(lengths) + 1, H * V), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.chunk_attention(q, kc, vc, out[:-1], desc, step)
    torch.cuda.synchronize()
    assert bool((out[-1] == 7).all())
    row = 0
    for n, start, f, t in zip(lengths, starts, first, total):
        k, v = (c[f:f + -(-t // BS)].reshape(-1, G, c.shape[-1])[:t].double().repeat_interleave(H // G, 1) for c in (kc, vc))
        s = torch.einsum("ihd,jhd->hij", q[row:row + n].reshape(n, H, D).double(), k) * D ** -0.5
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        i, j = torch.arange(start, t, device=DEV)[:, None], torch.arange(t, device=DEV)[None, :]
        s = s.masked_fill((j > i) | ((i // chunk != j // chunk) if chunk else False), -math.inf)
        m = s.amax(-1, keepdim=True)
        m = m if sink is None else m.clamp(min=sink)
        p = (s - m).exp()
        w = 1.5 * p / (p.sum(-1, keepdim=True) + (0.0 if sink is None else (sink - m).exp()))
        ref, size = torch.einsum("hij,jhd->ihd", w, v), torch.einsum("hij,jhd->ihd", w, v.abs())
        got = out[row:row + n].reshape(n, H, V).double()
        # the result and every weight rounded to bf16 (2^-8 of each); a score's error of up to 2e-4 (float arithmetic on scores of up to 2^8, the
        # series where they end)
        bound = 2.0 ** -8 * ref.abs() + (2.0 ** -8 + 2e-4) * size + 1e-37
        assert bool(((got - ref).abs() <= bound).all()), float(((got - ref).abs() / bound).max())
        row += n


@pytest.mark.parametrize("softcap,low", [(0.0, None), (50.0, None), (50.0, -10.0), (50.0, -60.0), (50.0, -150.0), (120.0, None)])
def test_the_sum_takes_unrounded_weights(softcap, low):
    """Every path a score can take.  One key has weight 1 and is the only one with a value; the others weigh half of 1 + 2^-8 + 2^-12, which bf16
    rounds up by nearly 2^-8.  With the exact result at 1 a sum of rounded weights is 2^-8 too large, the next bf16 number below."""
    D, T = 64, 256
    weight = 0.5 * (1 + 2.0 ** -8 + 2.0 ** -12)
    raw = torch.full((T,), math.log(weight), dtype=torch.float64)
    if softcap:
        raw = softcap * torch.atanh(raw / softcap)
    raw[0] = 0.0
    if low is not None:
        raw[[1, 65, 129]] = low           # decides the path of the halves of tiles that the last rows see whole
    k = torch.zeros(T, G, D, dtype=torch.float64)
    for c in range(3):                    # scores exact to 2^-24: three bf16 numbers each
        k[:, :, c] = (raw - k[:, 0].sum(-1)).to(torch.bfloat16).double()[:, None]
    s = k[:, 0].sum(-1)
    s = softcap * torch.tanh(s / softcap) if softcap else s
    p = s.exp()
    kc, vc = torch.zeros(3, BS, G, D, dtype=torch.bfloat16, device=DEV), torch.zeros(3, BS, G, D, dtype=torch.bfloat16, device=DEV)
    kc[1:] = k.to(torch.bfloat16).view(2, BS, G, D).to(DEV)
    vc[1, 0] = 1.0
    step = StepBatch.host([[0] * T], [0], [[1, 2]], [0], 2, BS).to(DEV)
    q = torch.zeros(T, H, D, dtype=torch.bfloat16, device=DEV)
    q[:, :, :3] = 1.0
    out = torch.empty(T, H * D, dtype=torch.bfloat16, device=DEV)
    desc = _lib.AttentionDesc(heads=H, kv_heads=G, dim=D, vdim=D, chunk=0, scale=1.0, softcap=softcap, sink=None, out_scale=float(p.sum()))
    ops.chunk_attention(q.view(T, H * D), kc, vc, out, desc, step)
    assert bool((out[-1].float() == 1.0).all()), out[-1].float().unique()


@pytest.mark.parametrize("chunk", [0, 639])         # 639: the second chunk has a single key in its first tile
@pytest.mark.parametrize("softcap,sink,kind", [
    (50.0, None, "jump"),         # a first tile near minus the cap, later keys near the cap
    (50.0, -45.0, "jump"),
    (50.0, 20.0, "jump"),
    (0.0, None, "jump"),
    (0.0, None, "stairs"),        # every half tile above the one before, for some rows; below, for others
    (120.0, -100.0, "stairs"),
    (50.0, None, "stairs"),
])
def test_references_that_move_far(softcap, sink, kind, chunk):
    """Scores that leave what came before far behind, with values of 2^40: a weight may be large against what is kept of a row, but not so large."""
    D, T = 64, 1000
    g = torch.Generator().manual_seed(chunk + int(softcap) + len(kind))
    key = torch.arange(T) % (chunk or T)
    lead = torch.where(key < 128 if not chunk else key < 1, -150.0, 150.0) if kind == "jump" else -130.0 + 20.0 * (torch.arange(T) // 64)
    k = torch.randn(T, G, D, generator=g)
    k[:, :, 0] = lead[:, None]
    v = torch.randn(T, G, D, generator=g) * 2.0 ** 40
    q = torch.randn(T, H, D, generator=g)
    q[:, :, 0] = 8.0 * (0.5 + torch.rand(T, H, generator=g)) * torch.where(torch.rand(T, H, generator=g) < 0.25, -1.0, 1.0)
    k, v, q = (t.to(torch.bfloat16) for t in (k, v, q))
    nb = -(-T // BS)
    kc, vc = (torch.zeros(nb + 1, BS, G, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    kc[1:].view(-1, G, D)[:T] = k.to(DEV)
    vc[1:].view(-1, G, D)[:T] = v.to(DEV)
    step = StepBatch.host([[0] * T], [0], [list(range(1, nb + 1))], [0], nb, BS).to(DEV)
    sinks = None if sink is None else torch.full((H,), sink, device=DEV)
    desc = _lib.AttentionDesc(heads=H, kv_heads=G, dim=D, vdim=D, chunk=chunk, scale=D ** -0.5, softcap=softcap,
                              sink=None if sinks is None else sinks.data_ptr(), out_scale=1.0)
    out = torch.empty(T, H * D, dtype=torch.bfloat16, device=DEV)
    ops.chunk_attention(q.to(DEV).view(T, H * D), kc, vc, out, desc, step)
    k, v, q = (t.to(DEV).double() for t in (k, v, q))
    s = torch.einsum("ihd,jhd->hij", q, k.repeat_interleave(H // G, 1)) * D ** -0.5
    s = softcap * torch.tanh(s / softcap) if softcap else s
    i, j = torch.arange(T, device=DEV)[:, None], torch.arange(T, device=DEV)[None, :]
    s = s.masked_fill((j > i) | ((i // chunk != j // chunk) if chunk else False), -math.inf)
    m = s.amax(-1, keepdim=True)
    m = m if sink is None else m.clamp(min=sink)
    p = (s - m).exp()
    w = p / (p.sum(-1, keepdim=True) + (0.0 if sink is None else (sink - m).exp()))
    ref, size = (torch.einsum("hij,jhd->ihd", w, t.repeat_interleave(H // G, 1)) for t in (v, v.abs()))
    got = out.view(T, H, D).double()
    # as above; beside a sink far above them all weights may vanish
    bound = 2.0 ** -8 * ref.abs() + (2.0 ** -8 + 2e-4) * size + 2.0 ** 40 * 1e-37
    assert bool(((got - ref).abs() <= bound).all()), float(((got - ref).abs() / bound).nan_to_num(math.inf).max())
