"""The linears and recurrent states of decode steps on both sides of the sizes at which their kernels change how much a thread has
under way, or who writes the output, against float64."""
import pytest
import torch

import nanoquantization_b200 as nq
from nanoquantization_b200 import _lib
from nanoquantization_b200.engine.batch import StepBatch
from nanoquantization_b200.layers import mixers as ops
from nanoquantization_b200.layers.sequence_mixers import RetentionMixer

pytestmark = pytest.mark.gpu
DEV, bf = "cuda", torch.bfloat16


def _step(batch, position):
    return StepBatch.host([[0]] * batch, [position] * batch, [[i] for i in range(batch)], list(range(batch)), 1, 256).to(DEV)


def _close(got, want, limit):
    assert float((got.double() - want).norm()) <= limit * float(want.norm())


# one request holds K or not (512, 1024, 2048), a wave of two or three CTAs per SM or more (296, 444 CTAs of 16 outputs), many weights or few
SIZES = [(1, 512, 40), (1, 520, 40), (8, 1024, 64), (8, 1032, 64), (5, 1032, 4736), (5, 1032, 4752), (3, 1032, 7104), (3, 1032, 7120), (9, 1024, 64), (16, 2048, 8000),
         (16, 2056, 5848), (16, 2056, 5824), (12, 4096, 2928), (16, 5000, 37)]


@pytest.mark.parametrize("M,K,N", SIZES)
@torch.no_grad()
def test_linears(M, K, N):
    """Tolerance: eight warps' chains of K / 128 tensor-core additions and the sum of the eight, each good to 2^-23; one rounding to
    bfloat16 (2^-9 in the 2-norm) where the result has that type."""
    exact = (K / 128 + 8) * 2.0 ** -23
    x, w, beta = torch.randn(M, K, device=DEV).to(bf), (torch.randn(N, K, device=DEV) * K ** -0.5).to(bf), 0.5
    want = x.double() @ w.double().t()
    _close(ops.linear(x, w), want, 2.0 ** -8)
    _close(ops.linear(x, w, torch.float32), want, exact)
    stream = torch.randn(M, N, device=DEV)
    total = beta * stream.double() + want
    _close(ops.linear_residual_(stream, x, w, beta), total, exact)
    # the unit's product has two matrices, minGRU's three: rows of w as they come
    half = N // 2
    gate, up = want[:, :half].clamp(max=0.7), want[:, half:2 * half].clamp(-0.7, 0.7)
    _close(ops.dense_glu(x, w[:2 * half], 0.7), gate * torch.sigmoid(1.702 * gate) * (up + 1), 2.0 ** -8)
    third = N // 3
    zb, xb, state = (torch.randn(n, device=DEV) for n in (third, third, M * third))
    state = state.view(M, third)
    z, u = torch.sigmoid(want[:, :third] + zb.double()), want[:, third:2 * third] + xb.double()
    s = (1 - z) * state.double() + z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
    got = ops.dense_mingru(x, w[:3 * third], zb, xb, state, _step(M, 3))
    _close(state, s, exact)
    _close(got, s * torch.nn.functional.silu(want[:, 2 * third:3 * third]), 2.0 ** -8)


@pytest.mark.parametrize("rot", [0, 64])
@pytest.mark.parametrize("heads,dim,vdim", [(4, 64, 64), (3, 100, 30), (2, 256, 512), (1, 512, 1024), (1, 1024, 8), (2, 600, 24)])
@pytest.mark.parametrize("batch", [1, 7, 40, 160])
@torch.no_grad()
def test_retention_step(batch, heads, dim, vdim, rot):
    """Values that take one thread per column or four, heads over one to eight CTAs, few rows of a state per thread and many, more
    elements of q and k than threads."""
    m = RetentionMixer(heads=heads, dim=dim, vdim=vdim, decay=[0.9 + 0.02 * h for h in range(heads)], eps=1e-6, out_scale=1.3, rot_base=70.0, rot_dims=rot, device=DEV)
    cols = sum(c for _, c in m.in_parts)
    proj = torch.randn(batch, 4 + cols, device=DEV).to(bf)
    act = torch.full((batch, heads * vdim + 8), 7.0, device=DEV).to(bf)
    state = torch.randn(batch, heads, dim, vdim, device=DEV)
    position = 11
    q, k, v, g = (t.double() for t in proj[:, 4:].split([c for _, c in m.in_parts], 1))
    q, k, v, g = q.view(batch, heads, dim), k.view(batch, heads, dim) * dim ** -0.5, v.view(batch, heads, vdim), g.view(batch, heads, vdim)
    a = position * m.inv_freq.double()
    for t in (q, k):
        lo, hi = t[..., :rot // 2].clone(), t[..., rot // 2:rot].clone()
        t[..., :rot // 2], t[..., rot // 2:rot] = lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()
    S = m.decay.double()[:, None, None] * state.double() + k[..., :, None] * v[..., None, :]
    o = torch.einsum("bhd,bhdv->bhv", q, S)
    want = 1.3 * o * torch.rsqrt(o.square().mean(-1, keepdim=True) + 1e-6) * torch.nn.functional.silu(g)
    ops.mixer_decode(proj, act, None, (m.desc(), 4, 8, state), _step(batch, position))
    assert (act[:, :8] == 7).all()
    # a float product and sum (angles of 11 radians are good to 7e-7); one rounding to bfloat16
    _close(state, S, 2e-6)
    _close(act[:, 8:], want.flatten(1), 2.0 ** -8)


@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 16])
@pytest.mark.parametrize("K,N", [(128, 32), (128, 544), (128, 51200), (256, 96256), (256, 102400)])
@pytest.mark.parametrize("dtype,bias", [(torch.float16, True), (torch.bfloat16, False)])
@torch.no_grad()
def test_packed_linears_whose_tiles_are_whole(M, K, N, dtype, bias):
    """A block that has a tile's whole K writes the output itself: tiles of 512 columns, the last ones of 32, 64 and 512; one tile a block
    and several."""
    lib, code = _lib.load(), 0 if dtype == torch.float16 else 1
    assert lib.nqb200_gemm_kernel_name(M, N, K, 128, code) == b"decode_stream"
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    m = nq.WQLinear_GEMM(4, 128, K, N, DEV, bias, dtype)
    words = lambda *s: torch.randint(-2 ** 31, 2 ** 31, s, generator=g, device=DEV, dtype=torch.int64).to(torch.int32)  # noqa: E731
    m.qweight.copy_(words(K, N // 8)); m.qzeros.copy_(words(K // 128, N // 8))
    m.qscales.copy_((torch.rand(K // 128, N, generator=g, device=DEV) * 9e-3 + 1e-3).to(dtype))
    if bias:
        m.bias.copy_(torch.randn(N, generator=g, device=DEV))
    x = torch.randn(M, K, generator=g, device=DEV).to(dtype)
    buf = torch.full((M + 2, N), -7.25, dtype=dtype, device=DEV)      # sentinel rows: a store past the tokens would change them
    m(x, out=buf[1:M + 1])
    torch.cuda.synchronize()
    assert bool((buf[0] == -7.25).all()) and bool((buf[M + 1] == -7.25).all())
    q, z = nq.unpack_int4(m.qweight).double(), nq.unpack_int4(m.qzeros).double()
    W = (q - z.repeat_interleave(128, 0)) * m.qscales.double().repeat_interleave(128, 0)
    ref = x.double() @ W + (m.bias.double() if bias else 0.0)
    # half a unit of the result's last place, and float32 sums of K products of x with q and with the zero-point (and 128 in bfloat16)
    size = x.double().abs() @ ((q + z.repeat_interleave(128, 0) + 256.0) * m.qscales.double().repeat_interleave(128, 0))
    bound = (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) * ref.abs() + K * 2.0 ** -24 * size + 2.0 ** -24
    assert bool(((buf[1:M + 1].double() - ref).abs() <= bound).all())
    _lib.check_workspaces()
