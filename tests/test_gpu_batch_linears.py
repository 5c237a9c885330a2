"""Linears of 17 to a few hundred tokens (the single-SM tcgen05 kernel) at the edges of its tiles and in each way it deals its
work: against the 16-bit weights in float64."""
import pytest
import torch

import nanoquantization_b200 as nq
from nanoquantization_b200 import _lib
from nanoquantization_b200.layers import fused
from nanoquantization_b200.layers.gemm import _w4a16

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# launches: 1 where every CTA has whole tiles, 2 where tiles are cut
@pytest.mark.parametrize("M,K,N,launches", [
    (17, 128, 32, 1),          # one unit in all
    (17, 128, 288, 1),         # a last tile of 32 columns
    (33, 256, 256, 1),
    (64, 4096, 96, 2),         # many parts of one tile
    (64, 5120, 1024, 2),       # more segments of a tile than one round of the second kernel's loads
    (49, 4096, 24576, 2),      # equal shares of every SM: a CTA ends one tile and begins the next
    (48, 384, 51200, 1),       # two tiles a CTA, two accumulators
    (65, 384, 51200, 1),       # the same with one accumulator
    (112, 1024, 3104, 2),
    (128, 4096, 24576, 1),
    (129, 1024, 3072, 2),      # two token tiles of 80
    (200, 1152, 1056, 2),
    (300, 128, 6144, 1),       # three token tiles, 72 tiles
    (1000, 128, 9600, 1),      # eight token tiles, several a CTA
])
@pytest.mark.parametrize("dtype,bias", [(torch.float16, True), (torch.bfloat16, False)])
def test_dealings_and_edges(M, K, N, launches, dtype, bias):
    lib, code = _lib.load(), 0 if dtype == torch.float16 else 1
    assert lib.nqb200_gemm_kernel_name(M, N, K, 128, code) == b"prefill_tcgen05"
    assert lib.nqb200_gemm_launch_count(M, N, K, 128, code) == launches
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
    m(x, out=buf[1:M + 1])                                            # a second call beside the first one's tail
    torch.cuda.synchronize()
    assert bool((buf[0] == -7.25).all()) and bool((buf[M + 1] == -7.25).all())
    W = nq.awq_dequantize(m.qweight, m.qscales, m.qzeros).double()
    ref = x.double() @ W + (m.bias.double() if bias else 0.0)
    # half a unit of the result's last place, and float32 sums of K products
    bound = (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) * ref.abs() + K * 2.0 ** -23 * (x.double().abs() @ W.abs())
    assert bool(((buf[1:M + 1].double() - ref).abs() <= bound).all())
    _lib.check_workspaces()


def in_one_call(m, x):
    return _w4a16(x, m.qweight, m.qscales, m.qzeros, m.bias, None, silu_mul=True)


@pytest.mark.parametrize("M,K,N", [
    (512, 256, 51200),        # several tiles a cluster: the staging area is handed back and forth
    (2048, 256, 51200),       # the same twenty times over, with little work between
    (2049, 256, 24576),       # a last tile of one token: one SM has tokens to finish, the other none
    (700, 4096, 24576),       # tokens beyond the input within a tile
    (1000, 1024, 19200),      # the columns of one half end inside what the plain call takes as a tile
    (4096, 1024, 6144),
])
@pytest.mark.parametrize("dtype,bias", [(torch.float16, True), (torch.bfloat16, False)])
def test_gate_up_silu_of_prompts_is_the_separate_steps(M, K, N, dtype, bias):
    lib, code = _lib.load(), 0 if dtype == torch.float16 else 1
    assert lib.nqb200_gemm_gate_up_silu_supported(M, N, K, 128, code) == 1
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    m = nq.WQLinear_GEMM(4, 128, K, N, DEV, bias, dtype)
    words = lambda *s: torch.randint(-2 ** 31, 2 ** 31, s, generator=g, device=DEV, dtype=torch.int64).to(torch.int32)  # noqa: E731
    m.qweight.copy_(words(K, N // 8)); m.qzeros.copy_(words(K // 128, N // 8))
    m.qscales.copy_((torch.rand(K // 128, N, generator=g, device=DEV) * 9e-3 + 1e-3).to(dtype))
    if bias:
        m.bias.copy_(torch.randn(N, generator=g, device=DEV))
    x = torch.randn(M, K, generator=g, device=DEV).to(dtype)
    x[0] *= 100.0                                                     # gates at both ends of the sigmoid
    want = fused.silu_mul(m(x))
    for _ in range(2):
        assert torch.equal(in_one_call(m, x), want)                   # every rounding is the same
    assert torch.equal(m.forward_silu_mul(x), want)                   # whichever way it takes
    _lib.check_workspaces()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gate_up_silu_of_every_gate(dtype):
    """Every gate but -0, as the bias of columns whose weights are zero."""
    M, K, N = 512, 256, 131072
    assert _lib.load().nqb200_gemm_gate_up_silu_supported(M, N, K, 128, 0 if dtype == torch.float16 else 1) == 1
    m = nq.WQLinear_GEMM(4, 128, K, N, DEV, True, dtype)
    m.qweight.zero_(); m.qzeros.zero_(); m.qscales.fill_(1.0)
    gates = torch.arange(-2 ** 15, 2 ** 15, device=DEV, dtype=torch.int32).to(torch.int16).view(dtype)
    x = torch.zeros(M, K, device=DEV, dtype=dtype)
    for up in (1.0, -0.7):
        m.bias.copy_(torch.cat([gates, torch.full_like(gates, up)]))
        want = fused.silu_mul(m(x))
        assert torch.equal(in_one_call(m, x).view(torch.int16), want.view(torch.int16))
    _lib.check_workspaces()


@pytest.mark.parametrize("dtype,scale,x_value", [(torch.float16, 2.0 ** -24, 2.0 ** -12), (torch.bfloat16, 2.0 ** -60, 2.0 ** -86)])
def test_gate_up_silu_of_minus_zero(dtype, scale, x_value):
    """Negative sums that vanish when they are rounded: the gate is -0, and so is what comes of it."""
    M, K, N = 512, 256, 51200
    assert _lib.load().nqb200_gemm_gate_up_silu_supported(M, N, K, 128, 0 if dtype == torch.float16 else 1) == 1
    m = nq.WQLinear_GEMM(4, 128, K, N, DEV, False, dtype)
    half = N // 2
    m.qzeros[:, :half // 8] = 0x11111111                               # weights of the gate: 0 - 1
    m.qweight[:, half // 8:] = 0x11111111                              # of the other half: 1 - 0
    m.qscales[:, :half] = scale
    m.qscales[:, half:] = 1.0
    x = torch.full((M, K), x_value, device=DEV, dtype=dtype)
    y = m(x)
    assert bool((y[:, :half].view(torch.int16) == -2 ** 15).all()) and bool((y[:, half:] > 0).all())
    got, want = in_one_call(m, x), fused.silu_mul(y)
    assert bool((want.view(torch.int16) == -2 ** 15).all())
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    _lib.check_workspaces()
