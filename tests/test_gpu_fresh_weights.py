"""Linears right behind what writes their weights: a kernel that lets its successors start early (as the library's own do), and torch."""
import pytest
import torch

import nanoquantization_b200 as nq
from nanoquantization_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,kernel", [(17, b"prefill_tcgen05"), (48, b"prefill_tcgen05"), (128, b"prefill_tcgen05"), (1000, b"prefill_tcgen05_pair")])
@pytest.mark.parametrize("writer", ["kernel", "torch"])
def test_weights_written_directly_ahead_are_the_ones_that_count(M, kernel, writer):
    K, N = 4096, 8192
    assert _lib.load().nqb200_gemm_kernel_name(M, N, K, 128, 0) == kernel
    g = torch.Generator(device=DEV).manual_seed(M)
    m = nq.WQLinear_GEMM(4, 128, K, N, DEV, False, torch.float16)
    m.qscales.fill_(2.0 ** -7)
    x = torch.randn(M, K, generator=g, device=DEV).half()
    rows, cols = K, N // 4                                             # the packed matrix as 16-bit numbers
    sources = [torch.randn(rows, 2 * cols, generator=g, device=DEV).half() for _ in range(3)]
    words = m.qweight.view(torch.float16).view(rows, cols)

    def write(i):
        if writer == "kernel":
            _lib.check(_lib.load().nqb200_silu_mul(sources[i].data_ptr(), words.data_ptr(), rows, cols, 0, _lib.stream_ptr()))
        else:
            words.copy_(sources[i][:, :cols])
    want = []
    for i in range(3):
        write(i)
        torch.cuda.synchronize()
        want.append(m(x).clone())
        torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    got = [torch.empty(M, N, dtype=torch.float16, device=DEV) for _ in range(30)]
    for k in range(30):
        write(k % 3)
        m(x, out=got[k])
    torch.cuda.synchronize()
    for k in range(30):
        assert torch.equal(got[k], want[k % 3]), k
    _lib.check_workspaces()
