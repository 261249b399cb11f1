"""The fp32 linear layer (omc_linear): the rows kernel, the tile kernel and every staging path against float64, and one order of sums in all."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xdt,wdt", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("N,K", [(65, 4), (130, 63), (72, 68), (1000, 1028), (515, 1091), (2048, 2112)])
def test_rows_do_not_depend_on_the_kernel_that_takes_them(N, K, xdt, wdt):
    gen = torch.Generator().manual_seed(N * 7 + K)
    M = 1 + 1480 * 148 // N + 70                       # above the line between the kernels (the first columns of a wide matrix stay below)
    x, w = torch.randn(M, K + 3, generator=gen), torch.randn(N, K, generator=gen)
    x, w = x.to(xdt).cuda()[:, :K], w.to(wdt).cuda()   # rows K + 3 apart: the vector loads take only some of these
    if K % 4 == 0 and K > 4:
        x = x.contiguous()
    y = torch.empty(M, N, device="cuda")
    seqlib.linear(x, w, y)
    ref = x.double() @ w.double().T
    if xdt == torch.bfloat16 and x.stride(0) % 8 == 0 and K % 8 == 0:
        return                                         # the tensor-core kernel's
    # 32 terms in a row, their pair, then the chunks: (34 + K / 64) roundings of at most the sum of magnitudes
    bound = (x.double().abs() @ w.double().abs().T) * (34 + K // 64) * 2.0 ** -24 + 1e-30
    assert ((y.double() - ref).abs() <= bound).all()
    for rows in (1, 3, 8, 17, 33):
        if rows * N <= 1480 * 148:
            part = torch.empty(rows, N, device="cuda")
            seqlib.linear(x[5:5 + rows], w, part)
            assert torch.equal(part, y[5:5 + rows]), rows
