"""The fp32 linear layer (omc_linear): the rows kernel, the tile kernel and every staging path against float64, and one order of sums in all."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu


def _operands(M, N, K, xdt, wdt, gen):
    """Rows of x that the vector loads take (K + 4 apart: for bf16 on no 16-byte boundary, which the tensor-core kernel would ask for) where K is a
    multiple of four, rows that they do not take otherwise."""
    x, w = torch.randn(M, K + (4 if K % 4 == 0 and K > 4 else 3), generator=gen), torch.randn(N, K, generator=gen)
    x, w = x.to(xdt).cuda()[:, :K], w.to(wdt).cuda()
    assert xdt == torch.float32 or K % 8 or x.stride(0) % 8
    return x, w


def _check(x, w, y):
    K = x.shape[1]
    # 32 terms in a row, their pair, then the chunks: (34 + K / 64) roundings of at most the sum of magnitudes
    bound = (x.double().abs() @ w.double().abs().T) * (34 + K // 64) * 2.0 ** -24 + 1e-30
    assert ((y.double() - x.double() @ w.double().T).abs() <= bound).all()


@pytest.mark.parametrize("xdt,wdt", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("N,K", [(65, 4), (130, 63), (72, 68), (1000, 1028), (515, 1091), (2048, 2112)])
def test_rows_do_not_depend_on_the_kernel_that_takes_them(N, K, xdt, wdt):
    gen = torch.Generator().manual_seed(N * 7 + K)
    M = 1 + 1480 * 148 // N + 70                       # above the line between the kernels (the first columns of a wide matrix stay below)
    x, w = _operands(M, N, K, xdt, wdt, gen)
    y = torch.empty(M, N, device="cuda")
    seqlib.linear(x, w, y)
    _check(x, w, y)
    for rows in (1, 3, 8, 17, 33):
        if rows * N <= 1480 * 148:
            part = torch.empty(rows, N, device="cuda")
            seqlib.linear(x[5:5 + rows], w, part)
            assert torch.equal(part, y[5:5 + rows]), rows


@pytest.mark.parametrize("xdt,wdt", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("K", [196, 203, 900, 901])
def test_many_tiles(K, xdt, wdt):
    """336 tiles: 4 x 8 outputs per thread for long sums in fp32, 4 x 4 otherwise. The same bits as in calls of fewer rows."""
    M, N = 1300, 1000
    x, w = _operands(M, N, K, xdt, wdt, torch.Generator().manual_seed(K))
    y = torch.empty(M, N, device="cuda")
    seqlib.linear(x, w, y)
    _check(x, w, y)
    for first, rows in ((3, 5), (700, 400)):           # the rows kernel; tiles of 256 threads
        part = torch.empty(rows, N, device="cuda")
        seqlib.linear(x[first:first + rows], w, part)
        assert torch.equal(part, y[first:first + rows]), rows


@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [68, 131, 801])
@pytest.mark.parametrize("tiles", [4, 33])             # 40 tiles, 330
def test_grouped_rows(tiles, K, wdt):
    """Row tiles of 64 that each name the matrix they meet; -1: rows that nobody asks for stay as they were."""
    N, G = 600, 5
    gen = torch.Generator().manual_seed(tiles)
    x, w = torch.randn(64 * tiles, K, generator=gen).cuda(), torch.randn(G, N, K, generator=gen).to(wdt).cuda()
    group = (torch.arange(tiles) * 3 % (G + 1) - 1).to(torch.int32)
    y = torch.full((64 * tiles, N), 5.0, device="cuda")
    seqlib.linear(x, w[0], y, tile_group=group.cuda(), group_stride=N * K)
    for t, g in enumerate(group.tolist()):
        rows = slice(64 * t, 64 * t + 64)
        if g < 0:
            assert (y[rows] == 5.0).all()
        else:
            _check(x[rows], w[g], y[rows])


@pytest.mark.parametrize("N,K", [(2048, 64), (2048, 63), (700, 16), (1024, 256), (1000, 250)])
def test_short_sums_on_both_sides_of_the_line(N, K):
    """Where the rows kernel gives way to tiles depends on K and on what its loads can take: the same bits from 1 row to 120."""
    x, w = _operands(120, N, K, torch.float32, torch.float32, torch.Generator().manual_seed(N))
    y = torch.empty(120, N, device="cuda")
    seqlib.linear(x, w, y)
    _check(x, w, y)
    for rows in (1, 2, 4, 8, 12, 16, 24, 48, 70, 100):
        part = torch.empty(rows, N, device="cuda")
        seqlib.linear(x[:rows], w, part)
        assert torch.equal(part, y[:rows]), rows
