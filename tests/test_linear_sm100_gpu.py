"""omc_linear's tensor-core kernel against float64: tails of every dimension and tile width, heads as column slices, an operand the batch shares,
gates and outputs off the 16-byte grid, and rows that do not depend on how many others there are."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("M", [1, 127, 129, 1300])
@pytest.mark.parametrize("N,K,batch", [(72, 64, 1), (200, 72, 3), (512, 128, 16), (136, 520, 5), (64, 1032, 2)])
@pytest.mark.parametrize("ydt,gate,odd", [(BF16, None, 0), (F32, F32, 0), (BF16, BF16, 0), (BF16, F32, 1), (F32, BF16, 1)])
def test_batched_column_slices(M, N, K, batch, ydt, gate, odd):
    gen = torch.Generator().manual_seed(M + N * K)
    x = torch.randn(M, batch * (K + 8), generator=gen).to(BF16).cuda()          # item b: columns b (K + 8) ..
    w = torch.randn(batch, N, K, generator=gen).to(BF16).cuda()
    y = torch.full((M, batch * (N + odd) + odd), 7.0, dtype=ydt, device="cuda")  # odd: outputs and gates on no 16-byte boundary
    g = torch.randn(M, batch * N + odd, generator=gen).to(gate).cuda()[:, odd:] if gate is not None else None
    seqlib.linear(x, w, y[:, odd:], M=M, N=N, K=K, ldx=x.stride(0), sx=K + 8, ldw=K, sw=N * K, ldy=y.stride(0), sy=N + odd, batch=batch, alpha=0.5,
                  gate=g)
    xs = x.view(M, batch, K + 8)[:, :, :K].double()
    want, mag = torch.einsum("mbk,bnk->mbn", xs, w.double()) * 0.5, torch.einsum("mbk,bnk->mbn", xs.abs(), w.double().abs()) * 0.5
    if g is not None:
        want, mag = want * torch.sigmoid(g.double()).view(M, batch, N), mag * torch.sigmoid(g.double()).view(M, batch, N)
    got = y[:, odd:].reshape(M, batch, N + odd)[:, :, :N].double()
    # products of bf16 are exact; K additions in fp32 (not all rounded to nearest), a fast exponential in the gate, the output's rounding
    bound = mag * (K * 2.0 ** -23 + 2.0 ** -20) + want.abs() * (2.0 ** -8 if ydt == BF16 else 0.0) + 1e-30
    assert ((got - want).abs() <= bound).all()
    if odd:
        assert (y[:, 0] == 7.0).all() and (y[:, odd:].reshape(M, batch, N + odd)[:, :, N:] == 7.0).all()
    if M > 129:      # few rows take narrower tiles
        part = torch.empty(3, batch * N, dtype=ydt, device="cuda")
        seqlib.linear(x[5:8], w, part, M=3, N=N, K=K, ldx=x.stride(0), sx=K + 8, ldw=K, sw=N * K, ldy=batch * N, sy=N, batch=batch, alpha=0.5,
                      gate=g[5:8] if g is not None else None)
        assert torch.equal(part.view(3, batch, N), y[5:8, odd:].reshape(3, batch, N + odd)[:, :, :N])


def test_a_batch_may_share_an_operand():
    gen = torch.Generator().manual_seed(1)
    x, w = torch.randn(40, 96, generator=gen).to(BF16).cuda(), torch.randn(4, 80, 96, generator=gen).to(BF16).cuda()
    y = torch.empty(40, 4 * 80, device="cuda")
    seqlib.linear(x, w, y, M=40, N=80, K=96, sx=0, ldw=96, sw=80 * 96, ldy=320, sy=80, batch=4)
    assert torch.allclose(y.double(), torch.einsum("mk,bnk->mbn", x.double(), w.double()).reshape(40, 320), atol=1e-4)
    seqlib.linear(w.view(4, 80, 96)[0], x, z := torch.empty(80, 40, device="cuda"))
    assert torch.allclose(z.double(), w[0].double() @ x.double().T, atol=1e-4)


@pytest.mark.parametrize("N,pad,gate", [(72, 3, F32), (72, 1, BF16), (73, 7, F32)])   # odd strides of rows; of batch items
def test_gates_that_do_not_come_in_pairs_use_the_precise_exponential(N, pad, gate):
    M, K = 150, 64
    g = torch.linspace(-34, -10, M * N).view(M, N)
    buf = torch.zeros(M, N + pad)
    buf[:, :N] = g
    g = buf.to(gate).cuda()[:, :N]
    x, w, y = torch.ones(M, K, dtype=BF16, device="cuda"), torch.ones(N, K, dtype=BF16, device="cuda"), torch.empty(M, N, device="cuda")
    seqlib.linear(x, w, y, gate=g)
    err = (y.double() / (K * torch.sigmoid(g.double())) - 1).abs()
    # the product is exact; two units of the last place for the exponential, half of one for the sum, the quotient and their effect on it
    assert err.max() <= 4 * 2.0 ** -23, float(err.max())


@pytest.mark.parametrize("N,K,batch,M", [(512, 64, 8, 3100), (128, 192, 8, 12900), (64, 64, 6, 25700)])   # six and eight tiles of 256, 128 and 64 columns per CTA
@pytest.mark.parametrize("gated", [False, True])
def test_a_cta_walks_over_many_tiles(N, K, batch, M, gated):
    gen = torch.Generator(device="cuda").manual_seed(N)
    x, w = (torch.randn(*s, generator=gen, device="cuda").to(BF16) for s in ((M, batch * K), (batch, N, K)))
    g = torch.randn(M, batch * N, generator=gen, device="cuda").to(BF16) if gated else None
    if gated:      # gates of no finite value: shut, open, undefined
        g[0, :3] = torch.tensor([-torch.inf, torch.inf, torch.nan], device="cuda")
        g[-1, -3:] = torch.tensor([-torch.inf, torch.inf, torch.nan], device="cuda")
    y = torch.empty(M, batch * N, dtype=BF16, device="cuda")
    seqlib.linear(x, w, y, M=M, N=N, K=K, ldx=batch * K, sx=K, ldw=K, sw=N * K, ldy=batch * N, sy=N, batch=batch, gate=g)
    for b in range(batch):
        cols = slice(b * N, (b + 1) * N)
        xs, ws = x[:, b * K:(b + 1) * K].double(), w[b].double()
        want, mag = xs @ ws.T, xs.abs() @ ws.abs().T
        if gated:
            want, mag = want * torch.sigmoid(g[:, cols].double()), mag * torch.sigmoid(g[:, cols].double())
        bound = mag * (K * 2.0 ** -23 + 2.0 ** -20) + want.abs() * 2.0 ** -8 + 1e-30   # as above
        ok = (y[:, cols].double() - want).abs() <= bound
        assert (ok | (want.isnan() & y[:, cols].isnan())).all(), b


@pytest.mark.parametrize("M,batch", [(131200, 64), (130900, 64), (40, 65535)])    # 65600 tiles, 65472 (the last that are placed by a multiplication), a tile per problem
def test_many_tiles_find_their_places(M, batch):
    gen = torch.Generator(device="cuda").manual_seed(M)
    N, K = 72, 64
    x, w = (torch.randn(*s, generator=gen, device="cuda").to(BF16) for s in ((M, K), (batch, N, K)))
    y = torch.full((M, batch * N), 7.0, dtype=BF16, device="cuda")
    seqlib.linear(x, w, y, M=M, N=N, K=K, ldx=K, sx=0, ldw=K, sw=N * K, ldy=batch * N, sy=N, batch=batch)
    rows = torch.cat([torch.arange(0, M, max(1, M // 40), device="cuda"), torch.tensor([M - 1], device="cuda")])
    want = torch.einsum("mk,bnk->mbn", x[rows].double(), w.double())
    bound = torch.einsum("mk,bnk->mbn", x[rows].double().abs(), w.double().abs()) * (K * 2.0 ** -23) + want.abs() * 2.0 ** -8
    assert ((y[rows].view(-1, batch, N).double() - want).abs() <= bound).all()
    assert not (y[:, ::61] == 7.0).all(1).any()
