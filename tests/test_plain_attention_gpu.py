"""The plain attention kernels (omc_window_attn, omc_latent_attn) at the widest rows they take, and what lies beyond; the same bits for few rows and for
many, at every width that a kernel is made for."""
import math

import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu
N, PAGE = 45, 16   # keys of the one request: more than the eight warps' first groups of four


def _addresses():
    return (torch.tensor([N - 1], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda(), torch.tensor([[2, 0, 1]], dtype=torch.int32).cuda())


def _check(got, q, keys, values, scale, widest):
    p = torch.softmax(q.double() @ keys.double().T * scale, -1)
    # scores of order one from sums of up to `widest` terms in fp32, a lane adding every 32nd; probabilities move by as much
    err = (widest / 32 + 5) * 2.0 ** -24 * math.sqrt(widest) * scale * 4 + 1e-5
    assert ((got.double().cpu() - p @ values.double()).abs() <= err * (p @ values.double().abs()) + 1e-6).all()


@pytest.mark.parametrize("d,dv", [(11256, 256), (12152, 32), (10230, 256)])
def test_window_attn_takes_the_widest_heads(d, dv):
    gen = torch.Generator().manual_seed(d)
    q, k, v = (torch.randn(n, w, generator=gen) for n, w in ((1, d), (N, d), (N, dv)))
    pool = torch.zeros(3 * PAGE, d + dv)
    pool[:N] = torch.cat([k, v], 1)
    pool = pool.view(3, PAGE, -1)[[1, 2, 0]].contiguous()                  # page i of the request is table[i]
    pos, slot, table = _addresses()
    out = torch.empty(1, dv, device="cuda")

    def run(q, width, pool):
        seqlib.window_attn(q.cuda(), 1, 1, width, dv, pool.cuda(), table, PAGE, pos, slot, seqlib.WINDOW_ALL, d ** -0.5, 0.0, None, out)
    run(q, d, pool)
    _check(out, q, k, v, d ** -0.5, d)
    if d != 10230:                                                         # the widest of its value width: one more is refused, as ever
        with pytest.raises(seqlib.OmcError):
            run(torch.zeros(1, d + 1), d + 1, torch.zeros(3, PAGE, d + 1 + dv))


@pytest.mark.parametrize("r,dr", [(1024, 7160), (32, 12120), (1024, 64)])
def test_latent_attn_takes_the_widest_rows(r, dr):
    gen = torch.Generator().manual_seed(r + dr)
    q, rows = torch.randn(1, 1, r + dr, generator=gen), torch.randn(N, r + dr, generator=gen)
    pool = torch.zeros(3 * PAGE, r + dr)
    pool[:N] = rows
    pool = pool.view(3, PAGE, -1)[[1, 2, 0]].contiguous()
    pos, slot, table = _addresses()
    out = torch.empty(1, 1, r, device="cuda")
    seqlib.latent_attn(q.cuda(), r, dr, pool.cuda(), table, PAGE, pos, slot, None, (r + dr) ** -0.5, out)
    _check(out[0], q[0], rows, rows[:, :r], (r + dr) ** -0.5, r + dr)
    if dr != 64:
        with pytest.raises(seqlib.OmcError):
            seqlib.latent_attn(torch.zeros(1, 1, r + dr + 1, device="cuda"), r, dr + 1, torch.zeros(3, PAGE, r + dr + 1, device="cuda"), table, PAGE, pos, slot,
                               None, 1.0, out)


def _many(T):
    """T rows of one request whose row t sees the keys 0 .. t % N."""
    return torch.arange(T, dtype=torch.int32).remainder(N).cuda(), torch.zeros(T, dtype=torch.int32).cuda(), torch.tensor([[2, 0, 1]], dtype=torch.int32).cuda()


@pytest.mark.parametrize("window,sink", [(seqlib.WINDOW_ALL, False), (7, True)])
@pytest.mark.parametrize("r,dr", [(20, 3), (256, 64), (290, 0), (512, 64), (700, 4)])
def test_latent_attn_few_rows_and_many(r, dr, window, sink):
    gen = torch.Generator().manual_seed(r)
    T, H = 2 * N, 7                                                        # 630 CTAs
    q, rows = torch.randn(T, H, r + dr, generator=gen), torch.randn(N, r + dr, generator=gen)
    pool = torch.zeros(3 * PAGE, r + dr)
    pool[:N] = rows
    pool = pool.view(3, PAGE, -1)[[1, 2, 0]].contiguous().cuda()
    pos, slot, table = _many(T)
    sk = torch.randn(H, generator=gen) if sink else None
    out, one = torch.empty(T, H, r, device="cuda"), torch.empty(1, H, r, device="cuda")
    run = lambda q, pos, slot, out: seqlib.latent_attn(q.cuda(), r, dr, pool, table, PAGE, pos, slot, sk.cuda() if sink else None, (r + dr) ** -0.5, out, window=window)  # noqa: E731
    run(q, pos, slot, out)
    for t in range(T):
        lo, n = max(0, t % N + 1 - window), t % N + 1
        s = q[t].double() @ rows[lo:n].double().T * (r + dr) ** -0.5
        p = torch.softmax(torch.cat([s, sk.double()[:, None]], 1) if sink else s, -1)[:, :n - lo]
        assert ((out[t].double().cpu() - p @ rows[lo:n, :r].double()).abs() <= 1e-5 * (p @ rows[lo:n, :r].double().abs()) + 1e-6).all(), t
        run(q[t:t + 1], pos[t:t + 1], slot[t:t + 1], one)
        assert torch.equal(one[0], out[t]), t


@pytest.mark.parametrize("window,chunk,kept", [(seqlib.WINDOW_ALL, seqlib.WINDOW_ALL, 0), (6, seqlib.WINDOW_ALL, 3), (30, 11, 0)])
@pytest.mark.parametrize("d,dv", [(20, 20), (64, 64), (33, 100), (128, 128), (24, 200)])
def test_window_attn_few_rows_and_many(d, dv, window, chunk, kept):
    gen = torch.Generator().manual_seed(d + dv)
    T, H = 2 * N, 7
    q, k, v = torch.randn(T, H, d, generator=gen), torch.randn(N, d, generator=gen), torch.randn(N, dv, generator=gen)
    pool = torch.zeros(3 * PAGE, d + dv)
    pool[:N] = torch.cat([k, v], 1)
    pool = pool.view(3, PAGE, -1)[[1, 2, 0]].contiguous().cuda()
    pos, slot, table = _many(T)
    out, one = torch.empty(T, H * dv, device="cuda"), torch.empty(1, H * dv, device="cuda")
    run = lambda q, pos, slot, out: seqlib.window_attn(q.reshape(-1, H * d).cuda(), H, 1, d, dv, pool, table, PAGE, pos, slot, window, d ** -0.5, 0.0, None, out,  # noqa: E731
                                                       keep_first=kept, chunk=chunk)
    run(q, pos, slot, out)
    for t in range(T):
        i, j = t % N, torch.arange(t % N + 1)
        see = ((i - j < window) & (j // chunk == i // chunk)) | (j < kept)
        p = torch.softmax((q[t].double() @ k[:i + 1].double().T * d ** -0.5).masked_fill(~see, -math.inf), -1)
        want, mag = p @ v[:i + 1].double(), p @ v[:i + 1].double().abs()
        assert ((out[t].view(H, dv).double().cpu() - want).abs() <= 1e-5 * mag + 1e-6).all(), t
        run(q[t:t + 1], pos[t:t + 1], slot[t:t + 1], one)
        assert torch.equal(one[0], out[t]), t
