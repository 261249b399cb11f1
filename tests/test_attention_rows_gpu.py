"""fp32 attention over shared key tiles (the route of omc_window_attn and omc_latent_attn for fp32 storage) against float64: key counts at the edges of its
tiles of 32, head groups that fill a CTA and that do not, value widths that leave threads idle, windows, chunks, caps, bias, sinks and gates."""
import math

import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu
PAGE, COUNTS = 7, (1, 2, 31, 32, 33, 63, 64, 65, 97, 128, 150)


def _paged(lens, width, gen):
    """Requests' rows [n, width] each, the pool that holds them in mixed pages, the block table."""
    rows, per = [torch.randn(n, width, generator=gen) for n in lens], max(-(-n // PAGE) for n in lens)
    pages = torch.randperm(len(lens) * per, generator=gen).view(len(lens), per).int()
    pool = torch.full((len(lens) * per, PAGE, width), math.nan)   # what no row sees may hold anything
    for r, pg in zip(rows, pages):
        for j in range(r.shape[0]):
            pool[pg[j // PAGE], j % PAGE] = r[j]
    return rows, pool.cuda(), pages.cuda()


def _err(d, scale):
    # scores from fp32 sums of d terms, d / 16 of them one after the other at most in a lane; probabilities move by as much; sums of 150 products
    return (d / 16 + 8) * 2.0 ** -24 * math.sqrt(d) * scale * 6 + 1e-5


@pytest.mark.parametrize("window,chunk", [(seqlib.WINDOW_ALL, seqlib.WINDOW_ALL), (32, seqlib.WINDOW_ALL), (200, 33)])
@pytest.mark.parametrize("H,G,d,dv,extras", [(8, 1, 64, 64, False), (14, 2, 128, 128, True), (8, 2, 96, 64, False), (9, 1, 96, 256, True), (6, 2, 36, 100, True),
                                             (4, 2, 32, 64, True), (3, 1, 20, 20, False), (20, 1, 64, 80, False)])
def test_window_rows(H, G, d, dv, extras, window, chunk):
    gen = torch.Generator().manual_seed(H * d + dv + min(window, 999))
    rows, pool, table = _paged(COUNTS, G * (d + dv), gen)
    pos, slot = torch.tensor([n - 1 for n in COUNTS], dtype=torch.int32), torch.arange(len(COUNTS), dtype=torch.int32)
    T, scale, cap = len(COUNTS), d ** -0.5, 2.0 if extras else 0.0
    q, gate = torch.randn(T, H * d, generator=gen), torch.randn(T, H * dv, generator=gen)
    bias = torch.randn(min(window, 200), H, generator=gen) if extras and window < 999 else None
    sink = torch.randn(H, generator=gen) if extras else None
    out = torch.empty(T, H * dv, device="cuda")
    kw = dict(sink=sink.cuda(), gate=gate.cuda(), gate_act=1) if extras else {}
    seqlib.window_attn(q.cuda(), H, G, d, dv, pool, table, PAGE, pos.cuda(), slot.cuda(), window, scale, cap, bias.cuda() if bias is not None else None, out, chunk=chunk, **kw)
    for t, n in enumerate(COUNTS):
        p = n - 1
        lo = max(0, p - window + 1, p - p % chunk)
        for h in range(H):
            g = h // (H // G)
            k, v = rows[t][lo:n, g * d:(g + 1) * d].double(), rows[t][lo:n, G * d + g * dv:G * d + (g + 1) * dv].double()
            s = k @ q[t, h * d:(h + 1) * d].double() * scale
            s = cap * torch.tanh(s / cap) if cap else s
            if bias is not None:
                s = s + bias[torch.arange(p - lo, -1, -1), h].double()
            pr = torch.softmax(torch.cat([s, sink[h:h + 1].double()]) if extras else s, 0)[:n - lo]
            z = gate[t, h * dv:(h + 1) * dv].double()
            f = z * torch.sigmoid(z) if extras else torch.ones(dv, dtype=torch.float64)
            got = out[t, h * dv:(h + 1) * dv].double().cpu()
            assert ((got - pr @ v * f).abs() <= _err(d, scale) * (pr @ v.abs()) * f.abs() + 1e-6).all(), (n, h)


@pytest.mark.parametrize("window", [seqlib.WINDOW_ALL, 32])
@pytest.mark.parametrize("H,r,dr", [(8, 256, 64), (16, 512, 64), (11, 500, 12), (4, 64, 32), (2, 128, 0), (5, 132, 8)])
def test_latent_rows(H, r, dr, window):
    gen = torch.Generator().manual_seed(H * r + dr)
    rows, pool, table = _paged(COUNTS, r + dr, gen)
    T, scale = len(COUNTS), (r + dr) ** -0.5
    q, sink, gate = torch.randn(T, H, r + dr, generator=gen), torch.randn(H, generator=gen), torch.randn(T, H, generator=gen)
    out = torch.empty(T, H, r, device="cuda")
    seqlib.latent_attn(q.cuda(), r, dr, pool, table, PAGE, torch.tensor([n - 1 for n in COUNTS], dtype=torch.int32).cuda(),
                       torch.arange(T, dtype=torch.int32).cuda(), sink.cuda(), scale, out, window=window, gate=gate.cuda())
    for t, n in enumerate(COUNTS):
        lo = max(0, n - window)
        k = rows[t][lo:n].double()
        pr = torch.softmax(torch.cat([q[t].double() @ k.T * scale, sink.double()[:, None]], 1), 1)[:, :n - lo]
        f = torch.sigmoid(gate[t].double())[:, None]
        assert ((out[t].double().cpu() - pr @ k[:, :r] * f).abs() <= _err(r + dr, scale) * (pr @ k[:, :r].abs()) * f + 1e-6).all(), n


@pytest.mark.parametrize("window", [63, 64, seqlib.WINDOW_ALL])       # fewer than 64 keys: the plain kernel
def test_one_query_head_per_key_head(window):
    test_window_rows(8, 8, 64, 64, False, window, seqlib.WINDOW_ALL)
    test_window_rows(3, 3, 64, 128, True, window, seqlib.WINDOW_ALL)
    test_latent_rows(1, 128, 64, window)


MANY = (1, 16, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129, 160, 257, 300)


@pytest.mark.parametrize("window,chunk", [(seqlib.WINDOW_ALL, seqlib.WINDOW_ALL), (32, seqlib.WINDOW_ALL), (64, seqlib.WINDOW_ALL), (200, 70)])
@pytest.mark.parametrize("H,G,d,dv,bf16", [(8, 1, 64, 64, False), (14, 2, 128, 128, False), (9, 1, 96, 256, True), (6, 2, 36, 100, False), (4, 2, 32, 64, True), (8, 8, 64, 64, False),
                                           (0, 1, 320, 256, False), (0, 1, 576, 512, False)])
def test_few_rows_and_many_give_the_same_bits(H, G, d, dv, bf16, window, chunk):
    """Two heads to a CTA and several tiles to a stage, or all heads and one tile: by the number of rows. H 0: latents, of d columns in all."""
    gen = torch.Generator().manual_seed(d + dv + min(window, 999))
    latent, H = H == 0, H or 16
    rows, pool, table = _paged(MANY, d if latent else G * (d + dv), gen)
    q, sink, gate = torch.randn(len(MANY), H * d, generator=gen), torch.randn(H, generator=gen).cuda(), torch.randn(len(MANY), H, generator=gen)
    bias = torch.randn(window, H, generator=gen).cuda() if window < 999 else None

    def run(of):
        pos, slot = torch.tensor([MANY[i] - 1 for i in of], dtype=torch.int32).cuda(), torch.tensor(of, dtype=torch.int32).cuda()
        out = torch.empty(len(of), H * dv, device="cuda", dtype=torch.bfloat16 if bf16 else torch.float32)
        if latent:
            seqlib.latent_attn(q[of].cuda().view(len(of), H, d), dv, d - dv, pool, table, PAGE, pos, slot, sink, d ** -0.5, out.view(len(of), H, dv), window=min(window, chunk),
                               gate=gate[of].cuda())
        else:
            seqlib.window_attn(q[of].cuda(), H, G, d, dv, pool, table, PAGE, pos, slot, window, d ** -0.5, 4.0, bias, out, sink=sink, gate=gate[of].cuda(), gate_act=2, chunk=chunk,
                               gate_heads=True)
        return out
    order = list(range(len(MANY)))
    many = run(order * 20)
    assert torch.isfinite(many).all()
    for i in (order[:1], order[4:6], order[-2:], order[8:12]):                # few rows: the CTAs of each of these run in one wave
        assert len(i) * G * -(-H // G // 2) <= 148 < 20 * len(MANY) * G
        assert torch.equal(run(i), many[i[0]:i[-1] + 1])
