"""omc_window_attn_mma's decode form (one token per request, the keys dealt to eight warps in tiles of 32) against float64."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu
BF16, F64 = torch.bfloat16, torch.float64
PAGE = 64


def _cache(lens, G, d, dv, maps, gen):
    """Rows of every request's keys and values, the pool that holds them on shuffled pages, the block table."""
    need = [-(-n // PAGE) for n in lens]
    order = torch.randperm(sum(need), generator=gen).tolist()
    W = G * (maps * d + dv)
    pool = torch.full((sum(need), PAGE, W), float("nan"), dtype=BF16)      # rows that hold no key must not matter
    table, rows = torch.zeros(len(lens), max(need), dtype=torch.int32), []
    for s, (n, k) in enumerate(zip(lens, need)):
        mine, order = order[:k], order[k:]
        table[s, :k] = torch.tensor(mine, dtype=torch.int32)
        rows.append(torch.randn(n, W, generator=gen).to(BF16))
        for i in range(k):
            part = rows[-1][i * PAGE:(i + 1) * PAGE]
            pool[mine[i], :part.shape[0]] = part
    return rows, pool, table


@pytest.mark.parametrize("bad", ["query", "one_key", "a_warps_keys", "an_infinite_key"])
@pytest.mark.parametrize("sink", [False, True])
def test_numbers_that_are_none_come_through(bad, sink):
    H, G, d, n = 8, 2, 64, 300
    gen = torch.Generator().manual_seed(3)
    rows, pool, table = _cache([n, n], G, d, d, 1, gen)
    q = torch.randn(2, H * d, generator=gen).to(BF16)
    spoil = {"query": [], "one_key": [70], "a_warps_keys": list(range(64, 96)) + list(range(0, 32)), "an_infinite_key": [299]}[bad]
    for j in spoil:                                                        # key/value head 0 of request 1
        pool[table[1, j // PAGE], j % PAGE, :d] = float("nan") if bad != "an_infinite_key" else float("inf")
    if bad == "query":
        q[1, :H // G * d] = float("nan")
    out = torch.empty(2, H * d, device="cuda")
    pos, slot = torch.tensor([n - 1, n - 1], dtype=torch.int32).cuda(), torch.arange(2, dtype=torch.int32).cuda()
    seqlib.window_attn_mma(q.cuda(), H, G, d, d, pool.cuda(), table.cuda(), PAGE, None, pos, slot, seqlib.WINDOW_ALL, d ** -0.5, 0.0, None, out,
                           sink=torch.ones(H, device="cuda") if sink else None)
    got = out.view(2, G, -1).cpu()
    assert torch.isfinite(got[0]).all() and torch.isfinite(got[1, 1]).all()
    assert torch.isnan(got[1, 0]).all()


@pytest.mark.parametrize("H,G,d,dv,maps", [(8, 2, 64, 64, 1), (16, 1, 128, 128, 1), (6, 3, 32, 48, 2), (10, 2, 256, 128, 1)])
@pytest.mark.parametrize("opt", ["plain", "window_bias_sink", "chunk_heads_gate", "kept_cap_gate"])
@pytest.mark.parametrize("copies", [1, 60])    # 60: more CTAs than a wave of eight warps has, four warps each
def test_rows_over_several_tiles_per_warp(H, G, d, dv, maps, opt, copies):
    """Rows that meet 257 to 1100 keys (every warp takes tiles, up to nine each), scores of some tens."""
    lens = [257, 300, 513, 1100, 1, 40]
    gen = torch.Generator().manual_seed(H * d)
    rows, pool, table = _cache(lens, G, d, dv, maps, gen)
    B, rep, scale, window, chunk, kept, cap = len(lens), H // G, 12.0 / d ** 0.5, seqlib.WINDOW_ALL, seqlib.WINDOW_ALL, 0, 0.0
    q = torch.randn(B, H * maps * d, generator=gen).to(BF16)
    bias = sink = gate = None
    act = 0
    if opt == "window_bias_sink":
        window, bias, sink = 400, torch.randn(400, H, generator=gen) * 3, torch.randn(H, generator=gen) * 10
    elif opt == "chunk_heads_gate":
        chunk, gate, act = 384, torch.randn(B, H * maps, generator=gen), 2
    elif opt == "kept_cap_gate":
        window, kept, cap, gate, act = 290, 70, 50.0, torch.randn(B, H * maps * dv, generator=gen), 1
    cu = lambda t: t.cuda() if t is not None else None
    out = torch.empty(copies * B, H * maps * dv, device="cuda")
    pos, slot = torch.tensor([n - 1 for n in lens], dtype=torch.int32).cuda(), torch.arange(B, dtype=torch.int32).cuda()
    again = lambda t: t.repeat(copies, *[1] * (t.dim() - 1)) if t is not None else None
    seqlib.window_attn_mma(again(q.cuda()), H, G, d, dv, pool.cuda(), table.cuda(), PAGE, None, again(pos), again(slot), window, scale, cap, cu(bias), out, maps=maps,
                           keep_first=kept, sink=cu(sink), gate=again(cu(gate)), gate_act=act, chunk=chunk, gate_heads=opt == "chunk_heads_gate")
    assert torch.equal(out.view(copies, -1), out[:B].view(1, -1).expand(copies, -1))
    got = out[:B].view(B, H, maps, dv).double().cpu()
    for b, n in enumerate(lens):
        j = torch.arange(n)
        back = n - 1 - j
        hidden = ((back >= window) | (j // chunk != (n - 1) // chunk)) & (j >= kept)
        for h in range(H):
            for m in range(maps):
                g = h // rep
                keys, vals = rows[b][:, (g * maps + m) * d:(g * maps + m + 1) * d].to(F64), rows[b][:, G * maps * d + g * dv:G * maps * d + (g + 1) * dv].to(F64)
                s = keys @ q[b].view(H, maps, d)[h, m].to(F64) * scale
                if cap:
                    s = cap * torch.tanh(s / cap)
                if bias is not None:
                    s = s + torch.where(back < window, bias.to(F64)[back.clamp(max=window - 1), h], 0.0)
                s = s.masked_fill(hidden, -torch.inf)
                p = torch.softmax(torch.cat([s, sink[h:h + 1].to(F64)]) if sink is not None else s, 0)[:n]
                want, mag = p @ vals, p @ vals.abs()
                if gate is not None:
                    z = gate[b, h * maps + m].to(F64) if opt == "chunk_heads_gate" else gate[b].view(H, maps, dv)[h, m].to(F64)
                    f = torch.sigmoid(z) * (z if act == 1 else 1.0)
                    want, mag = want * f, mag * f.abs()
                # probabilities rounded to bf16 above and below the line (2^-9 each); scores of up to 60 with fp32 sums, a cap within 3e-5: 2^-12
                assert ((got[b, h, m] - want).abs() <= mag * (2.0 ** -8 + 2.0 ** -12) + 1e-30).all(), (b, h, m)
