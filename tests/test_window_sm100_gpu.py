"""omc_window_attn_mma's prompt portions on tcgen05 (two items of the work list per CTA) and what stays with the mma.sync kernel, against float64."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu
BF16, F64 = torch.bfloat16, torch.float64


def _cache(lens, W, page, gen):
    """Rows of every request, the pool that holds them on shuffled pages (NaN where no key is), the block table."""
    need = [-(-n // page) for n in lens]
    order = torch.randperm(sum(need), generator=gen).tolist()
    pool = torch.full((sum(need), page, W), float("nan"), dtype=BF16)
    table, rows = torch.zeros(len(lens), max(need), dtype=torch.int32), []
    for s, (n, k) in enumerate(zip(lens, need)):
        mine, order = order[:k], order[k:]
        table[s, :k] = torch.tensor(mine, dtype=torch.int32)
        rows.append(torch.randn(n, W, generator=gen).to(BF16))
        for i in range(k):
            part = rows[-1][i * page:(i + 1) * page]
            pool[mine[i], :part.shape[0]] = part
    return rows, pool, table


def _inputs(portions, H, G, d, page, gen):
    lens = [p0 + n for n, p0 in portions]
    rows, pool, table = _cache(lens, 2 * G * d, page, gen)
    T = sum(n for n, _ in portions)
    q = torch.randn(T, H * d, generator=gen).to(BF16)
    at, plan = 0, []
    for s, (n, p0) in enumerate(portions):
        plan.append((at, n, s, p0))
        at += n
    return rows, pool, table, q, plan


def _oracle(rows, q, plan, H, G, d, window, chunk, scale, cap, bias, sink, gate, act, per_head):
    """Outputs and the same sums over the values' magnitudes, in 64 bits on the GPU."""
    T, rep = q.shape[0], H // G
    want, mag = torch.empty(T, H, d, dtype=F64, device="cuda"), torch.empty(T, H, d, dtype=F64, device="cuda")
    for first, n, s, p0 in plan:
        kv = rows[s].cuda().to(F64)
        keys, vals = (kv[:, m * G * d:(m + 1) * G * d].view(-1, G, d).transpose(0, 1).repeat_interleave(rep, 0) for m in (0, 1))
        sc = q[first:first + n].cuda().to(F64).view(n, H, d).transpose(0, 1) @ keys.transpose(1, 2) * scale
        if cap:
            sc = cap * torch.tanh(sc / cap)
        i, j = p0 + torch.arange(n, device="cuda")[:, None], torch.arange(p0 + n, device="cuda")[None]
        if bias is not None:
            sc = sc + bias.cuda().to(F64)[(i - j).clamp(0, window - 1)].permute(2, 0, 1)
        sc = sc.masked_fill((j > i) | (i - j >= window) | (i // chunk != j // chunk), -torch.inf)
        if sink is not None:
            sc = torch.cat([sc, sink.cuda().to(F64)[:, None, None].expand(-1, n, 1)], -1)
        p = torch.softmax(sc, -1)[..., :p0 + n]
        want[first:first + n], mag[first:first + n] = (p @ vals).transpose(0, 1), (p @ vals.abs()).transpose(0, 1)
    if gate is not None:
        z = gate.cuda().to(F64).view(T, H, -1) if not per_head else gate.cuda().to(F64)[:, :, None]
        f = torch.sigmoid(z) * (z if act == 1 else 1.0)
        want, mag = want * f, mag * f.abs()
    return want.reshape(T, -1), mag.reshape(T, -1)


PORTIONS = {
    "one_row": [(1, 0)],
    "edges": [(64, 0), (65, 63), (1, 64), (63, 1), (127, 129)],          # ends of key tiles, of items and of pairs of items
    "later": [(200, 331), (33, 700), (128, 512)],                        # portions behind cached keys, starts that items do not divide
    "many": [(n, (37 * n) % 90) for n in (5, 16, 17, 31, 32, 47, 48, 96)],
}


@pytest.mark.parametrize("portions", list(PORTIONS))
@pytest.mark.parametrize("H,G,d,page", [(2, 2, 64, 64), (8, 2, 128, 64), (6, 2, 64, 128), (8, 4, 128, 64), (16, 1, 64, 64), (64, 1, 128, 64)])
@pytest.mark.parametrize("opt", ["causal", "window_cap_bias", "window_bias_sink", "chunk_cap_sink_heads_gate", "short_chunk_gate"])
def test_against_float64(portions, H, G, d, page, opt):
    gen = torch.Generator().manual_seed(H * d + len(opt))
    rows, pool, table, q, plan = _inputs(PORTIONS[portions], H, G, d, page, gen)
    T, scale, window, chunk, cap, bias, sink, gate, act = q.shape[0], 8.0 / d ** 0.5, seqlib.WINDOW_ALL, seqlib.WINDOW_ALL, 0.0, None, None, None, 0
    if opt == "window_cap_bias":
        window, cap = 200, 50.0
        bias = torch.randn(window, H, generator=gen) * 3
    elif opt == "window_bias_sink":
        window = 64 if d == 128 else 192                                 # the least this kernel takes
        bias, sink = torch.randn(window, H, generator=gen) * 3, torch.randn(H, generator=gen) * 10
    elif opt == "chunk_cap_sink_heads_gate":
        chunk, cap, sink, gate, act = 96 if d == 128 else 200, 30.0, torch.randn(H, generator=gen) * 10, torch.randn(T, H, generator=gen), 2
    elif opt == "short_chunk_gate":
        chunk, gate, act = 24, torch.randn(T, H * d, generator=gen), 1
    cu = lambda t: t.cuda() if t is not None else None
    items = seqlib.window_attn_items(plan, H // G, "cuda", chunk)
    want, mag = _oracle(rows, q, plan, H, G, d, window, chunk, scale, cap, bias, sink, gate, act, opt == "chunk_cap_sink_heads_gate")
    for dt in (torch.float32, BF16):
        out = torch.full((T, H * d), float("nan"), device="cuda", dtype=dt)
        seqlib.window_attn_mma(q.cuda(), H, G, d, d, pool.cuda(), table.cuda(), page, items, None, None, window, scale, cap, cu(bias), out, sink=cu(sink), gate=cu(gate),
                               gate_act=act, chunk=chunk, gate_heads=opt == "chunk_cap_sink_heads_gate")
        # fp32 scores of up to some tens (in base 2: 2^7) after some eight roundings and a soft cap of a few 2^-23 of the cap: 2^-14; probabilities as
        # two bf16 numbers: 2^-17 (chunks too short for this kernel, on mma.sync: one, in the sums above and below the line, 2^-8); the gate through the
        # fast exponential: 2^-20. A bf16 output adds its own rounding
        err = (out.double() - want).abs()
        assert (err <= mag * (2.0 ** -13 + (2.0 ** -8 if opt == "short_chunk_gate" else 0.0)) + (want.abs() * 2.0 ** -8 if dt == BF16 else 0.0) + 1e-30).all(), (dt, float((err / (mag + 1e-30)).max()))


def test_requests_do_not_meet():
    """A request whose keys and values are NaN and infinite spoils no row of its neighbours in the step, whose items lie beside its own in the list."""
    H, G, d = 8, 2, 128
    gen = torch.Generator().manual_seed(5)
    portions = [(24, 0), (24, 40), (24, 8)]
    rows, pool, table, q, plan = _inputs(portions, H, G, d, 64, gen)
    want, _ = _oracle(rows, q, plan, H, G, d, seqlib.WINDOW_ALL, seqlib.WINDOW_ALL, d ** -0.5, 0.0, None, None, None, 0, False)
    pool[table[1, 0], 3] = float("nan")
    pool[table[1, 0], 5] = float("inf")
    out = torch.empty(q.shape[0], H * d, device="cuda")
    seqlib.window_attn_mma(q.cuda(), H, G, d, d, pool.cuda(), table.cuda(), 64, seqlib.window_attn_items(plan, H // G, "cuda"), None, None, seqlib.WINDOW_ALL,
                           d ** -0.5, 0.0, None, out)
    assert not torch.isfinite(out[24:48]).any()
    for a, b in ((0, 24), (48, 72)):
        assert (out[a:b].double() - want[a:b]).abs().max() < 1e-3


@pytest.mark.parametrize("d,window", [(64, 64), (64, 128), (64, 191), (64, 192), (128, 63), (128, 64)])     # either side of the line to the mma.sync kernel
def test_a_request_does_not_depend_on_the_others_of_the_step(d, window):
    """Alone, and beside so many others that the CTAs come in several waves: the same bits."""
    H, G = 8, 8
    gen = torch.Generator().manual_seed(window)
    rows, pool, table, q, plan = _inputs([(97, 150)] + [(64, 200)] * 80, H, G, d, 64, gen)
    scale, outs = d ** -0.5, []
    for some in (plan[:1], plan):
        n = some[-1][0] + some[-1][1]
        items = seqlib.window_attn_items(some, H // G, "cuda")
        assert (items.shape[0] * G >= 4 * 148) == (len(some) > 1)
        outs.append(torch.empty(n, H * d, device="cuda"))
        seqlib.window_attn_mma(q[:n].cuda(), H, G, d, d, pool.cuda(), table.cuda(), 64, items, None, None, window, scale, 0.0, None, outs[-1])
    assert torch.equal(outs[0], outs[1][:97])
    want, mag = _oracle(rows, q, plan, H, G, d, window, seqlib.WINDOW_ALL, scale, 0.0, None, None, None, 0, False)
    # as test_against_float64; on mma.sync one bf16 number per probability, in the sums above and below the line
    assert ((outs[1].double() - want).abs() <= mag * (2.0 ** -13 + 2.0 ** -8) + 1e-30).all()


def test_the_largest_probability_takes_no_rounding():
    """128 keys of one score, then one whose probability is 128.49 times theirs: as two bf16 numbers relative to either maximum it is exact to 2^-17."""
    import math
    d, n = 64, 129
    rows = torch.zeros(3 * 64, 2 * d)
    rows[n - 1, d:] = 1.0                                                 # the last key's value; the others' is zero
    rows[n - 1, 0] = 1.0                                                  # its score is the scale, theirs zero
    q = torch.zeros(1, d)
    q[:, 0] = 1.0
    out = torch.empty(1, d, device="cuda")
    seqlib.window_attn_mma(q.to(BF16).cuda(), 1, 1, d, d, rows.to(BF16).view(3, 64, 2 * d).cuda(), torch.arange(3, dtype=torch.int32).view(1, -1).cuda(), 64,
                           seqlib.window_attn_items([(0, 1, 0, n - 1)], 1, "cuda"), None, None, seqlib.WINDOW_ALL, math.log(128.49), 0.0, None, out)
    assert (out.double().cpu() - 128.49 / (128.49 + 128)).abs().max() < 2e-5
