"""The tcgen05 latent attention (omc_latent_attn_mma_rows, as seqlib calls it, and the two other entries, where r is a multiple of 128 and pages of 64 rows) against float64: tile edges, portions behind a cached prefix, windows that start inside a box, decode steps in key ranges, sinks, gates,
rows of the cache that hold no key."""
import math

import pytest
import torch

from omchat_b200 import seqlib
from omchat_b200.model.seq_latent import LatentAttention

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _reference(q, pool_rows, portions, r, scale, window, sink, gate):
    """out [T, H, r] and the weighted sums of |latent| that bound the effect of rounded probabilities."""
    out, mag = torch.zeros(*q.shape[:2], r, dtype=F64), torch.zeros(*q.shape[:2], r, dtype=F64)
    for row, n, slot, first in portions:
        keys = pool_rows[slot][:first + n].to(F64)
        s = torch.einsum("thd,jd->htj", q[row:row + n].to(F64), keys) * scale
        i, j = first + torch.arange(n)[:, None], torch.arange(first + n)[None, :]
        s = s.masked_fill((j > i) | (i - j >= window), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.to(F64)[:, None, None].expand(-1, n, 1)], -1)
        p = torch.softmax(s, -1)[..., :first + n]
        g = torch.sigmoid(gate[row:row + n].to(F64))[..., None] if gate is not None else 1.0
        out[row:row + n] = torch.einsum("htj,jr->thr", p, keys[:, :r]) * g
        mag[row:row + n] = torch.einsum("htj,jr->thr", p, keys[:, :r].abs()) * g
    return out, mag


@pytest.mark.parametrize("H,r,dr,page,window,portions", [
    (16, 512, 64, 64, 1 << 30, [(5, 0), (4, 123), (9, 124), (1, 127), (1, 128), (133, 60)]),
    (16, 512, 64, 128, 100, [(70, 0), (64, 300), (1, 511), (3, 190)]),
    (8, 256, 32, 64, 1 << 30, [(129, 0), (1, 640), (17, 63)]),
    (32, 512, 48, 64, 64, [(40, 50), (1, 0), (2, 2000)]),
    (5, 128, 16, 192, 1 << 30, [(13, 0), (30, 100)]),
    (3, 384, 0, 64, 33, [(50, 0), (1, 200)]),
    (64, 512, 64, 64, 1 << 30, [(3, 254)]),
])
@pytest.mark.parametrize("opt", ["plain", "sink_gate"])
def test_against_float64(H, r, dr, page, window, portions, opt):
    gen = torch.Generator().manual_seed(H * r + dr)
    D, row, slots, plist = r + dr, 0, [], []
    for s, (n, first) in enumerate(portions):
        plist.append((row, n, s, first))
        row += n
        slots.append(-(-(first + n) // page))
    T, pages = row, sum(slots) + 1
    pool = torch.full((pages, page, D), float("nan"), dtype=torch.bfloat16)      # rows that hold no key must not matter
    order, table, rows = (torch.randperm(pages - 1, generator=gen) + 1).tolist(), torch.zeros(len(slots), max(slots), dtype=torch.int32), []
    for s, ((_, n, _, first), k) in enumerate(zip(plist, slots)):
        mine, order = order[:k], order[k:]
        table[s, :k] = torch.tensor(mine, dtype=torch.int32)
        lat = torch.randn(first + n, D, generator=gen).to(torch.bfloat16)
        rows.append(lat)
        for i in range(k):
            part = lat[i * page:(i + 1) * page]
            pool[mine[i], :part.shape[0]] = part
    q = (torch.randn(T, H, D, generator=gen) * 2).to(torch.bfloat16)
    scale = 3.0 * D ** -0.5                                                      # scores of some tens: references move, sums are rescaled
    sink = torch.randn(H, generator=gen) * 3 if opt == "sink_gate" else None
    gate = torch.randn(T, H, generator=gen) if opt == "sink_gate" else None
    want, mag = _reference(q, rows, plist, r, scale, window, sink, gate)
    dev = lambda t: t.cuda() if t is not None else None  # noqa: E731
    pos = torch.cat([torch.arange(first, first + n) for _, n, _, first in plist]).to(torch.int32).cuda()
    slot = torch.cat([torch.full((n,), s) for _, n, s, _ in plist]).to(torch.int32).cuda()
    plans = [seqlib.LatentAttnPlan(plist, H, "cuda", window=window), seqlib.LatentAttnPlan(plist, H, "cuda", target_ctas=2, window=window)]
    for parts in (1, 3):                                                         # every row on its own, as a decode step addresses them
        plan = seqlib.DecodeAttnPlan(T, H, parts, "cuda", window=window)
        plan.fill(pos, slot)
        plans.append(plan)
    for plan in plans:
        for dt in (torch.float32, torch.bfloat16):
            out = torch.full((T, H, r), float("nan"), dtype=dt, device="cuda")
            seqlib.latent_attn_mma(q.cuda(), r, dr, pool.cuda(), table.cuda(), page, plan, dev(sink), scale, out, window=window, gate=dev(gate))
            err = (out.double().cpu() - want).abs()
            # a probability is rounded to 8 bits (its sum too: 2^-9 each), scores and sums in fp32 over D terms; then the output's own rounding
            bound = mag * (2.0 ** -8 + 1e-4) + 1e-6 + (want.abs() * 2.0 ** -8 if dt == torch.bfloat16 else 0.0)
            assert (err <= bound).all(), (plan.n_items, plan.max_rows, dt, float((err - bound).max()))


@pytest.mark.parametrize("r,dr,page", [(512, 64, 64), (256, 16, 64), (128, 64, 128), (512, 64, 32)])
@pytest.mark.parametrize("parts", [1, 2])
def test_the_largest_probability_takes_no_rounding(r, dr, page, parts):
    """128 keys of one score and, in the next tile, one whose probability is 128.49 times theirs: relative to the row's maximum every number is
    exact in bf16, relative to the first tile's 128.49 would become 128 (an error of 1e-3 in the output). Page 32: the mma.sync kernel."""
    H, n, D = 16, 129, r + dr
    pages = -(-n // page)
    rows = torch.zeros(pages * page, D)
    rows[n - 1, :r] = 1.0                                                        # the last key's value; the others' is zero
    rows[n - 1, r] = 1.0                                                         # its score is the scale, theirs zero
    q = torch.zeros(1, H, D)
    q[:, :, r] = 1.0
    pos, slot = torch.tensor([n - 1], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda()
    plan = seqlib.DecodeAttnPlan(1, H, parts, "cuda")
    plan.fill(pos, slot)
    out = torch.empty(1, H, r, device="cuda")
    table = torch.arange(pages, dtype=torch.int32).view(1, -1).cuda()
    seqlib.latent_attn_mma(q.to(torch.bfloat16).cuda(), r, dr, rows.to(torch.bfloat16).view(pages, page, D).cuda(), table, page, plan, None, math.log(128.49),
                           out)
    # the exponent (7) is known to 2^-21, the hardware exponential to 2^-22, the sums of 129 terms to 2^-17
    assert (out.double().cpu() - 128.49 / (128.49 + 128)).abs().max() < 1e-5


def test_no_wait_ran_out():
    import ctypes
    n = ctypes.c_uint(7)
    assert seqlib.load().omc_step_wait_failures(ctypes.byref(n)) == 0 and n.value == 0


@pytest.mark.parametrize("r,dr", [(128, 32), (256, 16), (512, 64)])
def test_a_pool_that_ends_with_its_mapping(r, dr):
    """The last row of the pool is the last of an allocation of whole 2 MB pages, and nothing is kept behind it: every copy stays inside the rows."""
    H, D, pages = 4, r + dr, 1024
    gen = torch.Generator().manual_seed(D)
    torch.cuda.empty_cache()
    pool = torch.zeros(pages, 64, D, dtype=torch.bfloat16, device="cuda")
    assert pool.numel() * 2 % (2 << 20) == 0
    rows, q = torch.randn(192, D, generator=gen).to(torch.bfloat16), torch.randn(3, H, D, generator=gen).to(torch.bfloat16)
    pool[-3:] = rows.view(3, 64, D).cuda()
    table = torch.arange(pages - 3, pages, dtype=torch.int32).view(1, 3).cuda()
    qd, out = q.cuda(), torch.empty(3, H, r, device="cuda")
    plist = [(0, 3, 0, 192 - 3)]                                                 # the last three positions: their rows end where the pool does
    plans = [seqlib.LatentAttnPlan(plist, H, "cuda", **cut) for cut in ({}, dict(target_ctas=148, min_keys=64))]
    pos = torch.arange(192 - 3, 192, dtype=torch.int32).cuda()
    plans.append(seqlib.DecodeAttnPlan(3, H, 2, "cuda"))
    plans[-1].fill(pos, torch.zeros(3, dtype=torch.int32, device="cuda"))
    want, mag = _reference(q, [rows], plist, r, D ** -0.5, 1 << 30, None, None)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    for plan in plans:
        seqlib.latent_attn_mma(qd, r, dr, pool, table, 64, plan, None, D ** -0.5, out)
        assert ((out.double().cpu() - want).abs() <= mag * (2.0 ** -8 + 1e-4) + 1e-6).all()


@pytest.mark.parametrize("H,r,dr,n,first", [(16, 512, 64, 9, 500), (16, 512, 0, 70, 300), (32, 512, 32, 40, 129), (16, 384, 64, 33, 60), (8, 128, 32, 20, 700)])
@pytest.mark.parametrize("decode", [0, 1, 3])
def test_probabilities_are_not_rounded_to_8_bits(H, r, dr, n, first, decode):
    """Two bf16 numbers per probability, in every place that shared memory has for them; whole contexts, key ranges and decode steps."""
    gen = torch.Generator().manual_seed(r + dr + n)
    D, pages = r + dr, -(-(n + first) // 64)
    rows, q = torch.randn(pages * 64, D, generator=gen).to(torch.bfloat16), torch.randn(n, H, D, generator=gen).to(torch.bfloat16)
    plist, scale = [(0, n, 0, first)], 3.0 * D ** -0.5
    if decode:
        plan = seqlib.DecodeAttnPlan(n, H, decode, "cuda")
        plan.fill(torch.arange(first, first + n, dtype=torch.int32).cuda(), torch.zeros(n, dtype=torch.int32).cuda())
    else:
        plan = seqlib.LatentAttnPlan(plist, H, "cuda", target_ctas=2)
    out = torch.empty(n, H, r, device="cuda")
    seqlib.latent_attn_mma(q.cuda(), r, dr, rows.view(pages, 64, D).cuda(), torch.arange(pages, dtype=torch.int32).view(1, -1).cuda(), 64, plan, None, scale, out)
    want, mag = _reference(q, [rows], plist, r, scale, 1 << 30, None, None)
    # 2^-18 per probability; scores of up to some 15 from fp32 sums of D products, exponentials and sums of up to 720 keys in fp32
    assert ((out.double().cpu() - want).abs() <= mag * (2.0 ** -17 + 6e-5) + 1e-6).all()


@pytest.mark.parametrize("H,r,portions,window", [(16, 512, [(40, 0), (3, 60)], 1 << 30), (32, 128, [(150, 0), (200, 40)], 70), (8, 256, [(5, 300)], 20)])
def test_steps_of_few_keys_take_the_other_kernel(H, r, portions, window):
    """_tcgen05_pays: no more than 64 keys per tile, or latents of 128 over short windows. Both kernels give the same within their rounding."""
    gen = torch.Generator().manual_seed(r)
    D, plist, row = r + 32, [], 0
    for s, (n, first) in enumerate(portions):
        plist.append((row, n, s, first))
        row += n
    assert not LatentAttention._tcgen05_pays(plist, H, r, window) and LatentAttention._tcgen05_pays(plist, H, 256, 1 << 30) == (max(n + f for n, f in portions) > 64)
    pages = max(-(-(n + f) // 64) for n, f in portions)
    lat = [torch.randn(pages * 64, D, generator=gen).to(torch.bfloat16) for _ in portions]
    q = torch.randn(row, H, D, generator=gen).to(torch.bfloat16)
    want, mag = _reference(q, lat, plist, r, D ** -0.5, window, None, None)
    table = torch.arange(pages * len(portions), dtype=torch.int32).view(len(portions), -1).cuda()
    for tcgen05 in (True, False):
        out = torch.empty(row, H, r, device="cuda")
        plan = LatentAttention._prompt_plan(plist, H, "cuda", window, tcgen05)
        seqlib.latent_attn_mma(q.cuda(), r, 32, torch.cat(lat).view(-1, 64, D).cuda(), table, 64, plan, None, D ** -0.5, out, window=window)
        assert ((out.double().cpu() - want).abs() <= mag * (2.0 ** (-17 if tcgen05 else -8) + 6e-5) + 1e-6).all(), tcgen05


@pytest.fixture(params=["omc_latent_attn_mma", "omc_latent_attn_mma_pool"])
def other_entry(request, monkeypatch):
    """seqlib.latent_attn_mma through one of the entries that it does not call itself."""
    lib = seqlib.load()

    def call(qcat, T, H, r, dr, pool, table, max_pages, page, items, n_items, max_rows, *rest):
        if request.param == "omc_latent_attn_mma":
            return lib.omc_latent_attn_mma(qcat, T, H, r, dr, pool, table, max_pages, page, items, n_items, *rest)
        return lib.omc_latent_attn_mma_pool(qcat, T, H, r, dr, pool, 0, table, max_pages, page, items, n_items, max_rows, *rest)
    monkeypatch.setattr(lib, "omc_latent_attn_mma_rows", call)


@pytest.mark.parametrize("H,r,dr,page,window,portions", [
    (16, 512, 64, 64, 1 << 30, [(5, 0), (4, 123), (9, 124), (1, 127), (1, 128), (133, 60)]),
    (32, 512, 48, 128, 100, [(70, 0), (64, 300), (1, 511), (3, 190)]),
    (5, 128, 16, 192, 1 << 30, [(13, 0), (30, 100)]),
    (8, 384, 0, 64, 33, [(50, 0), (1, 200)]),
])
def test_other_entries_against_float64(other_entry, H, r, dr, page, window, portions):
    test_against_float64(H, r, dr, page, window, portions, "sink_gate")


@pytest.mark.parametrize("H,r,dr,n,first", [(16, 512, 64, 9, 500), (16, 512, 0, 70, 300), (16, 384, 64, 33, 60), (8, 128, 32, 20, 700)])
@pytest.mark.parametrize("decode", [0, 1, 3])
def test_other_entries_do_not_round_probabilities(other_entry, H, r, dr, n, first, decode):
    test_probabilities_are_not_rounded_to_8_bits(H, r, dr, n, first, decode)


def test_other_entries_stay_inside_the_pool(other_entry):
    test_a_pool_that_ends_with_its_mapping(512, 64)
