"""omc_causal_conv with unit vectors: groups that lie in neighbouring lanes of a warp (rows kernel) and groups that do not, in portions of long and of
one-token steps, against float64; the ring of the last inputs."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ch,group,unit,scaled", [(384, 128, 256, 128), (256, 4, 8, 4), (512, 32, 512, 0), (128, 16, 112, 64), (640, 64, 320, 64),
                                                  (384, 24, 240, 48), (200, 8, 40, 8), (512, 256, 256, 256)])
@pytest.mark.parametrize("taps,ydt", [(4, torch.float32), (2, torch.bfloat16), (1, torch.float32)])
def test_unit_groups(ch, group, unit, scaled, taps, ydt):
    gen = torch.Generator().manual_seed(ch + group)
    lens = [270, 3, 41]                       # one step of 314 rows, then one row per request
    T = sum(lens)
    x, nxt = torch.randn(T, ch, generator=gen), torch.randn(3, ch, generator=gen)
    w = torch.randn(ch, taps, generator=gen).to(torch.bfloat16)
    pos = torch.tensor([p for n in lens for p in range(n)], dtype=torch.int32).cuda()
    slot = torch.tensor([i for i, n in enumerate(lens) for _ in range(n)], dtype=torch.int32).cuda()
    state = torch.full((3, max(taps - 1, 1), ch), float("nan"), device="cuda") if taps > 1 else None
    kw = dict(unit_channels=unit, unit_group=group, unit_eps=1e-6, scaled_channels=scaled, unit_mult=0.25)
    y, y1 = torch.empty(T, ch, dtype=ydt, device="cuda"), torch.empty(3, ch, dtype=ydt, device="cuda")
    seqlib.causal_conv_silu(x.cuda(), w.cuda(), pos, slot, state, y, **kw)
    ends = torch.tensor(lens, dtype=torch.int32).cuda()
    seqlib.causal_conv_silu(nxt.cuda(), w.cuda(), ends, torch.arange(3, dtype=torch.int32).cuda(), state, y1, single_rows=True, **kw)
    at = 0
    for s, n in enumerate(lens):
        full = torch.cat([x[at:at + n], nxt[s:s + 1]]).double()
        want = torch.zeros(n + 1, ch, dtype=torch.float64)
        for j in range(taps):
            back = taps - 1 - j
            want[back:] += w[:, j].double() * full[:n + 1 - back]
        want = torch.nn.functional.silu(want)
        u = want[:, :unit].view(n + 1, -1, group)
        u = u / torch.sqrt((u * u).sum(-1, keepdim=True) + 1e-6)
        want = torch.cat([u.reshape(n + 1, unit), want[:, unit:]], 1)
        want[:, :scaled] *= 0.25
        got = torch.cat([y[at:at + n], y1[s:s + 1]]).double().cpu()
        # a few roundings of values of order one (taps, silu, sum of squares, quotient), then the output's own
        assert ((got - want).abs() <= 4e-6 * (1 + want.abs()) + (want.abs() * 2.0 ** -8 if ydt == torch.bfloat16 else 0)).all()
        at += n


@pytest.mark.parametrize("T", [256, 259, 263, 700])
@pytest.mark.parametrize("unit", [0, 64])
def test_tiles_of_four_and_eight_rows_agree(T, unit):
    """Weights of 16 bits take tiles of four rows, of 32 bits tiles of eight; the ring is written beside the end of the convolution and read by the next one."""
    gen = torch.Generator().manual_seed(T)
    x = torch.randn(2 * T, 512, generator=gen).cuda()
    w = torch.randn(512, 4, generator=gen).to(torch.bfloat16).cuda()
    lens = [T - 11, 2, 9]
    slot = torch.tensor([i for i, n in enumerate(lens) for _ in range(n)], dtype=torch.int32).cuda()
    pos = torch.tensor([p for n in lens for p in range(n)], dtype=torch.int32).cuda()
    after = pos + torch.tensor(lens, dtype=torch.int32).cuda()[slot.long()]
    kw = dict(unit_channels=256, unit_group=unit, unit_eps=1e-6, scaled_channels=128, unit_mult=0.5) if unit else {}
    got = []
    for wt in (w, w.float()):
        state, y = torch.full((3, 3, 512), float("nan"), device="cuda"), torch.empty(2 * T, 512, device="cuda")
        seqlib.causal_conv_silu(x[:T], wt, pos, slot, state, y[:T], **kw)
        seqlib.causal_conv_silu(x[T:], wt, after, slot, state, y[T:], **kw)
        got.append((y, state))
    assert torch.isfinite(got[0][0]).all() and torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    whole = torch.empty(2 * lens[0], 512, device="cuda")     # the first request in one go
    rows = torch.cat([x[:lens[0]], x[T:T + lens[0]]])
    n = torch.arange(2 * lens[0], dtype=torch.int32).cuda()
    seqlib.causal_conv_silu(rows, w, n, torch.zeros_like(n), torch.full((1, 3, 512), float("nan"), device="cuda"), whole, **kw)
    assert torch.equal(torch.cat([got[0][0][:lens[0]], got[0][0][T:T + lens[0]]]), whole)
