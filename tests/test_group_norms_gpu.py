"""The gated RMS norms over groups of a row (gate in front or behind) at the widths that lanes of one warp hold, and beside them; the convolution's rows that start
inside and at the edges of a tile of rows."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu
BF16, F64 = torch.bfloat16, torch.float64
ACT = {0: lambda z: z, seqlib.GATE_SILU: torch.nn.functional.silu, seqlib.GATE_SIGMOID: torch.sigmoid}


@pytest.mark.parametrize("n", [4, 31, 32, 64, 96, 128, 256, 512, 1024, 2048])
@pytest.mark.parametrize("T,groups", [(1, 1), (7, 3), (300, 8)])
@pytest.mark.parametrize("dt", [torch.float32, BF16])
@pytest.mark.parametrize("pad", [0, 1, 4])     # columns behind a row: strides that the vector loads take and one that they do not
def test_norms(n, T, groups, dt, pad):
    gen = torch.Generator().manual_seed(n + T)
    cols = groups * n
    x = (torch.randn(T, cols + pad, generator=gen) * 2)[:, :cols].cuda()
    for front in (True, False):
        for act in (0, seqlib.GATE_SILU, seqlib.GATE_SIGMOID):
            gate = torch.randn(T, cols + pad, generator=gen).to(dt if front else torch.float32)[:, :cols].cuda()
            w = (1 + 0.3 * torch.randn(cols if front else n, generator=gen)).to(dt).cuda()
            out = torch.full((T, cols + pad), float("nan"), dtype=dt, device="cuda")[:, :cols]
            g = ACT[act](gate.to(F64)).view(T, groups, n)
            v = x.to(F64).view(T, groups, n)
            if front:
                seqlib.gate_rms_rows(x, groups, w, 1e-6, gate, act, out)
                v = v * g
            else:
                seqlib.gated_rms_rows(x, groups, n, w, 1e-6, gate, act, out)
            want = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6) * w.to(F64).view(groups if front else 1, n) * (1.0 if front else g)
            # a sum of n squares in fp32, an activation and some five products: 2^-24 (log2 n + 12); eight significant bits round by up to 2^-8
            bound = want.abs() * (2.0 ** -24 * (n.bit_length() + 12) + (2.0 ** -8 if dt == BF16 else 0.0)) + 1e-30
            assert ((out.to(F64).view(T, groups, n) - want).abs() <= bound).all(), (front, act)


@pytest.mark.parametrize("taps", [1, 2, 4])
@pytest.mark.parametrize("portions", [[(1, 0)], [(8, 0), (8, 5), (8, 1)], [(3, 2), (1, 0), (300, 0), (2, 1), (9, 7), (64, 3)]])
@pytest.mark.parametrize("offset", [0, 1])     # the weights on 16 bytes or not
def test_convolution_rows(taps, portions, offset):
    ch, P = 128, len(portions)
    gen = torch.Generator().manual_seed(taps)
    T = sum(n for n, _ in portions)
    x = torch.randn(T, ch, generator=gen)
    w = torch.randn(ch * taps + offset, generator=gen).to(BF16)[offset:].view(ch, taps)
    b = torch.randn(ch, generator=gen).to(BF16)
    pos = torch.cat([torch.arange(p, p + n) for n, p in portions]).int()
    slot = torch.cat([torch.full((n,), s) for s, (n, _) in enumerate(portions)]).int()
    ring = torch.randn(P, max(1, taps - 1), ch, generator=gen)
    want, kept, at = torch.empty(T, ch, dtype=F64), ring.to(F64).clone(), 0
    for s, (n, p) in enumerate(portions):
        for i in range(n):
            acc = b.to(F64)
            for j in range(taps):
                back, sp = taps - 1 - j, p + i - (taps - 1 - j)
                if sp >= 0:
                    acc = acc + w[:, j].to(F64) * (x[at + i - back].to(F64) if back <= i else ring[s, sp % (taps - 1)].to(F64))
            want[at + i] = acc
        for i in range(max(0, n - taps + 1), n):
            kept[s, (p + i) % max(1, taps - 1)] = x[at + i].to(F64)
        at += n
    state = ring.cuda()
    y = torch.empty(T, ch, device="cuda")
    wd = torch.empty(ch * taps + offset, dtype=BF16, device="cuda")[offset:].view(ch, taps)
    wd.copy_(w)
    seqlib.causal_conv_silu(x.cuda(), wd, pos.cuda(), slot.cuda(), state if taps > 1 else None, y, act=seqlib.CONV_LINEAR, bias=b.cuda())
    assert ((y.cpu().to(F64) - want).abs() <= 2.0 ** -21 * (1 + want.abs()) * 4).all()     # five products and sums of numbers of a few units
    if taps > 1:
        assert torch.equal(state.cpu().to(F64), kept)
