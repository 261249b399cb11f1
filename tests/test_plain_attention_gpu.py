"""The plain attention kernels (omc_window_attn, omc_latent_attn) at the widest rows they take, and what lies beyond."""
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
