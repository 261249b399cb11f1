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
