"""A decoding step of the tcgen05 latent attention without a work list gives the bits that it gives with the list of omc_latent_decode_items: ranges that end in a tile, empty
ranges, windows, one to 64 heads, sink and gate. A pool off the 16-byte grid, which no tensor-core kernel can read, is refused on the host."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("H,r,dr", [(1, 128, 0), (16, 512, 64), (33, 256, 32), (64, 512, 64)])
@pytest.mark.parametrize("parts", [1, 3, 64])
@pytest.mark.parametrize("window", [seqlib.WINDOW_ALL, 100])
def test_the_bits_of_the_listed_step(H, r, dr, parts, window):
    gen = torch.Generator(device="cuda").manual_seed(H + r)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    ctx, page, D = [0, 63, 64, 700, 1], 64, r + dr
    T, mp = len(ctx), 700 // 64 + 1
    pool = rn(T * mp, page, D).to(BF16)
    table = torch.randperm(T * mp, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(T, mp).cuda()
    pos, slot = torch.tensor(ctx, dtype=torch.int32, device="cuda"), torch.tensor([3, 0, 4, 1, 2], dtype=torch.int32, device="cuda")
    q, sink, gate = rn(T, H, D).to(BF16), rn(H), rn(T, H)
    out = [torch.full((T, H, r), 7.0, dtype=BF16, device="cuda") for _ in range(2)]
    listed = seqlib.DecodeAttnPlan(T, H, parts, "cuda", window=window)
    listed.fill(pos, slot)
    for o, plan in zip(out, (listed, seqlib.DecodeRows(pos, slot, T, H, parts, window))):
        seqlib.latent_attn_mma(q, r, dr, pool, table, page, plan, sink, D ** -0.5, o, window=window, gate=gate)
    assert torch.equal(*out) and torch.isfinite(out[0]).all() and (out[0] != 7.0).any(-1).all()


@pytest.mark.parametrize("plan", ["listed", "rows"])
def test_a_pool_off_the_grid_is_refused(plan):
    pool = torch.zeros(64 * 128 + 8, dtype=BF16, device="cuda")[4:4 + 64 * 128].view(1, 64, 128)
    zero, table = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(1, 1, dtype=torch.int32, device="cuda")
    q, out = torch.zeros(1, 16, 128, dtype=BF16, device="cuda"), torch.empty(1, 16, 128, dtype=BF16, device="cuda")
    work = seqlib.DecodeRows(zero, zero, 1, 16, 1)
    if plan == "listed":
        work = seqlib.DecodeAttnPlan(1, 16, 1, "cuda")
        work.fill(zero, zero)
    with pytest.raises(seqlib.OmcError):
        seqlib.latent_attn_mma(q, 128, 0, pool, table, 64, work, None, 1.0, out)
