"""omc_latent_rope_store by pieces of four against float64: latents beyond what waits in registers, rotations of all, a part or none of a head, both pairings, short steps (heads spread
over CTAs) and long ones, queries kept beside; rows off the 16-byte grid take the kernel that goes column by column."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu
F32, BF16 = torch.float32, torch.bfloat16


@pytest.mark.parametrize("dt,qdt,keep", [(BF16, F32, True), (BF16, BF16, False), (F32, F32, False)])
@pytest.mark.parametrize("r,dr,rot,H,dn", [(512, 64, 64, 16, 128), (2052, 40, 8, 3, 4), (64, 32, 0, 33, 128), (256, 64, 32, 5, 64)])
@pytest.mark.parametrize("T", [1, 64, 65])
@pytest.mark.parametrize("halves", [False, True])
@pytest.mark.parametrize("off", [0, 1])
def test_rows_and_queries_against_float64(dt, qdt, keep, r, dr, rot, H, dn, T, halves, off):
    gen = torch.Generator(device="cuda").manual_seed(r + T)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    page, pages = 64, 4
    dkv = rn(T, r + dr + 4)[:, off:off + r + dr]
    q, w = rn(T, H * (dn + dr)).to(qdt), (1 + 0.2 * rn(r)).to(dt)
    angle = rn(page * pages, max(1, rot // 2))
    cs = torch.stack([angle.cos(), angle.sin()], -1).contiguous()
    pos = torch.arange(3, 3 + T, dtype=torch.int32, device="cuda")
    slot = torch.zeros(T, dtype=torch.int32, device="cuda")
    table = torch.tensor([[2, 0, 3, 1]], dtype=torch.int32, device="cuda")
    pool, qcat = torch.full((pages, page, r + dr), 7.0, device="cuda", dtype=dt), torch.full((T, H, r + dr), 7.0, device="cuda", dtype=dt)
    qn = torch.empty(T, H * dn, device="cuda", dtype=dt) if keep else None
    seqlib.latent_rope_store(dkv, r, dr, w, 1e-6, cs, rot, pos, slot, table, page, pool, q, H, dn, qcat, qn=qn, rot_halves=halves)

    def turn(x):     # [T, ..., dr]
        x = x.double().clone()
        c, s = (cs[pos.long(), :rot // 2, i].double().view(T, *([1] * (x.dim() - 2)), rot // 2) for i in (0, 1))
        a, b = (slice(0, rot // 2), slice(rot // 2, rot)) if halves else (slice(0, rot, 2), slice(1, rot, 2))
        u, v = x[..., a].clone(), x[..., b].clone()
        x[..., a], x[..., b] = u * c - v * s, v * c + u * s
        return x

    d = dkv.double()
    want = torch.cat([d[:, :r] / torch.sqrt((d[:, :r] ** 2).mean(-1, keepdim=True) + 1e-6) * w.double(), turn(dkv[:, r:])], 1)
    got = pool[table[0, pos.long() // page].long(), pos.long() % page].double()
    # a sum of r squares, a few roundings in fp32, the output's own
    eps = 2.0 ** -8 if dt == BF16 else 0.0
    assert ((got - want).abs() <= want.abs() * (eps + 2e-6) + 2e-6).all()
    q3 = q.view(T, H, dn + dr)
    wq = turn(q3[..., dn:])
    assert ((qcat[..., r:].double() - wq).abs() <= wq.abs() * (eps + 2e-6) + 2e-6).all() and (qcat[..., :r] == 7.0).all()
    if keep:
        assert torch.equal(qn.view(T, H, dn), q3[..., :dn].to(dt))


@pytest.mark.parametrize("dt,qdt", [(BF16, F32), (BF16, BF16), (F32, F32)])
@pytest.mark.parametrize("r,dr,rot,H,dn", [(512, 64, 64, 16, 128), (2052, 40, 8, 3, 4), (64, 32, 0, 33, 128), (256, 64, 32, 5, 64), (1200, 64, 48, 2, 32)])
@pytest.mark.parametrize("T", [7, 65])
@pytest.mark.parametrize("halves", [False, True])
def test_rows_have_the_same_bits_on_and_off_the_grid(dt, qdt, r, dr, rot, H, dn, T, halves):
    gen = torch.Generator(device="cuda").manual_seed(r + T)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    row, q, w = rn(T, r + dr), rn(T, H * (dn + dr)).to(qdt), (1 + 0.2 * rn(r)).to(dt)
    angle = rn(128, max(1, rot // 2))
    cs = torch.stack([angle.cos(), angle.sin()], -1).contiguous()
    pos, slot, table = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (list(range(3, 3 + T)), [0] * T, [[1, 0]]))
    got = []
    for off in (0, 1):      # rows off 16 bytes go column by column
        dkv = torch.zeros(T, r + dr + 4, device="cuda")[:, off:off + r + dr]
        dkv.copy_(row)
        pool, qcat, qn = torch.zeros(2, 64, r + dr, device="cuda", dtype=dt), torch.zeros(T, H, r + dr, device="cuda", dtype=dt), torch.empty(T, H * dn, device="cuda", dtype=dt)
        seqlib.latent_rope_store(dkv, r, dr, w, 1e-6, cs, rot, pos, slot, table, 64, pool, q, H, dn, qcat, qn=qn, rot_halves=halves)
        got.append((pool, qcat, qn))
    assert all(torch.equal(a, b) for a, b in zip(*got))
