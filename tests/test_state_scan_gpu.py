"""omc_linear_state_scan: token by token (the kernel that shares a sum through shared memory), a few tokens at a time and whole portions (the one that
defers the read-out) give the same bits, at every number of key channels per thread, ragged widths and both stage lengths."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("kind", ["steps", "delta", "delta_channel", "const"])
@pytest.mark.parametrize("H,G,dim,vdim", [(2, 1, 32, 36), (3, 3, 60, 34), (2, 2, 64, 64), (4, 2, 128, 96), (2, 1, 136, 33), (2, 1, 256, 64), (200, 1, 128, 64)])
def test_one_token_at_a_time_gives_the_bits_of_the_whole(H, G, dim, vdim, kind):
    gen = torch.Generator().manual_seed(H * dim + vdim)
    rn = lambda *s: torch.randn(*s, generator=gen).cuda()  # noqa: E731
    lens = [35, 16, 1]                     # past two stages, exactly one, one token
    T, P = sum(lens), len(lens)
    q, v = rn(T, G * dim), rn(T, H * vdim)
    k = torch.nn.functional.normalize(rn(T, G, dim), dim=-1).reshape(T, -1).contiguous()
    a, beta, A_log, dtb, D = rn(T, H * dim if kind == "delta_channel" else H), rn(T, H), rn(H) - 1, rn(H * dim if kind == "delta_channel" else H) - 1, rn(H)

    def scan(rows, state, out, row_begin, portions, pos, slot):
        kw = {"steps": dict(step_size=True, a=a[rows], A_log=A_log, dt_bias=dtb, D=D), "const": dict(decay_const=torch.sigmoid(D), silu_in=True),
              "delta": dict(a=a[rows], A_log=A_log, dt_bias=dtb, beta=beta[rows]),
              "delta_channel": dict(a=a[rows], A_log=A_log, dt_bias=dtb, beta=beta[rows], channel_decay=True)}[kind]
        seqlib.linear_state_scan(q[rows], k[rows], v[rows], state, out, row_begin, portions, pos, slot, H, G, dim, vdim, **kw)

    starts = [sum(lens[:i]) for i in range(P + 1)]
    pos, slot = _i32([p for n in lens for p in range(n)]), _i32([i for i, n in enumerate(lens) for _ in range(n)])
    whole, S = torch.empty(T, H * vdim, device="cuda"), torch.full((P, H, dim, vdim), float("nan"), device="cuda")
    scan(slice(None), S, whole, _i32(starts), P, pos, slot)
    assert torch.isfinite(whole).all() and torch.isfinite(S).all()
    for step in (1, 3):                    # 3: portions of few tokens, which take shorter stages
        S1 = torch.full_like(S, float("nan"))
        for t in range(0, max(lens), step):
            pieces = [list(range(starts[i] + t, starts[i] + min(t + step, n))) for i, n in enumerate(lens) if t < n]
            rows = sum(pieces, [])
            out = torch.empty(len(rows), H * vdim, device="cuda")
            begin = _i32([sum(map(len, pieces[:i])) for i in range(len(pieces) + 1)])
            scan(torch.tensor(rows, device="cuda"), S1, out, begin, len(pieces), pos[rows].contiguous(), slot[rows].contiguous())
            assert torch.equal(out, whole[rows]), (step, t)
        assert torch.equal(S1, S), step
