"""The recurrence's kernel for portions of several tokens (64 or 128 key channels): CTAs of 16 columns where those are few, of 32 beyond; whole and ragged stages of eight
tokens. The same bits as a token at a time, which the general kernel computes, from a fresh state and from one that is carried on."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("kind", ["steps", "delta", "const", "given", "given_plain", "given_minus_one"])
@pytest.mark.parametrize("H,G,vdim", [(3, 1, 20), (2, 2, 132), (80, 2, 36)])       # 80 heads of 36 columns, three portions: 480 CTAs
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("first", [0, 5])
def test_portions_give_the_bits_of_single_tokens(kind, H, G, dim, vdim, first):
    gen = torch.Generator().manual_seed(H * dim + vdim)
    rn = lambda *s: torch.randn(*s, generator=gen).cuda()  # noqa: E731
    lens = [9, 16, 31]
    T, P = sum(lens), len(lens)
    q, v = rn(T, G * dim), rn(T, H * vdim)
    k = torch.nn.functional.normalize(rn(T, G, dim), dim=-1).reshape(T, -1).contiguous()
    a, beta, A_log, dtb, D = rn(T, H * dim if "given" in kind else H), rn(T, H), rn(H) - 1, rn(H) - 1, rn(H)
    if "given" in kind:
        a = torch.sigmoid(a + 3) - (1.0 if kind == "given_minus_one" else 0.0)

    def scan(rows, state, out, row_begin, portions, pos, slot):
        kw = {"steps": dict(step_size=True, a=a[rows], A_log=A_log, dt_bias=dtb, D=D), "const": dict(decay_const=torch.sigmoid(D), out_scale=0.5),
              "delta": dict(a=a[rows], A_log=A_log, dt_bias=dtb, beta=beta[rows]), "given": dict(a=a[rows], beta=beta[rows], channel_decay=True, decay_given=True),
              "given_plain": dict(a=a[rows], channel_decay=True, decay_given=True),
              "given_minus_one": dict(a=a[rows], channel_decay=True, decay_given=True, sigmoid_pow=1.0)}[kind]
        seqlib.linear_state_scan(q[rows], k[rows], v[rows], state, out, row_begin, portions, pos, slot, H, G, dim, vdim, **kw)

    starts = [sum(lens[:i]) for i in range(P + 1)]
    pos, slot = _i32([first + p for n in lens for p in range(n)]), _i32([i for i, n in enumerate(lens) for _ in range(n)])
    S = rn(P, H, dim, vdim) if first else torch.full((P, H, dim, vdim), float("nan"), device="cuda")
    S1, whole = S.clone(), torch.empty(T, H * vdim, device="cuda")
    scan(slice(None), S, whole, _i32(starts), P, pos, slot)
    assert torch.isfinite(whole).all() and torch.isfinite(S).all()
    for t in range(max(lens)):
        rows = [starts[i] + t for i, n in enumerate(lens) if t < n]
        out = torch.empty(len(rows), H * vdim, device="cuda")
        scan(torch.tensor(rows, device="cuda"), S1, out, _i32(list(range(len(rows) + 1))), len(rows), pos[rows].contiguous(), slot[rows].contiguous())
        assert torch.equal(out, whole[rows]), t
    assert torch.equal(S1, S)
