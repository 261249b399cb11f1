"""The recurrence's portions may be taken in the order of their lengths, and in CTAs of 64 columns where those are many: every portion has the bits that it has alone."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,vdim", [(16, 64), (64, 64), (70, 100), (3, 20)])     # 32 columns per CTA in order of length, 64, 64 with a ragged end, few CTAs
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("kind", ["steps", "head"])
def test_portions_have_the_bits_that_they_have_alone(H, vdim, dim, kind):
    lens = [300, 20, 150, 400, 1]
    gen = torch.Generator(device="cuda").manual_seed(H)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    T, P, G = sum(lens), len(lens), 1
    q, v, a = rn(T, G * dim) * dim ** -0.5, rn(T, H * vdim), rn(T, H)
    k = torch.nn.functional.normalize(rn(T, G * dim), dim=-1)
    A_log, dtb, D = rn(H), rn(H) - 2, rn(H)
    starts = [sum(lens[:i]) for i in range(P + 1)]
    S0 = rn(P, H, dim, vdim)

    def scan(rows, begin, slots, S):
        n = rows.stop - rows.start
        out = torch.empty(n, H * vdim, device="cuda")
        kw = dict(step_size=True, D=D) if kind == "steps" else {}
        slot = torch.repeat_interleave(i32(slots), torch.diff(i32(begin)).long()).to(torch.int32)
        seqlib.linear_state_scan(q[rows], k[rows], v[rows], S, out, i32(begin), len(begin) - 1, torch.full((n,), 9, dtype=torch.int32, device="cuda"), slot,
                                 H, G, dim, vdim, a=a[rows], A_log=A_log, dt_bias=dtb, **kw)
        return out

    S = S0.clone()
    whole = scan(slice(0, T), starts, list(range(P)), S)
    assert torch.isfinite(whole).all()
    S1 = S0.clone()
    for i, n in enumerate(lens):
        rows = slice(starts[i], starts[i + 1])
        assert torch.equal(scan(rows, [0, n], [i], S1), whole[rows]), i
    assert torch.equal(S, S1)
