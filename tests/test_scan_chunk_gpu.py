"""The recurrence's kernel for long portions (64 rows and more of the delta rule, 32 with per-channel decays): against float64 over whole and ragged stages of eight tokens
and column counts, beside short portions that keep the bits of single tokens, from a fresh state and one that is carried on."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu
KINDS = ["delta", "delta_const", "given", "given_plain", "given_minus_one"]


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


class Case:
    def __init__(self, kind, H, G, dim, vdim, lens, first):
        gen = torch.Generator().manual_seed(H * dim + vdim)
        rn = lambda *s: torch.randn(*s, generator=gen).cuda()  # noqa: E731
        self.kind, self.H, self.G, self.dim, self.vdim, self.lens, self.first = kind, H, G, dim, vdim, lens, first
        T = sum(lens)
        self.q, self.v = rn(T, G * dim) * dim ** -0.5, rn(T, H * vdim)
        self.k = torch.nn.functional.normalize(rn(T, G, dim), dim=-1).reshape(T, -1).contiguous()
        self.a, self.beta, self.A_log, self.dtb = rn(T, H * dim if "given" in kind else H), rn(T, H), rn(H) - 1, rn(H) - 1
        self.const = torch.sigmoid(rn(H) + 2)
        if "given" in kind:
            self.a = torch.sigmoid(self.a + 3) - (1.0 if kind == "given_minus_one" else 0.0)
        self.starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
        self.S0 = rn(len(lens), H, dim, vdim) if first else torch.zeros(len(lens), H, dim, vdim, device="cuda")

    def prepared(self, rows=slice(None), lens=None, slots=None, first=None, longest=None):
        """The call with everything on the device: nothing but the launches is left."""
        lens = self.lens if lens is None else lens
        slots = range(len(lens)) if slots is None else slots
        first = self.first if first is None else first
        kw = {"delta": dict(a=self.a[rows], A_log=self.A_log, dt_bias=self.dtb, beta=self.beta[rows]), "delta_const": dict(decay_const=self.const, beta=self.beta[rows], out_scale=0.5),
              "given": dict(a=self.a[rows], beta=self.beta[rows], channel_decay=True, decay_given=True),
              "given_plain": dict(a=self.a[rows], channel_decay=True, decay_given=True),
              "given_minus_one": dict(a=self.a[rows], channel_decay=True, decay_given=True, sigmoid_pow=1.0)}[self.kind]
        begin = _i32([sum(lens[:i]) for i in range(len(lens) + 1)])
        pos, slot = _i32([first + p for n in lens for p in range(n)]), _i32([s for s, n in zip(slots, lens) for _ in range(n)])
        q, k, v = self.q[rows], self.k[rows], self.v[rows]
        return lambda out, S: seqlib.linear_state_scan(q, k, v, S, out, begin, len(lens), pos, slot, self.H, self.G, self.dim, self.vdim, longest=longest, **kw)

    def run(self, rows=slice(None), lens=None, slots=None, S=None, first=None):
        S = self.S0.clone() if S is None else S
        out = torch.empty(sum(self.lens if lens is None else lens), self.H * self.vdim, device="cuda")
        self.prepared(rows, lens, slots, first)(out, S)
        return out, S

    def exact(self):
        d = lambda x: x.double()  # noqa: E731
        H, dim = self.H, self.dim
        q, k = (d(x).view(-1, self.G, dim).repeat_interleave(H // self.G, 1) for x in (self.q, self.k))
        v, b = d(self.v).view(-1, H, self.vdim), torch.sigmoid(d(self.beta))
        if self.kind == "delta":
            g = torch.exp(-torch.exp(d(self.A_log)) * torch.nn.functional.softplus(d(self.a) + d(self.dtb), threshold=1e9))[..., None]
        elif self.kind == "delta_const":
            g = d(self.const)[None, :, None].expand(len(v), H, 1)
        else:
            g = (d(self.a) + (1.0 if self.kind == "given_minus_one" else 0.0)).view(-1, H, dim)
        S, out = d(self.S0), torch.empty_like(v)
        for i, n in enumerate(self.lens):
            for t in range(self.starts[i], self.starts[i] + n):
                S[i] *= g[t][..., None]
                u = v[t] if self.kind in ("given_plain", "given_minus_one") else b[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S[i], k[t]))
                S[i] += k[t][..., None] * u[:, None]
                out[t] = torch.einsum("hdv,hd->hv", S[i], q[t])
        return out.reshape(len(v), -1) * (0.5 if self.kind == "delta_const" else 1.0), S


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("H,G,vdim", [(3, 1, 20), (2, 2, 132), (4, 2, 64)])
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("first", [0, 5])
def test_long_portions_are_as_exact_as_fp32_sums(kind, H, G, dim, vdim, first):
    c = Case(kind, H, G, dim, vdim, [64, 9, 71, 130], first)
    out, S = c.run()
    want, Sw = c.exact()
    # sums of dim + 8 products, a rounding of the state by a decay per stage: a few units of 2^-24 of the largest terms, which 2-norms see as about one
    assert _rel(out, want) < 5e-7 and _rel(S, Sw) < 5e-7, (_rel(out, want), _rel(S, Sw))
    # the short portion beside them: the bits of one token at a time; a long one alone: the bits it has in company
    S1 = c.S0.clone()
    for t in range(9):
        one, _ = c.run(slice(64 + t, 65 + t), [1], [1], S1, first + t)
        assert torch.equal(one[0], out[64 + t])
    assert torch.equal(S1[1], S[1])
    alone, S2 = c.run(slice(73, 144), [71], [2])
    assert torch.equal(alone, out[73:144]) and torch.equal(S2[2], S[2])


@pytest.mark.parametrize("kind", ["delta", "given", "given_plain"])
def test_what_is_not_finite_reaches_no_earlier_token_and_no_other_column(kind):
    c = Case(kind, 2, 1, 128, 64, [75], 0)
    clean, _ = c.run()
    c.v[37, 5], c.v[61, 70] = torch.inf, torch.nan
    out, S = c.run()
    out, clean = out.view(75, 2, 64), clean.view(75, 2, 64)
    hit = torch.zeros(75, 2, 64, dtype=torch.bool, device="cuda")
    hit[37:, 0, 5] = hit[61:, 1, 6] = True
    assert torch.equal(out[~hit], clean[~hit]) and not torch.isfinite(out[hit]).any()
    assert torch.isfinite(S).all(2).view(-1).sum() == 2 * 64 - 2


def test_many_portions_of_which_few_are_long():
    lens = [3] * 140 + [64, 200, 1]      # more portions than a CTA sorts by length
    c = Case("delta", 2, 1, 64, 36, lens, 0)
    out, S = c.run()
    want, Sw = c.exact()
    assert _rel(out, want) < 5e-7 and _rel(S, Sw) < 5e-7


@pytest.mark.parametrize("kind", ["delta", "given"])
@pytest.mark.parametrize("lens", [[3] * 128 + [70, 1, 64] + [2] * 170 + [97], [1] * 40 + [200], [5] * 24])   # more portions than a CTA orders, two kernels side by side, none long
def test_long_portions_among_many_short_ones(kind, lens):
    c = Case(kind, 4, 2, 64, 64, lens, 3)
    out, S = c.run()
    for i in {0, len(lens) // 2, len(lens) - 1} | {i for i, n in enumerate(lens) if n >= 64}:
        rows = slice(c.starts[i], c.starts[i + 1])
        o1, S1 = c.run(rows, [lens[i]], [i])
        assert torch.equal(o1, out[rows]) and torch.equal(S1[i], S[i]), i


@pytest.mark.parametrize("kind,H,dim", [("delta", 4, 128), ("delta", 2, 64), ("given", 2, 64), ("given", 32, 128), ("given_minus_one", 32, 64)])   # 32 heads: the general kernel has the short ones
@pytest.mark.parametrize("lens", [[1, 2000], [9, 64, 1], [1] * 8 + [2000], [1500, 1]])   # a short portion is the second kernel's first: one of its CTAs waits all the same
@pytest.mark.parametrize("graph", [False, True])
def test_what_follows_a_step_sees_the_ends_of_both_kernels(kind, H, dim, lens, graph):
    c = Case(kind, H, 1, dim, 64, lens, 3)
    want, Sw = c.run()
    torch.cuda.synchronize()
    scan, out, S = c.prepared(), torch.empty_like(want), torch.empty_like(Sw)
    out2, S2 = torch.empty_like(want), torch.empty_like(Sw)

    def step():     # copies right behind the scan read what they see then
        scan(out, S)
        out2.copy_(out)
        S2.copy_(S)

    if graph:
        side = torch.cuda.Stream()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            step()
    for _ in range(3):
        S.copy_(c.S0)
        for x in (out, out2, S2):
            x.fill_(torch.nan)
        torch.cuda.synchronize()
        g.replay() if graph else step()
        torch.cuda.synchronize()
        assert torch.equal(out2, want) and torch.equal(S2, Sw)


@pytest.mark.parametrize("n", [75, 72])     # a ragged last stage, and a whole one
def test_heads_that_forget_at_once(n):
    c = Case("delta", 2, 1, 128, 64, [n], 5)
    c.A_log[1] = 90.0     # its exponential is an infinity: a decay of zero
    out, S = c.run()
    S1 = c.S0.clone()
    single = torch.cat([c.run(slice(t, t + 1), [1], [0], S1, 5 + t)[0] for t in range(n)])
    assert torch.isfinite(single).all() and torch.isfinite(out).all() and torch.isfinite(S).all()
    # each form is within 5e-7 of float64 (above), so the two are within twice that of each other
    assert _rel(out, single.double()) < 1e-6 and _rel(S, S1.double()) < 1e-6


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("lens,rows", [([40], 100), ([1], 64), ([100, 3, 80], 70), ([100, 3, 80], 183), ([30, 64, 9], 200)])   # rows of the tensors: more than the portions have, fewer, as many
def test_what_is_computed_is_a_matter_of_row_begin(kind, lens, rows):
    n = sum(lens)
    c = Case(kind, 2, 1, 64, 36, lens + [max(rows - n, 1)], 5)
    out, S = torch.full((len(c.q), 2 * 36), torch.nan, device="cuda"), c.S0.clone()
    c.prepared(slice(0, rows), lens)(out, S)
    want, Sw = c.exact()
    assert _rel(out[:n], want[:n]) < 5e-7 and _rel(S[:-1], Sw[:-1]) < 5e-7
    assert out[n:].isnan().all() and torch.equal(S[-1], c.S0[-1])


@pytest.mark.parametrize("kind", ["delta", "given"])
@pytest.mark.parametrize("lens", [[8] * 8, [3] * 32, [63, 2], [64, 2], [40] * 2 + [90], [64, 0, 5], [31] * 3, [32, 31]])
def test_what_the_host_knows_of_lengths_changes_no_bits(kind, lens):
    c = Case(kind, 3, 1, 64, 36, lens, 2)
    want, Sw = c.run()
    for longest in (max(lens), max(lens) + 70):
        out, S = torch.full_like(want, torch.nan), c.S0.clone()
        c.prepared(longest=longest)(out, S)
        assert torch.equal(out, want) and torch.equal(S, Sw)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("same", [False, True])     # decays that differ from token to token; each channel's (head's) the same in all, close to one: errors that do not cancel
def test_eight_at_a_time_are_no_less_exact_than_one(kind, dim, same):
    c = Case(kind, 8, 4, dim, 64, [1000], 3)
    if same and "given" in kind:
        c.a = (0.998 + 0.001 * torch.rand(1, c.a.shape[1], device="cuda")).expand(1000, -1).contiguous() - (1.0 if kind == "given_minus_one" else 0.0)
    elif same:
        c.a, c.A_log, c.const = c.a[:1].expand(1000, -1).contiguous(), c.A_log - 6, 1 - 0.002 * torch.rand(8, device="cuda")
    want, Sw = c.exact()
    out, S = c.run()
    S1, outs = c.S0.clone(), []
    for lo in range(0, 1000, 20):     # portions this short go token by token
        outs.append(c.run(slice(lo, lo + 20), [20], [0], S1, 3 + lo)[0])
    # the same number of roundings or fewer; 2-norms of half a million errors, which scatter by a few parts in a thousand
    assert _rel(out, want) < 1.03 * _rel(torch.cat(outs), want) and _rel(S, Sw) < 1.03 * _rel(S1, Sw)


@pytest.mark.parametrize("kind,line", [("delta", 64), ("given", 32), ("given_plain", 32), ("given_minus_one", 32)])
def test_a_portion_has_the_same_bits_in_any_company(kind, line):
    """On both sides of the line between the kernels, and whoever else is in the step."""
    lens = [line, line - 1, line + 1, line - 7, 1, 150]
    c = Case(kind, 4, 2, 128, 64, lens, 3)
    out, S = c.run()
    want, Sw = c.exact()
    assert _rel(out, want) < 5e-7 and _rel(S, Sw) < 5e-7
    for i, n in enumerate(lens):
        rows = slice(c.starts[i], c.starts[i + 1])
        o1, S1 = c.run(rows, [n], [i])
        assert torch.equal(o1, out[rows]) and torch.equal(S1[i], S[i]), i
        if n < line:     # token by token
            S2 = c.S0.clone()
            single = torch.cat([c.run(slice(rows.start + t, rows.start + t + 1), [1], [i], S2, 3 + t)[0] for t in range(n)])
            assert torch.equal(single, o1) and torch.equal(S2[i], S1[i]), i
