"""Sigmoids and what they gate have the bits of a division by 1 + exp(-z), also where kernels form the quotients of several numbers together: over the whole range of z, beside
numbers that are out of the common range, and for numbers that are none."""
import pytest
import torch

from omchat_b200 import seqlib

pytestmark = pytest.mark.gpu
F32, BF16 = torch.float32, torch.bfloat16
ODD = [0.0, -0.0, torch.inf, -torch.inf, torch.nan, 1e-30, -1e-42, 3e38, -3e38, -88.8, -87.0, 44.0, -44.0, 44.00001, -103.0, -200.0]


def _numbers(n):
    """Over every magnitude that matters, with odd ones in every 32nd group of four."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    z = torch.empty(n, device="cuda").uniform_(-1, 1, generator=gen)
    scale = torch.tensor([1.0, 10.0, 44.0, 120.0], device="cuda").repeat_interleave(-(-n // 4))[:n]
    z = z * scale
    odd = torch.tensor(ODD, device="cuda").repeat(-(-n // 128))[:len(range(5, n, 128))]
    z[5::128] = odd
    return z


def _same(got, want):
    return torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0))


@pytest.mark.parametrize("T,ch", [(1024, 512), (3, 512), (7, 130)])   # tiles of rows, single rows, the general kernel
@pytest.mark.parametrize("wdt", [F32, BF16])
def test_silu_behind_the_convolution(T, ch, wdt):
    z = _numbers(T * ch).view(T, ch)
    y, ids = torch.empty_like(z), torch.arange(T, dtype=torch.int32, device="cuda")
    seqlib.causal_conv_silu(z, torch.ones(ch, 1, dtype=wdt, device="cuda"), ids, torch.zeros_like(ids), None, y)
    z = z + 0.0     # the sum of taps begins with zero
    assert _same(y, z / (1 + torch.exp(-z)))


def test_silu_of_rows_in_place():
    z = _numbers(1 << 20).view(256, 4096)
    want = z / (1 + torch.exp(-z))
    assert _same(seqlib.map_rows(z, seqlib.MAP_SILU), want)


@pytest.mark.parametrize("n", [64, 128, 512, 96])    # lanes of one warp that hold one piece of four or four of them; the kernel for other widths
@pytest.mark.parametrize("act", [seqlib.GATE_SILU, seqlib.GATE_SIGMOID])
@pytest.mark.parametrize("front", [False, True])
def test_gates_beside_a_norm(n, act, front):
    rows = 2000
    z = _numbers(rows * n).view(rows, n)
    if front:       # what a norm can take
        z = torch.where(z.abs() < 1e3, z, torch.full_like(z, -60.0))
    g = z / (1 + torch.exp(-z)) if act == seqlib.GATE_SILU else 1 / (1 + torch.exp(-z))
    one, x, got, want = (torch.ones(*s, device="cuda") for s in ((n,), (rows, n), (rows, n), (rows, n)))
    if front:       # the gate as it is against the gate that the kernel forms
        seqlib.gate_rms_rows(x, 1, one, 1e-6, z, act, got)
        seqlib.gate_rms_rows(x, 1, one, 1e-6, g, seqlib.GATE_NONE, want)
    else:
        seqlib.gated_rms_rows(x, 1, n, one, 0.0, z, act, got)
        want = g
    assert _same(got, want)


@pytest.mark.parametrize("gdt", [F32, BF16])
def test_gated_products(gdt):
    M, N = 3000, 128
    gate = _numbers(M * N).view(M, N).to(gdt)
    x = _numbers(M * N + 77)[77:].view(M, N).roll(1, 1).nan_to_num(2.0, 3.0, -3.0).to(BF16)
    x[::7] *= 1e-25
    x[1::7] *= 1e20
    w = torch.eye(N, device="cuda").to(BF16)
    y, part = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    seqlib.linear(x, w, y, M=M, N=N, K=N, ldx=N, ldw=N, ldy=N, gate=gate)
    seqlib.linear(x, w[:N - 2], part, M=M, N=N - 2, K=N, ldx=N, ldw=N, ldy=N, gate=gate[:, :N - 2])     # its last 62 columns are divided one by one
    assert _same(y[:, :N - 2], part[:, :N - 2])
    want = x.double() * torch.sigmoid(gate.double())
    normal = (want.abs() > 1e-36) & x.isfinite().all(1, keepdim=True) & gate.isfinite() & (gate > -88)     # from 88.7 on the exponential is an infinity, the result zero
    err = (y.double() - want).abs()
    # the product is exact; a fast exponential (its argument is off by 2^-24 of up to 88 / ln 2), a sum, a quotient
    assert (err[normal] <= 128 * 2.0 ** -23 * want.abs()[normal]).all() and normal.sum() > 0.8 * M * N
