"""The reciprocal, the sigmoid and the quotient without branches that the generalized delta rule works with: over their whole ranges, against 64 bits and CUDA's own division."""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

RECIPROCAL, SIGMOID, QUOTIENT = 0, 1, 2


def run(what, a, b=None):
    from borrowed_compute_b200 import ops

    out = torch.empty_like(a)
    status = ops.lib().bc_delta_arithmetic(ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(0 if b is None else b.data_ptr()), ctypes.c_void_p(out.data_ptr()), ctypes.c_int(what),
                                           ctypes.c_int(a.numel()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert status == 0
    return out


def floats(n, least, most, seed, signs=False):
    """Random significands at all exponents from least to most, and the floats next to the powers of two."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    e = torch.randint(least, most, (n,), generator=g, device="cuda")
    v = torch.ldexp(1.0 + torch.randint(0, 1 << 23, (n,), generator=g, device="cuda").double() * 2.0 ** -23, e)
    p = torch.ldexp(torch.ones(most - least + 1, dtype=torch.float64, device="cuda"), torch.arange(least, most + 1, device="cuda"))
    near = torch.cat([p, p[:-1] * (1 + 2.0 ** -23), p[1:] * (1 - 2.0 ** -24)])
    v = torch.cat([v, near]).float()
    return v * (torch.randint(0, 2, v.shape, generator=g, device="cuda") * 2 - 1) if signs else v


def ulp(want):
    """Of a float of that size: 2^-23 of its power of two, and 2^-149 at least."""
    return torch.ldexp(torch.ones_like(want), (torch.frexp(want.abs())[1] - 24).clamp_min(-149))


def test_reciprocal():
    x = floats(2_000_000, -126, 126, 1)
    want = 1.0 / x.double()
    off = ((run(RECIPROCAL, x).double() - want).abs() / ulp(want)).max().item()
    assert off <= 0.51, off
    assert run(RECIPROCAL, torch.full((1,), float("nan"), device="cuda")).isnan().all()


def test_sigmoid():
    x = torch.cat([floats(500_000, -126, 7, 2, signs=True), torch.linspace(-90, 90, 1_000_001, device="cuda")])
    x = x[x.abs() < 88.7]
    want = torch.sigmoid(x.double())
    # The exponential, 2 ulp; the sum, half an ulp; the reciprocal; below 2^-126 a rounding to 2^-149.
    off = ((run(SIGMOID, x).double() - want).abs() / ulp(want)).max().item()
    assert off <= 4.5, off
    ends = torch.tensor([float("inf"), 3e38, 89.0, -89.0, -3e38, -float("inf"), 0.0, float("nan")], device="cuda")
    got = run(SIGMOID, ends)
    assert got[:7].tolist() == [1.0, 1.0, 1.0, 0.0, 0.0, 0.0, 0.5] and got[7].isnan()


def test_quotient():
    """Keys over their lengths: the bits of CUDA's division where neither what is divided nor the quotient is tiny, and half an ulp of the quotient anyhow."""
    b = floats(2_000_000, -74, 64, 3)
    a = floats(2_000_000, -60, 60, 4, signs=True)[:b.numel()]
    b = b[:a.numel()]
    got, want = run(QUOTIENT, a, b), a / b
    plain = (want.abs() >= 2.0 ** -100) & (want.abs() < 2.0 ** 120) & (a.abs() >= 2.0 ** -100)
    assert plain.float().mean() > 0.9 and torch.equal(got[plain], want[plain])
    exact = a.double() / b.double()
    finite = want.isfinite()
    assert ((got.double() - exact).abs() / ulp(exact))[finite].max().item() <= 0.51
    inf = float("inf")
    a, b = torch.tensor([0.0, 1.0, -2.0, 0.0, inf, 0.0, float("nan"), 1.0], device="cuda"), torch.tensor([1.0, inf, inf, inf, inf, 0.0, 1.0, float("nan")], device="cuda")
    got = run(QUOTIENT, a, b)
    assert got[:4].tolist() == [0.0, 0.0, 0.0, 0.0] and got[4:].isnan().all()
