"""The end of the generalized delta rule: heads of one run of lanes and of several, in groups of four and less, gates over the whole range."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,heads,dim", [(1, 1, 4), (3, 4, 32), (5, 5, 36), (2, 7, 60), (9, 64, 64), (3, 3, 68), (2, 2, 128)])
def test_finish(dtype, rows, heads, dim):
    from borrowed_compute_b200 import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(rows + heads + dim)
    rnd = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    HD, eps = heads * dim, 1e-5
    o, proj, weight, out = rnd(rows, HD), rnd(rows, HD + 8), rnd(HD), torch.empty((rows, HD), dtype=dtype, device="cuda")
    gates = torch.tensor([float("inf"), -float("inf"), 3e38, -3e38, -87.0, -88.5, 88.5, 17.0, -17.0, 0.0, -100.0, 1e-40], device="cuda")
    n = min(HD, len(gates))
    proj[0, 8:8 + n] = gates[:n]
    ops.delta_finish(o, proj, 8, weight, out, heads, dim, eps)
    x = o.double().view(rows, heads, dim)
    want = (x / (x.square().mean(-1, keepdim=True) + eps).sqrt()).view(rows, HD) * weight.double() * torch.sigmoid(proj[:, 8:].double())
    # Seven additions of positive numbers and a square, halved by the root; a quotient, a root and two products; an exponential (2 ulp), a sum and a
    # reciprocal; the rounding to the result's type.  A gate below 2^-126 is off by the smallest float, below 2^-128 (its exponential overflows) it is
    # zero; a result is off by half the smallest of its type.
    u = 2.0 ** -24
    store, least = (u, 2.0 ** -150) if dtype == torch.float32 else (2.0 ** -8, 2.0 ** -134)
    gate = torch.sigmoid(proj[:, 8:].double())
    size = (want / gate).abs().nan_to_num(0.0, 0.0, 0.0)
    gate_off = torch.where(gate < 2.0 ** -127.9, 2.0 ** -127.9, 2.0 ** -149)
    assert ((out.double() - want).abs() <= (16 * u + store) * want.abs() + gate_off * (size + 1) + least).all()
    assert (out[0, :n][gates[:n] < -89.0] == 0.0).all(), "a gate that is shut lets nothing through"
    # With an infinity behind it the result is not a number: zero times infinity.
    weight[0], proj[0, 8] = float("inf"), -100.0
    ops.delta_finish(o, proj, 8, weight, out, heads, dim, eps)
    assert out[0, 0].isnan()
