"""Decays of the generalized delta rule in chunks: 64 inner channels at a time, sixteen bytes of weights a copy where they start on such a border, against 64 bits."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows,heads,inner,offset", [(17, 1, 4, 0), (64, 2, 64, 0), (65, 3, 68, 0), (63, 2, 60, 0), (129, 2, 128, 0), (80, 2, 132, 0), (80, 2, 64, 1)])
def test_decays(rows, heads, inner, offset):
    from borrowed_compute_b200 import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(rows + inner + offset)
    rnd = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    D, scale = 64, 0.6
    HD = heads * D
    proj = rnd(rows, 5 * HD + inner)
    w2t = (rnd(inner * HD + offset) / inner ** 0.5)[offset:].view(inner, HD)
    w0, bias, state, decay, out = rnd(HD), rnd(HD), rnd(2, heads, D, D), torch.full((rows, HD), 7.0, device="cuda"), torch.empty((rows, HD), device="cuda")
    need = ops.delta_chunked_scratch(rows, 1, heads, D, inner, scale)
    seq_rows, seq_slot = torch.tensor([0, rows], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.delta_chunked(proj, w2t, w0, bias, decay, torch.empty((need,), device="cuda"), state, seq_rows, seq_slot, out, 1, rows, heads, D, scale, 1e-6)
    t = torch.tanh(proj[:, 5 * HD:5 * HD + inner].double())
    z, size = t @ w2t.double() + w0.double(), t.abs() @ w2t.double().abs() + w0.double().abs()
    want = torch.exp(-scale * torch.sigmoid(z))
    # z is off by at most (inner + 3) U of its terms' sizes (tanhf 2 U); a decay moves by at most scale / 4 of that; two exponentials, a sum, a quotient and a product.
    assert ((decay.double() - want).abs() <= 2.0 ** -24 * ((inner + 3) * size * scale / 4 + 12) * want).all()


@pytest.mark.parametrize("gate,key", [(0.0, 1.0), (300.0, 1.0), (-300.0, 1.0), (-87.5, 1e-25), (0.0, 1e25)])
def test_removals_at_the_ends_of_the_range(gate, key):
    """A last row whose removal gate is shut or open all the way, whose key is nearly nothing or whose key's norm is an infinity (its unit key is then zero)."""
    from borrowed_compute_b200 import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    rows, H, D, inner = 19, 2, 64, 8
    HD = H * D
    rnd = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    proj, w2t, w0, bias, before = rnd(rows, 5 * HD + inner), rnd(inner, HD), rnd(HD), torch.zeros(HD, device="cuda"), rnd(1, H, D, D)
    proj[-1, HD:2 * HD] *= key
    proj[-1, 4 * HD:5 * HD] = gate
    state, out, decay = before.clone(), torch.empty((rows, HD), device="cuda"), torch.empty((rows, HD), device="cuda")
    pack = torch.empty((ops.delta_chunked_scratch(rows, 1, H, D, inner, 0.6),), device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    ops.delta_chunked(proj, w2t, w0, bias, decay, pack, state, i32([0, rows]), i32([0]), out, 1, rows, H, D, 0.6, 1e-6)
    P = proj.double()
    r, k, v, _, a = (P[:, i * HD:(i + 1) * HD].view(rows, H, D) for i in range(5))
    w = decay.double().view(rows, H, D)
    u = k / torch.sqrt((proj[:, HD:2 * HD].view(rows, H, D) ** 2).sum(-1, keepdim=True) + 1e-6).double()
    S, size = before[0].double(), None
    for t in range(rows):
        e = (S * u[t][:, None]).sum(-1, keepdim=True)
        size = S.abs() + (e * u[t][:, None]).abs() + (v[t][..., None] * k[t][:, None]).abs()
        S = S * w[t][:, None] - e * (torch.sigmoid(a[t]) * u[t])[:, None] + v[t][..., None] * k[t][:, None]
    # Errors grow along the chain of removals; 1e-5 of the largest summand is far below what a gate or a unit key that is off by a part in a thousand gives.
    assert ((state[0].double() - S).abs() <= 1e-5 * size.amax()).all()
    assert ((out[-1].double().view(H, D) - (S * r[-1][:, None]).sum(-1)).abs() <= 1e-5 * (size * r[-1][:, None].abs()).sum(-1).amax()).all()
