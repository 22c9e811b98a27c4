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
