"""The step before latent attention, at the sizes and borders where it goes from quads to single values: queries, cached vectors, rotated parts and gates against 64 bits."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -24


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("QR,R,ROT,H,pad,offset", [
    (4, 4, 0, 4, 0, 0), (512, 508, 2, 2, 0, 0), (516, 512, 64, 20, 0, 0), (2048, 512, 128, 16, 0, 0),        # quads
    (2052, 512, 64, 16, 0, 0), (512, 256, 64, 16, 2, 0), (512, 256, 64, 16, 0, 1), (513, 255, 64, 3, 1, 0), (6, 510, 4, 1, 1, 0)])
def test_prepare(dtype, QR, R, ROT, H, pad, offset):
    from borrowed_compute_b200 import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(QR + R + ROT + pad + offset)
    rnd = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    rows, P, eps = 5, QR + R + ROT + H + pad, 1e-6
    proj = rnd(rows * P + offset)[offset:].view(rows, P)
    q_w, kv_w, cos_sin = rnd(QR), rnd(R), rnd(200, max(ROT // 2, 1), 2)
    row_slot = torch.tensor([1, 0, -1, 1, 0], dtype=torch.int32, device="cuda")
    row_pos = torch.tensor([0, 63, 4, 64, 130], dtype=torch.int32, device="cuda")
    table = torch.tensor([[5, 1, 2], [3, 0, 4]], dtype=torch.int32, device="cuda")
    c_pages, r_pages = torch.full((6, 1, 64, R), 7.0, device="cuda", dtype=dtype), torch.full((6, 1, 64, max(ROT, 1)), 7.0, device="cuda", dtype=dtype)
    cq, gate = torch.empty((rows, QR), dtype=dtype, device="cuda"), torch.empty((rows, H), device="cuda")
    ops.latent_prepare(proj, QR, QR, R, ROT, QR + R + ROT, H, q_w, kv_w, cos_sin if ROT else None, row_pos, row_slot, table, c_pages, r_pages if ROT else None, cq, gate, eps)

    x, half = proj.double(), ROT // 2
    store = U if dtype == torch.float32 else 2.0 ** -8
    def near(got, want, size, terms):     # a sum of n squares is off by at most n U of itself, its root by half of that; a root, a quotient and two products, then the rounding
        assert ((got.double() - want).abs() <= ((terms / 2 + 6) * U + store) * 1.01 * size).all()
    norm = lambda v, w: v / (v.square().mean(1, keepdim=True) + eps).sqrt() * w.double()
    want = norm(x[:, :QR], q_w)
    near(cq, want, want.abs(), QR)
    want = torch.sigmoid(x[:, QR + R + ROT:QR + R + ROT + H])
    assert ((gate.double() - want).abs() <= 8 * U * want).all()
    c, z = norm(x[:, QR:QR + R], kv_w), x[:, QR + R:QR + R + ROT]
    places = {(3, 0): 0, (5, 63): 1, (0, 0): 3, (2, 2): 4}
    untouched = torch.ones((6, 64), dtype=torch.bool, device="cuda")
    for (page, at), row in places.items():
        near(c_pages[page, 0, at], c[row], c[row].abs(), R)
        untouched[page, at] = False
        if ROT:
            f, u, v = cos_sin[row_pos[row].item()].double(), z[row, :half], z[row, half:]
            near(r_pages[page, 0, at], torch.cat([u * f[:, 0] - v * f[:, 1], v * f[:, 0] + u * f[:, 1]]),
                 torch.cat([(u * f[:, 0]).abs() + (v * f[:, 1]).abs(), (v * f[:, 0]).abs() + (u * f[:, 1]).abs()]), 0)
    assert (c_pages[:, 0][untouched] == 7.0).all() and (r_pages[:, 0][untouched] == 7.0).all()
