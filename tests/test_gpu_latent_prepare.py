"""The step before latent attention, at the sizes where a row fits the threads' registers and beyond, and at odd borders: queries, cached vectors, rotated parts and gates against 64 bits."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -24


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("QR,R,ROT,H,pad,offset", [
    (4, 4, 0, 4, 0, 0), (512, 508, 2, 2, 0, 0), (516, 512, 64, 20, 0, 0), (2048, 512, 128, 16, 0, 0),
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


def _one_over_rms(v, eps):
    """1 / rms of rows of floats with few bits, rounded as the kernel's order rounds: 128 threads' running sums of every 128th square, each warp's by
    halves, the four warps' as (0 + 2) + (1 + 3).  A square and a sum of such values are exact in 64 bits, so that one rounding follows."""
    import numpy as np

    rows, n = v.shape
    padded = np.zeros((rows, -(-n // 128) * 128))
    padded[:, :n] = v
    s = np.zeros((rows, 128), dtype=np.float32)
    for part in np.split(padded, padded.shape[1] // 128, axis=1):
        s = (part * part + s).astype(np.float32)
    s = s.reshape(rows, 4, 32)
    for half in (16, 8, 4, 2, 1):
        s = s[..., :half] + s[..., half:2 * half]
    w = s[..., 0]
    total = (w[:, 0] + w[:, 2]) + (w[:, 1] + w[:, 3])
    return np.float32(1.0) / np.sqrt(total / np.float32(n) + np.float32(eps))


@pytest.mark.parametrize("QR,R,pad", [(1536, 512, 0), (2048, 512, 0), (2052, 256, 0), (510, 254, 1), (100, 8, 0)])
def test_sums_in_one_order(QR, R, pad):
    """Whatever the sizes and borders, a row's sums are added up in one order, to the bit."""
    import numpy as np

    from borrowed_compute_b200 import ops

    rows, P, eps = 64, QR + R + 1 + pad, 1e-6
    rng = np.random.default_rng(QR + R)
    x = rng.standard_normal((rows, P)).astype(np.float32)
    x = torch.from_numpy(x).bfloat16().float()
    dev = x.cuda()
    ones = torch.ones(max(QR, R), device="cuda")
    slot, pos = torch.zeros(rows, dtype=torch.int32, device="cuda"), torch.arange(rows, dtype=torch.int32, device="cuda")
    table = torch.zeros((1, 1), dtype=torch.int32, device="cuda")
    c_pages, cq, gate = torch.empty((1, 1, 64, R), device="cuda"), torch.empty((rows, QR), device="cuda"), torch.empty((rows, 1), device="cuda")
    ops.latent_prepare(dev, QR, QR, R, 0, QR + R, 1, ones[:QR], ones[:R], None, pos, slot, table, c_pages, None, cq, gate, eps)
    v = x.numpy()
    assert np.array_equal(cq.cpu().numpy(), v[:, :QR] * _one_over_rms(v[:, :QR], eps)[:, None])
    assert np.array_equal(c_pages[0, 0].cpu().numpy(), v[:, QR:QR + R] * _one_over_rms(v[:, QR:QR + R], eps)[:, None])
