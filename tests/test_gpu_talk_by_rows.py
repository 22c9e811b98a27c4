"""Talking attention where the mix goes by rows (sixteen heads of sixteen rows or thirty-two of eight a block), and the kernel that prepares its operands a
warp a head: rows and positions around their tiles of 8, 16 and 32, windows and kept first positions around a tile's borders, pages that
are not held, numbers that are none in positions of no sequence, positions shared out over several blocks.

Tolerance of the attention: a weight is rounded to bf16 (2^-9 of it) before it meets the values and the result once more, so a result is
off by at most 2 x 2^-9 of the largest value (gates are at most 1); 2^-8 of it is allowed, and 1e-4 for the scores' float sums."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEV = "cuda:0"


def i32(a):
    return torch.tensor(a, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("window,keep", [(0, 0), (1, 0), (32, 0), (33, 5), (64, 32), (65, 33), (100, 70)])
@pytest.mark.parametrize("H,G,D", [(16, 8, 64), (16, 4, 128), (32, 16, 64), (32, 8, 128)])
def test_mixed_by_rows(H, G, D, window, keep):
    from borrowed_compute_b200 import ops

    gen = torch.Generator(device=DEV)
    gen.manual_seed(H + D + window)
    rnd = lambda *shape: torch.randn(*shape, generator=gen, device=DEV)       # noqa: E731
    seqs = [(0, 1), (0, 16), (0, 17), (5, 33), (100, 40), (63, 2), (200, 70), (0, 5)]       # (positions held, new rows)
    n_pages = sum(-(-(a + n) // 64) for a, n in seqs) + 2
    perm = torch.randperm(n_pages, generator=gen, device=DEV).tolist()
    k, v = rnd(n_pages, G, 64, D).bfloat16(), rnd(n_pages, G, 64, D).bfloat16()
    rows = sum(n for _, n in seqs)
    q, gate = rnd(rows, H * D).bfloat16(), torch.sigmoid(rnd(rows, H * D))
    temp, talk, scale, cap = 1.0 + 0.2 * rnd(H), torch.eye(H, device=DEV) + 0.3 * rnd(H, H) / H ** 0.5, 1.5 / D ** 0.5, 6.0
    table = torch.full((len(seqs), 6), -1, dtype=torch.int32)
    ref, at, used, owned = torch.zeros(rows, H * D, dtype=torch.float64, device=DEV), 0, 0, torch.zeros(n_pages, 64, dtype=torch.bool, device=DEV)
    bounds, slot = [0], []
    for s, (held, n) in enumerate(seqs):
        total = held + n
        ids = perm[used:used + -(-total // 64)]
        used += len(ids)
        kk, vv = (t[ids].permute(1, 0, 2, 3).reshape(G, -1, D)[:, :total].double().repeat_interleave(H // G, 0) for t in (k, v))
        raw = torch.einsum("rhd,hnd->hrn", q[at:at + n].view(n, H, D).double(), kk) * scale * temp.double()[:, None, None]
        mixed = torch.einsum("hm,mrn->hrn", talk.double(), cap * torch.tanh(raw / cap))
        i, j = torch.arange(held, total, device=DEV)[:, None], torch.arange(total, device=DEV)[None]
        sees = (j <= i) & ((i - j < window) | (j < keep) | (window == 0))
        p = torch.softmax(mixed.masked_fill(~sees, -float("inf")), -1)
        if s < len(seqs) - 1:
            ref[at:at + n] = torch.einsum("hrn,hnd->rhd", p, vv).reshape(n, -1) * gate[at:at + n].double()
        for b, page in enumerate(ids):                                       # pages that no row sees are given back
            seen = sees[:, b * 64:(b + 1) * 64].any()
            table[s, b] = page if seen else -1
            if seen:
                owned[page, :min(64, total - b * 64)] = True
        at += n
        bounds.append(at)
        slot += [s if s < len(seqs) - 1 else -1] * n
    for t in (k, v):
        t.masked_fill_(~owned[:, None, :, None], float("nan"))
    for splits in (1, 3):
        out = torch.full((rows, H * D), 3.0, dtype=torch.bfloat16, device=DEV)
        ops.talk_tiles(q, k, v, table.to(DEV), i32(bounds), i32(list(range(len(seqs) - 1)) + [-1]), i32([a for a, _ in seqs]), gate, temp, talk, out,
                       len(seqs), max(n for _, n in seqs), H, G, D, window, keep, scale, cap, splits=splits, row_slot=i32(slot))
        live = bounds[-2]
        assert (out[:live].double() - ref[:live]).abs().max() <= 2.0 ** -8 * v[owned[:, None, :, None].expand_as(v)].abs().max().double() + 1e-4, splits


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,D,rot,extra", [(3, 1, 4, 0, 0), (5, 2, 128, 128, 0), (9, 3, 64, 16, 4), (2, 1, 20, 8, 0), (4, 4, 36, 4, 0), (3, 3, 40, 40, 1),
                                             (2, 2, 132, 8, 0), (7, 7, 6, 2, 0)])
def test_operands_a_warp_a_head(dtype, H, G, D, rot, extra):
    """Widths that four neighbouring values a lane take and widths that they do not; ``extra`` columns move the gate off a 16-byte border."""
    from borrowed_compute_b200 import ops

    gen = torch.Generator(device=DEV)
    gen.manual_seed(H * D + rot)
    rnd = lambda *shape: torch.randn(*shape, generator=gen, device=DEV)       # noqa: E731
    rows, g_at = 50, (H + G) * D + extra                     # (no two rows at one position of a slot)
    proj, bias, eps = rnd(rows, g_at + H * D), rnd((H + G) * D), 1e-5
    pos = [(i * 3) % 150 for i in range(rows)]
    slots = [i % 2 if i % 7 else -1 for i in range(rows)]
    table = i32([[1, 3, 0], [2, -1, 4]])
    angles = torch.arange(150, device=DEV)[:, None] * 100.0 ** (-2.0 * torch.arange(max(rot // 2, 1), device=DEV) / max(rot, 1))
    cos_sin = torch.stack([angles.cos(), angles.sin()], -1).float().contiguous()
    z = (proj[:, :(H + G) * D] + bias).double().view(rows, H + G, D)
    turned = z.clone()
    if rot:
        c, s = (cos_sin[pos][:, None, :, i].double() for i in (0, 1))
        a, b = z[..., :rot // 2], z[..., rot // 2:rot]
        turned[..., :rot // 2], turned[..., rot // 2:rot] = a * c - b * s, b * c + a * s
    unit = turned / torch.sqrt((turned ** 2).mean(-1, keepdim=True) + eps)
    tol = 1e-5 if dtype == torch.float32 else 2.0 ** -8
    for write in (True, False):
        q, gate = torch.empty((rows, H * D), dtype=dtype, device=DEV), torch.empty((rows, H * D), device=DEV)
        k, v = (torch.full((5, G, 64, D), 9.0, dtype=dtype, device=DEV) for _ in range(2))
        want_k, want_v = k.double(), v.double()
        ops.talk_prepare(proj, g_at, bias, cos_sin if rot else None, i32(pos), i32(slots), table, q, k, v, gate, H, G, D, rot, eps, write_cache=write)
        assert (q.double() - unit[:, :H].reshape(rows, -1)).abs().max() <= tol * unit.abs().max()
        assert (gate.double() - torch.sigmoid(proj[:, g_at:].double())).abs().max() <= 1e-6
        for r in range(rows if write else 0):
            page = int(table[slots[r], pos[r] // 64]) if slots[r] >= 0 else -1
            if page >= 0:
                want_k[page, :, pos[r] % 64], want_v[page, :, pos[r] % 64] = unit[r, H:], z[r, H:]
        assert (k.double() - want_k).abs().max() <= tol * max(unit.abs().max(), 1.0)
        assert (v.double() - want_v).abs().max() <= tol * max(z.abs().max(), 1.0)


@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("H,G,D", [(16, 8, 64), (32, 8, 128)])
def test_more_tiles_than_pages_are_kept(H, G, D, splits):
    """A block keeps the pages of its first 256 tiles of 32 positions and looks the others up: rows that see 8,300 positions without a window, a
    page that is not held and a last page that is not full beyond them."""
    from borrowed_compute_b200 import ops

    gen = torch.Generator(device=DEV)
    gen.manual_seed(H)
    rnd = lambda *shape: torch.randn(*shape, generator=gen, device=DEV)       # noqa: E731
    held, n, scale, cap = 8297, 9, 1.5 / D ** 0.5, 6.0
    total = held + n
    pages = -(-total // 64)
    table = torch.randperm(pages, generator=gen, device=DEV).int()
    k, v = rnd(pages, G, 64, D).bfloat16(), rnd(pages, G, 64, D).bfloat16()
    for t in (k, v):
        t[table[-1].long(), :, (total - 1) % 64 + 1:] = float("nan")
    kk, vv = (t[table.long()].permute(1, 0, 2, 3).reshape(G, -1, D)[:, :total].double().repeat_interleave(H // G, 0) for t in (k, v))
    gone = torch.zeros(total, dtype=torch.bool, device=DEV)
    for page in (3, 128):
        gone[page * 64:(page + 1) * 64] = True
        table[page] = -1
    # Some weight on every part: the positions past the 256th tile are as likely as the others, so a wrong page among them shows.
    q, gate = rnd(n, H * D).bfloat16(), torch.sigmoid(rnd(n, H * D))
    temp, talk = 1.0 + 0.2 * rnd(H), torch.eye(H, device=DEV) + 0.3 * rnd(H, H) / H ** 0.5
    kk[:, 8192:] *= 3.0
    k[table[129].long(), :, :] *= 3.0
    raw = torch.einsum("rhd,hnd->hrn", q.view(n, H, D).double(), kk) * scale * temp.double()[:, None, None]
    mixed = torch.einsum("hm,mrn->hrn", talk.double(), cap * torch.tanh(raw / cap))
    i, j = torch.arange(held, total, device=DEV)[:, None], torch.arange(total, device=DEV)[None]
    p = torch.softmax(mixed.masked_fill(~((j <= i) & ~gone), -float("inf")), -1)
    ref = torch.einsum("hrn,hnd->rhd", p, vv).reshape(n, -1) * gate.double()
    assert p[:, :, 8256:].sum(-1).mean() > 0.02
    out = torch.full((n, H * D), 3.0, dtype=torch.bfloat16, device=DEV)
    ops.talk_tiles(q, k, v, table[None].contiguous(), i32([0, n]), i32([0]), i32([held]), gate, temp, talk, out, 1, n, H, G, D, 0, 0, scale, cap, splits=splits,
                   row_slot=i32([0] * n))
    # (8,300 weights of about the same size: the largest value that a result has is far below the largest value that it is a mean of)
    assert (out.double() - ref).abs().max() <= 2.0 ** -8 * ref.abs().max() + 1e-4
    without = torch.einsum("hrn,hnd->rhd", torch.softmax(mixed.masked_fill(~((j <= i) & ~gone & (j < 8192)), -float("inf")), -1), vv).reshape(n, -1) * gate.double()
    assert (without - ref).abs().max() > 4 * (2.0 ** -8 * ref.abs().max() + 1e-4)
