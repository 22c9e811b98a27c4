"""Sequences of several lengths go through the scan of chunks longest first, one a lane or two, and every one has the bits that it has alone."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def step(kind, lens, proj, weights, before):
    from borrowed_compute_b200 import ops

    H, D, inner, rows, state = 2, 32, 8, sum(lens), before.clone()
    starts = i32([sum(lens[:i]) for i in range(len(lens) + 1)])
    out = torch.full((rows, H * D), 7.0, device="cuda")
    if kind == "delta":
        pack = torch.empty((ops.delta_chunked_scratch(rows, len(lens), H, D, inner, 0.6),), device="cuda")
        ops.delta_chunked(proj, *weights, torch.empty_like(out), pack, state, starts, i32(range(len(lens))), out, len(lens), max(lens), H, D, 0.6, 1e-6)
    else:
        hd = H * D
        pack = torch.empty((ops.gla_chunked_scratch(proj, 2 * hd, len(lens), H, D, D, inner),), device="cuda")
        ops.gla_chunked(proj, 0, hd, 2 * hd, 4 * hd, *weights[:2], 16.0, 0.2, pack, state, starts, i32(range(len(lens))), out, len(lens), max(lens), H, D, D)
    return out, state


@pytest.mark.parametrize("kind", ["delta", "linear"])
@pytest.mark.parametrize("lens", [[40, 3], [17, 200, 16], [5 * i % 37 + 1 for i in range(32)], [1] * 32 + [90], [7 * i % 61 + 1 for i in range(64)], [20, 9] * 32 + [30], [18] * 5, [16] * 8 + [700]],
                         ids=["2", "3", "32", "33", "64", "65", "alike", "alone"])
def test_mixed_lengths(kind, lens):
    g = torch.Generator(device="cuda")
    g.manual_seed(len(lens))
    rnd = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    HD, rows = 64, sum(lens)
    proj, weights, before = rnd(rows, (5 if kind == "delta" else 4) * HD + 8), (rnd(8, HD), rnd(HD), rnd(HD)), 0.3 * rnd(len(lens), 2, 32, 32)
    out, state = step(kind, lens, proj, weights, before)
    at = 0
    for i, n in enumerate(lens):
        if i % 7 == 0 or n == max(lens):
            own, after = step(kind, [n], proj[at:at + n].contiguous(), weights, before[i:i + 1])
            assert torch.equal(out[at:at + n], own) and torch.equal(state[i:i + 1], after), (i, n)
        at += n
