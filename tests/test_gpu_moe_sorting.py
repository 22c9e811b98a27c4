"""Pairs sorted by expert and the products over them: whole numbers, so the sort is compared exactly, with a stable sort on the host, at numbers
of pairs around a warp's share, a run of 1,024 and several runs, and numbers of experts up to and past what the run's kernels count.

Tolerance of the products: a sum of K products in float, which the tensor core may cut off instead of rounding:
at most K 2^-23 sum |x w|; then bf16's 2^-8 where the result is bf16."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEV = "cuda:0"


def plan(choice, experts, tile_rows):
    from borrowed_compute_b200 import ops

    tiles = ops.moe_max_tiles(choice.numel(), experts, tile_rows)
    make = lambda n: torch.full((n,), -7, dtype=torch.int32, device=DEV)       # noqa: E731
    counts, offsets, table, perm, place = make(experts), make(experts + 1), make(1 + 3 * tiles), make(choice.numel()), make(choice.numel())
    ops.moe_plan(choice, experts, counts, offsets, table, perm, place, tile_rows)
    return counts, offsets, table, perm, place, tiles


@pytest.mark.parametrize("pairs", [1, 31, 33, 255, 257, 1000, 1024, 1025, 2047, 2048, 2049, 5000])
@pytest.mark.parametrize("experts", [1, 3, 64, 1000, 1024, 1025])
def test_sorted_by_expert(pairs, experts):
    rng = np.random.default_rng(pairs + experts)
    choice = rng.integers(-1, experts + 2, pairs).astype(np.int32)             # -1: a padding row; past the experts: identities
    if experts == 64:
        choice[rng.random(pairs) < 0.5] = 7                                    # half of all at one expert
    valid = (choice >= 0) & (choice < experts)
    order = np.flatnonzero(valid)[np.argsort(choice[valid], kind="stable")]
    for tile_rows in (16, 256):
        counts, offsets, table, perm, place, _ = (t.cpu().numpy() if torch.is_tensor(t) else t for t in plan(torch.tensor(choice, device=DEV), experts, tile_rows))
        want = np.bincount(choice[valid], minlength=experts)
        assert np.array_equal(counts, want) and np.array_equal(offsets, np.concatenate([[0], np.cumsum(want)]))
        assert np.array_equal(perm[:len(order)], order) and np.array_equal(place[order], np.arange(len(order)))
        tiles = [(e, int(offsets[e]) + a, min(tile_rows, int(want[e]) - a)) for e in range(experts) for a in range(0, int(want[e]), tile_rows)]
        assert table[0] == len(tiles) and np.array_equal(table[1:1 + 3 * len(tiles)].reshape(-1, 3), np.array(tiles, dtype=np.int32).reshape(-1, 3))


@pytest.mark.parametrize("tile_rows", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("N,K,kind", [(40, 8, "plain"), (136, 72, "gated"), (300, 520, "plain"), (128, 200, "relu2"), (264, 128, "gated")])
def test_products_over_groups_of_every_size(tile_rows, N, K, kind):
    """Groups of no rows, one, and numbers around 16, 64 and the tile's rows; more pieces than a device has multiprocessors."""
    from borrowed_compute_b200 import ops

    sizes = [0, 1, 15, 16, 17, 0, 63, 64, 65, 127, 129, 255, 256, 257, 300, 2, 0]
    gen = torch.Generator(device=DEV)
    gen.manual_seed(N + K)
    M = len(sizes)
    choice = torch.tensor(np.repeat(np.arange(M), sizes), dtype=torch.int32, device=DEV)
    rows = choice.numel()
    x = torch.randn(rows, K, generator=gen, device=DEV).bfloat16()
    w = (torch.randn(M, N * (2 if kind == "gated" else 1), K, generator=gen, device=DEV) / K ** 0.5).bfloat16()
    _, _, table, _, _, tiles = plan(choice, M, tile_rows)
    out = torch.full((rows, N), float("nan"), dtype=torch.float32 if kind == "plain" else torch.bfloat16, device=DEV)
    ops.gemm_tc_grouped(x, w, out, table, kind == "gated", tile_rows, tiles, relu2=kind == "relu2")
    at = 0
    for m, n in enumerate(sizes):
        if not n:
            continue
        full = x[at:at + n].double() @ w[m].double().T
        err = (K + 8) * 2.0 ** -23 * (x[at:at + n].double().abs() @ w[m].double().abs().T)
        if kind == "gated":
            g, u = full[:, :N], full[:, N:]
            act = g * torch.sigmoid(g)
            ref = act * u
            err = 1.1 * err[:, :N] * u.abs() + err[:, N:] * act.abs() + err[:, :N] * err[:, N:] + 2.0 ** -8 * ref.abs() + 1e-30
        elif kind == "relu2":
            ref = full.clamp(min=0) ** 2
            err = 2 * full.abs() * err + err ** 2 + 2.0 ** -8 * ref + 1e-30
        else:
            ref = full
        assert ((out[at:at + n].double() - ref).abs() <= err).all(), (m, n)
        at += n


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [1, 8, 12, 2048, 2052])
def test_gathered_rows(dtype, K):
    from borrowed_compute_b200 import ops

    rows, top, experts = 50, 3, 5
    gen = torch.Generator(device=DEV)
    gen.manual_seed(K)
    choice = torch.randint(-1, experts, (rows, top), generator=gen, device=DEV, dtype=torch.int32)
    x, weight = torch.randn(rows, K, generator=gen, device=DEV).to(dtype), torch.rand(rows, top, generator=gen, device=DEV)
    x[3] = float("nan")
    choice[3] = -1
    _, offsets, _, perm, _, _ = plan(choice.view(-1), experts, 32)
    n = int(offsets[experts])
    pair = perm[:n].long()
    for on_input in (False, True):
        out = torch.full((rows * top, K), 5.0, dtype=dtype, device=DEV)
        ops.moe_gather(x, perm, offsets, weight, out, experts, top, on_input)
        ref = x[pair // top]
        if on_input:
            ref = (weight.view(-1)[pair][:, None] * ref.float()).to(dtype)
        assert torch.equal(out[:n], ref) and (out[n:] == 0).all()
