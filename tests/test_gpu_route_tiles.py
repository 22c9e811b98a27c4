"""Router logits by tiles of sixteen rows and sixteen experts: the bits of the kernel that takes a warp an expert, at the edges of tiles and of the 256 k and 128 k
that a block and a warp take at a time."""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,E,K", [(1, 16, 8), (16, 17, 128), (17, 33, 136), (5, 16, 256), (33, 64, 264), (40, 20, 1000), (3, 2048, 512)])
def test_tiles_give_the_bits_of_single_rows(dtype, rows, E, K):
    from borrowed_compute_b200 import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(rows + E + K)
    x = torch.randn(rows, K, generator=g, device="cuda").to(dtype)
    w = torch.randn(E, K, generator=g, device="cuda") / K ** 0.5
    got = []
    for tiles in (1, 0, -1):
        ops.lib().bc_moe_set_route_tiles(ctypes.c_int(tiles))
        logits = torch.full((rows, E), float("nan"), device="cuda")
        choice, weight = torch.empty((rows, 2), dtype=torch.int32, device="cuda"), torch.empty((rows, 2), device="cuda")
        try:
            ops.moe_route(x, w, None, logits, choice, weight, softmax=True, renorm=True, factor=1.0, correction=None, groups=1, keep=1)
        finally:
            ops.lib().bc_moe_set_route_tiles(ctypes.c_int(-1))
        got.append((logits, choice, weight))
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))
    full, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert ((got[0][0].double() - full).abs() <= (K + 4) * 2.0 ** -24 * size).all()
