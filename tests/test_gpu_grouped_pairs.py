"""The product over groups of rows on pairs of SMs, where it goes wrong first: tiles of one row to 256, rows that are no multiple of what a pair multiplies, two and
four weight tiles with and without a remainder, short and ragged K.

Tolerance: a float sum of K products in any order is off by at most K 2^-23 sum |x w| (the tensor core truncates); then one rounding to bfloat16, 2^-8."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kind", ["plain", "gated", "relu2"])
@pytest.mark.parametrize("counts,N,K", [([1, 256, 31, 33, 255], 256, 64), ([129, 0, 200, 64, 3], 200, 72), ([300, 17], 512, 584), ([16, 32, 160], 400, 8)])
def test_pairs_give_what_single_blocks_give(counts, N, K, kind):
    from borrowed_compute_b200 import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(N + K)
    rows, at, table = sum(counts), 0, []
    for m, c in enumerate(counts):
        for o in range(0, c, 256):
            table += [m, at + o, min(256, c - o)]
        at += c
    tiles = len(table) // 3
    table = torch.tensor([tiles] + table, dtype=torch.int32, device="cuda")
    x = torch.randn(rows, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(len(counts), (2 if kind == "gated" else 1) * N, K, generator=g, device="cuda") / K ** 0.5).bfloat16()
    outs = []
    for pair in (True, False):
        out = torch.full((rows, N), float("nan"), dtype=torch.float32 if kind == "plain" else torch.bfloat16, device="cuda")
        ops.set_gemm_tc_pair(pair)
        try:
            ops.gemm_tc_grouped(x, w, out, table, kind == "gated", 256, tiles, relu2=kind == "relu2")
        finally:
            ops.set_gemm_tc_pair(True)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    at = 0
    for m, c in enumerate(counts):
        a, b = x[at:at + c].double(), w[m].double()
        full, off = a @ b.T, (K + 4) * 2.0 ** -23 * (a.abs() @ b.abs().T)
        got = outs[0][at:at + c].double()
        at += c
        if kind == "plain":
            assert ((got - full).abs() <= off).all()
        elif kind == "relu2":
            want = full.clamp(min=0) ** 2
            assert ((got - want).abs() <= 2 * off * full.abs() + off ** 2 + 2.0 ** -8 * want + 1e-30).all()
        else:
            gate, up, og, ou = full[:, :N], full[:, N:], off[:, :N], off[:, N:]
            act = gate * torch.sigmoid(gate)
            # |silu'| <= 1.1; the hardware's exponential and quotient are good to a few 2^-22, far inside bfloat16's 2^-8
            assert ((got - act * up).abs() <= 1.1 * og * up.abs() + ou * act.abs() + og * ou + (2.0 ** -8 + 2.0 ** -18) * (act * up).abs() + 1e-30).all()
