"""Results of the paired product that go out through shared memory: the bits of those that go straight to memory, at the edges of tiles, of the 16 or 32 tokens
and 128 outputs of a buffer, of outputs whose rows tensor copies do and do not take, and nothing past them."""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("epilogue", ["store", "add", "glu", "relu2"])
@pytest.mark.parametrize("T,N,K", [(129, 128, 64), (200, 520, 72), (257, 136, 200), (300, 1000, 264), (513, 2052, 128), (130, 131, 64), (1025, 640, 64)])
def test_both_ways_give_the_same_bits(T, N, K, epilogue):
    from borrowed_compute_b200 import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(T + N + K)
    epi = {"store": ops.EPI_STORE, "add": ops.EPI_ADD_F32, "glu": ops.EPI_SWIGLU, "relu2": ops.EPI_RELU2}[epilogue]
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn((2 if epilogue == "glu" else 1) * N, K, generator=g, device="cuda") / K ** 0.5).bfloat16()
    dtype = torch.float32 if epilogue == "add" else torch.bfloat16
    base = torch.randn(T, N, generator=g, device="cuda").to(dtype)
    outs = []
    for staged in (1, 0):
        room = torch.full((T * N + 64,), 7.0, dtype=dtype, device="cuda")
        out = room[:T * N].view(T, N)
        out.copy_(base)
        ops.lib().bc_gemm_tc_set_pair_staged(ctypes.c_int(staged))
        try:
            ops.gemm_tc(x, w, out, epi, splits=1)
        finally:
            ops.lib().bc_gemm_tc_set_pair_staged(ctypes.c_int(1))
        assert (room[T * N:] == 7.0).all(), "something was written past the output"
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    full = x.double() @ w.double().T
    off = (K + 4) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)      # truncated float sums
    if epilogue == "add":
        ref = base.double() + full
        assert ((outs[0].double() - ref).abs() <= off + 2.0 ** -23 * ref.abs()).all()
    elif epilogue == "store":
        assert ((outs[0].double() - full).abs() <= off + 2.0 ** -8 * full.abs()).all()
