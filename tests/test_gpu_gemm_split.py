"""The true 32-bit product on the tensor cores: tiles of 128 weight rows and up to 128 rows of x, chunks of 32 k, sums taken out every 64,
one piece of K or a cluster of two to eight.

Tolerance, in units of sum |x w|: the product of parts that is left out, at most 2^-33; a stretch of 64 k is four truncated additions, 4 x 2^-23;
its sums are added in float, one rounding a stretch and one a piece; the smaller products are at most 2^-6 of the whole and truncated 7 K / 16 times."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def bound(K):
    return 2.0 ** -33 + 4 * 2.0 ** -23 + (K / 64 + 8 + 3) * 2.0 ** -24 + 7 * K / 16 * 2.0 ** -29


def operands(M, N, K, seed=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N + K + seed)
    return torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda") / K ** 0.5


@pytest.mark.parametrize("M,N,K", [
    (1, 1, 516), (16, 64, 516), (17, 65, 544), (128, 128, 548), (129, 127, 576), (112, 129, 600), (257, 192, 640),       # tiles, a chunk's and a stretch's ends
    (33, 128, 1024), (5, 130, 1028), (140, 64, 2052), (20, 200, 4100), (130, 128, 8196)])                                # two, four and eight pieces
def test_products_around_the_edges_of_tiles_stretches_and_pieces(M, N, K):
    from borrowed_compute_b200 import ops

    x, w = operands(M, 2 * N, K)
    full, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    wn = w[:N].contiguous()
    out = torch.full((M, N), float("nan"), device="cuda")
    ops.gemm_simt(x, wn, out, ops.EPI_STORE_F32)
    off = bound(K) * size
    assert ((out.double() - full[:, :N]).abs() <= off[:, :N]).all()
    base = torch.randn(M, N, device="cuda")
    acc = base.clone()
    ops.gemm_simt(x, wn, acc, ops.EPI_ADD_F32)
    ref = base.double() + full[:, :N]
    assert ((acc.double() - ref).abs() <= off[:, :N] + 2.0 ** -23 * ref.abs()).all()
    glu = torch.empty((M, N), device="cuda")
    ops.gemm_simt(x, w, glu, ops.EPI_SWIGLU)
    gate, up = full[:, :N], full[:, N:]
    act = gate * torch.sigmoid(gate)                                      # |silu'| <= 1.1; a few roundings of the quotient
    assert ((glu.double() - act * up).abs() <= 1.1 * off[:, :N] * up.abs() + off[:, N:] * act.abs() + off[:, :N] * off[:, N:] + 2.0 ** -21 * (act * up).abs()).all()
    for rows in (slice(M - 1, M), slice(0, min(M, 20)), slice(0, min(M, 60))):      # the same bits alone, among a few and among all
        few = torch.empty((rows.stop - rows.start, N), device="cuda")
        ops.gemm_simt(x[rows].contiguous(), wn, few, ops.EPI_STORE_F32)
        assert torch.equal(few, out[rows])


def distances(x, w):
    """How far the product on the tensor cores and the one on the CUDA cores are from 64 bits: 2-norms and largest differences, over those of the result."""
    from borrowed_compute_b200 import ops

    full, off = x.double() @ w.double().T, []
    for cores in (False, True):
        out = torch.empty((x.shape[0], w.shape[0]), device="cuda")
        ops.gemm_simt(x, w, out, ops.EPI_STORE_F32, cores=cores)
        d = out.double() - full
        off += [(d.norm() / full.norm()).item(), (d.abs() / full.abs().clamp_min(1e-300)).max().item()]
    return off


@pytest.mark.parametrize("M,N,K", [(7, 128, 1024), (300, 256, 2048), (40, 200, 2048), (130, 128, 8192), (130, 12416, 8192), (20, 12416, 16384), (3, 12416, 32768)])
@pytest.mark.parametrize("values", ["normal", "uniform", "squares", "one sign"])
def test_no_further_from_64_bits_than_one_multiply_add_after_another(values, M, N, K):
    """Also where all products have one sign, so that truncated additions all err one way.  (12,416 weight rows: K in one piece.)"""
    x, w = operands(M, N, K, 1)
    if values == "uniform":
        x, w = torch.rand_like(x), torch.rand_like(w)
    if values == "squares":
        x = x.clamp_min(0.0).square()
    if values == "one sign":
        x, w = x.square(), w.abs()
    here, _, there, _ = distances(x, w)
    assert here <= there, (here, there)


@pytest.mark.parametrize("M", [40, 300])
@pytest.mark.parametrize("kept", [1, 2, 3, 4, 8, 16, 64])
def test_rows_of_few_numbers(M, kept):
    """What a sum of one or a few products loses to the parts that are left out: nothing that shows."""
    N, K = 256, 2048
    x, w = operands(M, N, K, 2)
    at = torch.rand(M, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(kept)).argsort(1)[:, :kept]
    few = torch.zeros_like(x).scatter_(1, at, x.gather(1, at))
    here, most, there, most_there = distances(few, w)
    # Beside the rounding of the result, 2^-24 of it, the smaller products' seven additions are truncated, at 2^-23 of 2^-6.
    assert here <= 1.01 * there, (here, there)
    if kept == 1:
        assert most <= 2.0 ** -24 + 2.0 ** -26 and most_there <= 2.0 ** -24, (most, most_there)


@pytest.mark.parametrize("M", [40, 130])
def test_numbers_at_the_ends_of_the_range(M):
    """Infinities and not-a-numbers reach every output of their row and column and no other; the largest floats and small ones keep their bits."""
    from borrowed_compute_b200 import ops

    N, K = 140, 1032
    inf, biggest = float("inf"), 3.4028234663852886e38
    x, w = torch.ones((M, K), device="cuda"), torch.ones((N, K), device="cuda")
    x[2, K - 1], x[3, 0], x[5, 7], w[9, 40] = inf, float("nan"), -inf, inf
    x[4, 1:] = 0.0
    x[4, 0], w[:, 0] = biggest, 1.0
    x[6], x[7, :] = 2.0 ** -100 * (1 + 2.0 ** -23), 0.0
    out = torch.empty((M, N), device="cuda")
    ops.gemm_simt(x, w, out, ops.EPI_STORE_F32)
    others = [n for n in range(N) if n != 9]
    assert (out[2] == inf).all() and out[3].isnan().all() and (out[5][others] == -inf).all() and out[5, 9].isnan()
    assert (out[4][others] == biggest).all() and out[4, 9].isnan()
    assert (out[[0, 1, 8]][:, others] == K).all() and (out[[0, 1, 8], 9] == inf).all()
    assert ((out[6][others].double() / (K * 2.0 ** -100 * (1 + 2.0 ** -23)) - 1).abs() <= bound(K)).all() and (out[7][others] == 0).all()
    # Results within a rounded first part of the largest float, and sums that are larger.
    x[8, 1:], x[9, 2:], w[20, :], w[20, 0] = 0.0, 0.0, 0.0, 2.0 ** 64
    x[8, 0], x[9, 0], x[9, 1], w[21, 1] = (2 - 2.0 ** -9) * 2.0 ** 63, biggest, biggest, 1.0
    ops.gemm_simt(x, w, out, ops.EPI_STORE_F32)
    assert out[8, 20] == (2 - 2.0 ** -9) * 2.0 ** 127 and (out[8][[n for n in others if n != 20]] == (2 - 2.0 ** -9) * 2.0 ** 63).all() and out[9, 21] == inf
    alone = torch.empty((1, N), device="cuda")
    ops.gemm_simt(x[8:9].contiguous(), w, alone, ops.EPI_STORE_F32)
    assert torch.equal(alone[0][others], out[8][others])
    # A payload below bfloat16's bits is still not a number.
    odd = torch.full((1, K), 1.0, device="cuda")
    odd.view(torch.int32)[0, 3] = 0x7F800001
    got = torch.empty((1, N), device="cuda")
    ops.gemm_simt(odd, w, got, ops.EPI_STORE_F32)
    assert got.isnan().all()


@pytest.mark.parametrize("M,N,K", [(1, 70, 1028), (40, 130, 516), (112, 64, 2100), (113, 130, 1028), (300, 64, 2100)])
@pytest.mark.parametrize("of_x,of_w", [(-108, 90), (-115, 100), (-125, 100), (-135, 110), (-147, 120), (110, -135), (100, -115), (-60, -60), (-70, -65), (-75, -70)])
def test_small_floats_are_whole(M, N, K, of_x, of_w):
    """Floats whose last bits bfloat16 does not reach, subnormal ones among them, and results down to the last bit of a float."""
    from borrowed_compute_b200 import ops

    x, w = operands(M, N, K, 3)
    x, w = x * 2.0 ** of_x, w * K ** 0.5 * 2.0 ** of_w
    out = torch.empty((M, N), device="cuda")
    ops.gemm_simt(x, w, out, ops.EPI_STORE_F32)
    full, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # Eight products of sixteen k and two additions a stretch may each drop what lies below 2^-149.
    assert ((out.double() - full).abs() <= bound(K) * size + (K / 2 + K / 32 + 8) * 2.0 ** -149).all()
    few = torch.empty((1, N), device="cuda")
    ops.gemm_simt(x[M - 1:].contiguous(), w, few, ops.EPI_STORE_F32)
    assert torch.equal(few, out[M - 1:])


@pytest.mark.parametrize("M", [40, 130])
def test_rows_with_small_floats_leave_the_others_alone(M):
    from borrowed_compute_b200 import ops

    N, K, inf = 200, 1032, float("inf")
    x, w = operands(M, N, K, 4)
    plain, gated = torch.empty((M, N), device="cuda"), torch.empty((M, N // 2), device="cuda")
    ops.gemm_simt(x, w, plain, ops.EPI_STORE_F32)
    x[3, 5], x[M - 1, K - 1], w[7, 600], w[150, 0] = 2.0 ** -149, 2.0 ** -120 * (1 + 2.0 ** -23), 2.0 ** -130 * 1.9, -2.0 ** -140
    x[9, 600], x[11, 2] = inf, inf
    w[8, 2], w[20, 2], w[21, 2], w[21, 1] = 2.0 ** -148, -2.0 ** -148, 0.0, 1.0
    out = torch.empty((M, N), device="cuda")
    ops.gemm_simt(x, w, out, ops.EPI_STORE_F32)
    rows, cols = [m for m in range(M) if m not in (3, 9, 11, M - 1)], [n for n in range(N) if n not in (7, 8, 20, 21, 150)]
    assert torch.equal(out[rows][:, cols], plain[rows][:, cols])
    full, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    near = (out.double() - full).abs() <= bound(K) * size
    assert (near | (out.double() == full) | (out.isnan() & full.isnan())).all()      # an infinity times a small float is one, times zero it is no number
    assert out[9, 7] == inf and out[11, 8] == inf and out[11, 20] == -inf and out[11, 21].isnan()
    ops.gemm_simt(x, w, gated, ops.EPI_SWIGLU)
    up = full[:, N // 2:]
    want = full[:, :N // 2] * torch.sigmoid(full[:, :N // 2]) * up
    assert (((gated.double() - want).abs() <= 2.0 ** -14 * (1 + size[:, :N // 2]) * (1 + up.abs())) | (gated.double() == want) | (gated.isnan() & want.isnan())).all()


def test_operands_that_tensor_copies_cannot_take_go_the_other_way():
    """K no multiple of four, or operands off their 16 bytes: the CUDA-core kernel, as before."""
    from borrowed_compute_b200 import ops

    for K, shift in ((1030, 0), (1032, 1)):
        x, w = operands(9, 70, K)
        room = torch.empty(9 * K + 4, device="cuda")
        moved = room[shift:shift + 9 * K].view(9, K)
        moved.copy_(x)
        out = torch.empty((9, 70), device="cuda")
        ops.gemm_simt(moved, w, out, ops.EPI_STORE_F32)
        size = x.double().abs() @ w.double().abs().T
        assert ((out.double() - x.double() @ w.double().T).abs() <= (K + 4) * 2.0 ** -24 * size).all()
