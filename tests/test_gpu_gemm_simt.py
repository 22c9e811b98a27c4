"""The CUDA-core product (``cores``: also where float32 sums go to the tensor cores by themselves) where its kernels change over: short sums of few outputs, tiles of 16 and of 64 rows, sums over K in one
piece and in clusters of two to eight, widths with and without 16-byte loads.

Tolerance: a float sum of K products in any order is off by at most K 2^-24 sum |x w| (plus the roundings of what follows it)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [
    (1, 1, 1), (5, 33, 7), (17, 31, 144), (16, 64, 176), (128, 512, 512), (3, 70, 511), (512, 512, 512), (2048, 128, 64),   # short sums; 262,144 outputs are the most they take
    (513, 512, 512), (129, 2050, 40),                                                         # one more, in tiles
    (1, 40, 1030), (32, 129, 1030), (33, 129, 1030), (65, 64, 2051), (70, 127, 4100),         # two, four and eight pieces
    (300, 130, 1024), (48, 2048, 2048), (96, 2048, 2048), (128, 512, 1024)])
def test_products_around_the_edges_of_their_kernels(dtype, M, N, K):
    from borrowed_compute_b200 import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    w = (torch.randn(2 * N, K, generator=g, device="cuda") / K ** 0.5).to(dtype)
    full, bound = x.double() @ w.double().T, (K + 4) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    wn = w[:N].contiguous()
    out = torch.full((M, N), float("nan"), device="cuda")
    ops.gemm_simt(x, wn, out, ops.EPI_STORE_F32, cores=True)
    assert ((out.double() - full[:, :N]).abs() <= bound[:, :N]).all()
    base = torch.randn(M, N, generator=g, device="cuda")
    acc = base.clone()
    ops.gemm_simt(x, wn, acc, ops.EPI_ADD_F32, cores=True)
    ref = base.double() + full[:, :N]
    assert ((acc.double() - ref).abs() <= bound[:, :N] + 2.0 ** -23 * ref.abs()).all()
    glu = torch.empty((M, N), dtype=dtype, device="cuda")
    ops.gemm_simt(x, w, glu, ops.EPI_SWIGLU, cores=True)
    gate, up = full[:, :N], full[:, N:]
    act = gate * torch.sigmoid(gate)
    unit = 2.0 ** -21 if dtype == torch.float32 else 2.0 ** -8                                 # the quotient's few roundings, or bf16's one
    # |silu'| <= 1.1
    assert ((glu.double() - act * up).abs() <= 1.1 * bound[:, :N] * up.abs() + bound[:, N:] * act.abs() + bound[:, :N] * bound[:, N:]
            + unit * (act * up).abs() + 1e-30).all()
    # A row alone, and a few of them, give the bits that they give among all.
    for rows in (slice(M - 1, M), slice(0, min(M, 20)), slice(0, min(M, 60))):
        few = torch.empty((rows.stop - rows.start, N), device="cuda")
        ops.gemm_simt(x[rows].contiguous(), wn, few, ops.EPI_STORE_F32, cores=True)
        assert torch.equal(few, out[rows])


def test_an_infinity_stays_in_its_row():
    from borrowed_compute_b200 import ops

    for M, N, K in ((5, 33, 70), (40, 140, 1030), (70, 140, 520), (5, 140, 1032)):
        x, w = torch.ones((M, K), device="cuda"), torch.ones((N, K), device="cuda")
        x[2, K - 1], x[3, 0] = float("inf"), float("nan")
        out = torch.empty((M, N), device="cuda")
        ops.gemm_simt(x, w, out, ops.EPI_STORE_F32, cores=True)
        assert torch.isinf(out[2]).all() and torch.isnan(out[3]).all()
        assert (out[[0, 1, 4]] == K).all() and np.isfinite(out[4:].cpu().numpy()).all()


@pytest.mark.parametrize("epilogue", ["store", "glu"])
@pytest.mark.parametrize("M,N,K,cores", [(1, 64, 64, True), (16, 512, 512, True), (70, 130, 520, True), (70, 130, 520, False), (130, 130, 1032, False)])
def test_a_matrix_that_the_kernel_before_has_just_written(M, N, K, cores, epilogue):
    """Kernels may start while the one before still runs; no operand is read before that one's end.  Sums of ones: exact."""
    from borrowed_compute_b200 import ops

    glu = epilogue == "glu"
    x, w = torch.full((M, K), 2.0 ** -10, device="cuda"), torch.ones((2 * N if glu else N, K), device="cuda")
    outs = [torch.empty((M, N), device="cuda") for _ in range(12)]
    for out in outs:
        ops.scale_scores(w, 2.0)
        ops.gemm_simt(x, w, out, ops.EPI_SWIGLU if glu else ops.EPI_STORE_F32, cores=cores)
    for i, out in enumerate(outs):
        s = K * 2.0 ** (i + 1 - 10)
        want = s * s / (1.0 + np.exp(-s)) if glu else s
        assert ((out.double() - want).abs() <= (2.0 ** -20 if glu else 0.0) * want).all(), i
