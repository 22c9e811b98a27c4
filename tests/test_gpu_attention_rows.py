"""The row attention kernel at head sizes on both sides of every width it is compiled for, and at numbers of positions around the
eight (or four) it fetches values for at once, its tiles of 32 and a page.

Tolerance: float sums of D products and of n weights that add up to one, against float64: (D + n + 16) 2^-24 of the largest value
times the largest score's size; 2e-5 allows for scores up to about 10.  bfloat16 operands are exact in float; the result is rounded once, by at most 2^-8 of it (half of its last place)."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [4, 32, 33, 64, 65, 128, 129, 256])
def test_row_attention_at_every_width(D, dtype):
    from borrowed_compute_b200 import ops

    H, G, lens = 4, 2, [1, 3, 4, 5, 7, 8, 9, 31, 32, 33, 40, 63, 64, 65, 130]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(D)
    pages = sum(-(-n // 64) for n in lens)
    k, v = (torch.randn(pages, G, 64, D, generator=gen, device="cuda").to(dtype) for _ in range(2))
    table = torch.full((len(lens), 3), -1, dtype=torch.int32)
    at, refs = 0, []
    q = torch.randn(len(lens), H * D, generator=gen, device="cuda").to(dtype)
    for i, n in enumerate(lens):
        ids = list(range(at, at - (-n // 64)))
        table[i, :len(ids)] = torch.tensor(ids)
        at += len(ids)
        kk, vv = (t[ids].permute(1, 0, 2, 3).reshape(G, -1, D)[:, :n].double().repeat_interleave(H // G, 0) for t in (k, v))
        p = torch.softmax(torch.einsum("hd,hnd->hn", q[i].view(H, D).double(), kk) * D ** -0.5, -1)
        refs.append(torch.einsum("hn,hnd->hd", p, vv).reshape(-1))
        k[ids[-1], :, (n - 1) % 64 + 1:] = float("nan")
        v[ids[-1], :, (n - 1) % 64 + 1:] = float("nan")
    out = torch.empty(len(lens), H * D, dtype=dtype, device="cuda")
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")     # noqa: E731
    ops.attention_rows(q, H * D, k, v, table.cuda(), i32([n - 1 for n in lens]), i32(list(range(len(lens)))), out, H, G, D, 0, D ** -0.5)
    ref = torch.stack(refs)
    assert ((out.double() - ref).abs() <= 2e-5 + (0.0 if dtype == torch.float32 else 2.0 ** -8) * ref.abs()).all()
