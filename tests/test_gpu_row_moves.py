"""Kernels that move rows sixteen bytes at a time where sizes and addresses allow it, and by the value elsewhere: the latents' heads and
gathered pages, a bias added to rows.

Tolerance: copies and single additions are exact; a rotated value has two products and an addition in float (2^-22 of the head's
largest) and is rounded to bf16 once (2^-9, 2^-8 allowed)."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEV = "cuda:0"


def i32(a):
    return torch.tensor(a, dtype=torch.int32, device=DEV)


def draw(seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return lambda *shape: torch.randn(*shape, generator=gen, device=DEV)


@pytest.mark.parametrize("heads,dim,rot,padded", [(1, 8, 0, 64), (3, 64, 64, 128), (17, 16, 16, 64), (5, 40, 24, 64), (2, 12, 4, 16), (7, 56, 8, 64), (4, 96, 32, 128)])
def test_heads_with_their_rotated_part(heads, dim, rot, padded):
    from borrowed_compute_b200 import ops

    rnd, rows = draw(dim + rot), 37
    q = rnd(rows, heads * (dim + rot))
    pos = [(5 * i) % 90 for i in range(rows)]
    angles = torch.arange(90, device=DEV)[:, None] * 100.0 ** (-2.0 * torch.arange(max(rot // 2, 1), device=DEV) / max(rot, 1))
    cos_sin = torch.stack([angles.cos(), angles.sin()], -1).float().contiguous()
    for shift in (0, 1):                       # a query that starts off a 16-byte border
        held = torch.empty(q.numel() + 1, device=DEV)
        mine = held[shift:shift + q.numel()].view(q.shape).copy_(q)
        out = torch.full((rows, heads, padded), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.latent_heads(mine, cos_sin if rot else None, i32(pos), out, heads, dim, rot)
        x = q.double().view(rows, heads, dim + rot)
        ref = torch.zeros(rows, heads, padded, dtype=torch.float64, device=DEV)
        ref[..., :dim + rot] = x
        if rot:
            c, s = (cos_sin[pos][:, None, :, i].double() for i in (0, 1))
            a, b = x[..., dim:dim + rot // 2], x[..., dim + rot // 2:]
            ref[..., dim:dim + rot // 2], ref[..., dim + rot // 2:dim + rot] = a * c - b * s, b * c + a * s
        assert torch.equal(out[..., :dim], ref[..., :dim].bfloat16()) and (out[..., dim + rot:] == 0).all()
        assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -22 * x.abs().max()).all()


@pytest.mark.parametrize("R,rot", [(8, 0), (512, 64), (40, 8), (136, 24)])
def test_gathered_pages(R, rot):
    from borrowed_compute_b200 import ops

    rnd = draw(R)
    c, r = rnd(4, 64, R).bfloat16(), rnd(4, 64, rot).bfloat16() if rot else None
    table = i32([[2, 0, -1], [3, -1, 9]])                                     # (page 9 is none of the pool)
    slot, at, last = [0, 0, 0, 1, 1, -1, 0, 1], [0, 64, 128, 0, 128, 0, 64, 0], [200, 200, 200, 17, 150, 63, 64, 6]
    out_c = torch.full((len(slot) * 64, R), 9.0, dtype=torch.bfloat16, device=DEV)
    out_r = torch.full((len(slot) * 64, max(rot, 1)), 9.0, dtype=torch.bfloat16, device=DEV)
    ops.latent_gather(c, r, table, i32(slot), i32(at), i32(last), out_c, out_r if rot else None, len(slot))
    for p, (s, a, n) in enumerate(zip(slot, at, last)):
        page = int(table[s, a // 64]) if s >= 0 else -1
        held = max(0, min(64, n - a + 1)) if 0 <= page < 4 else 0
        for src, out in ((c, out_c), (r, out_r)):
            if src is None:
                continue
            rows = out[p * 64:(p + 1) * 64]
            assert (held == 0 or torch.equal(rows[:held], src[page, :held])) and (rows[held:] == 0).all(), p


@pytest.mark.parametrize("rows,E", [(1, 1), (7, 3), (8, 4), (9, 1024), (17, 1028), (300, 4096), (5, 1027), (2049, 1), (3000, 5), (1025, 8), (70, 130), (3, 256), (2, 257),
                                    (524299, 3)])
def test_bias_added_to_rows(rows, E):
    from borrowed_compute_b200 import ops

    rnd = draw(rows + E)
    x, b = rnd(rows, E), rnd(E)
    for shift in (0, 1):                       # rows that start off a 16-byte border
        held = torch.full((x.numel() + 2,), 4.0, device=DEV)
        mine = held[shift:shift + x.numel()].view(x.shape).copy_(x)
        ops.add_bias(mine, b)
        assert torch.equal(mine, x + b)
        assert (held[:shift] == 4.0).all() and (held[shift + x.numel():] == 4.0).all()


def test_bias_added_to_as_many_rows_as_an_int_counts():
    from borrowed_compute_b200 import ops

    x = torch.zeros((2 ** 31 - 1, 1), device=DEV)
    ops.add_bias(x, torch.ones(1, device=DEV))
    low, high = torch.aminmax(x)
    assert low == 1.0 and high == 1.0


def test_bias_of_rows_that_no_tile_divides_is_added_as_fast_as_the_others():
    """Narrow and unaligned rows take no longer than an element a thread takes (an elementwise product over the same bytes, three times over)."""
    from borrowed_compute_b200 import ops

    def micros(run):
        times = []
        for _ in range(12):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            for _ in range(10):
                run()
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end) * 100.0)
        return sorted(times)[3]

    for rows, E in ((500000, 16), (500000, 13), (20480, 1023)):
        x, b = torch.zeros((rows, E), device=DEV), torch.ones(E, device=DEV)
        mine, plain = micros(lambda: ops.add_bias(x, b)), micros(lambda: ops.scale_scores(x, 1.0))
        assert mine <= 2.0 * plain, (rows, E, mine, plain)
