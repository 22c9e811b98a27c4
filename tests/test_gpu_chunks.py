"""The recurrences that take sixteen rows at a time (csrc/delta_chunks.cu, csrc/linear_chunks.cu) against float64 sums and against the row-by-row
scans they stand in for: sequences around the edges of a chunk, several beside one another and one of no slot, states that are not
zero, channel counts that fill a tile and that do not, scratch for the whole step and for one chunk a sequence at a time, decays at the
ends of their range, and an infinity that may reach later rows but no earlier one.

Tolerance: 32-bit sums over a chunk and a head (at most 16 + 256 terms) and their chain over a prompt that the decays forget, measured
at 2.5e-7 of a tensor's 2-norm at most; 2e-6 is allowed, and no value may be off by 2e-5 of the largest."""

from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEV = "cuda:0"


def i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def close(got, ref, what):
    got, ref = got.double().cpu().numpy(), ref.cpu().numpy()
    assert np.isfinite(got).all(), what
    assert np.linalg.norm(got - ref) <= 2e-6 * np.linalg.norm(ref), f"{what}: {np.linalg.norm(got - ref) / np.linalg.norm(ref):.3g}"
    assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max(), what


def batch(lens):
    """Row ranges and slots of sequences of these lengths, then one more of no slot over the last rows."""
    at = np.concatenate([[0], np.cumsum(lens)])
    return int(at[-1]), i32([int(a) for a in at]), i32([len(lens) - i for i in range(len(lens) - 1)] + [-1])


def draw(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return lambda *shape: torch.randn(*shape, generator=g, device=DEV)


@pytest.mark.parametrize("lens,heads,dim,inner,scale,segments", [
    ([1, 15, 16, 17, 5], 2, 64, 8, math.exp(-0.5), False), ([33, 47, 3], 3, 24, 12, math.exp(-0.5), True),
    ([130, 2], 1, 4, 4, 4.0, False), ([200, 64, 16], 2, 60, 40, 0.0, True)])
def test_delta_rule_in_chunks(lens, heads, dim, inner, scale, segments):
    from borrowed_compute_b200 import ops

    rnd, HD = draw(dim), heads * dim
    rows, seq_rows, seq_slot = batch(lens)
    proj, w2t, w0, a_b = 1.2 * rnd(rows, 5 * HD + inner), 0.5 * rnd(inner, HD), rnd(HD), 0.5 * rnd(HD)
    before = 0.3 * rnd(len(lens) + 1, heads, dim, dim)
    state, out, decay = before.clone(), torch.full((rows, HD), 7.0, device=DEV), torch.empty((rows, HD), device=DEV)
    need = ops.delta_chunked_scratch(rows, len(lens), heads, dim, inner, scale)
    assert need > 0
    chunk = 4 * 16 * 64 + 16 * 20 + 64
    pack = torch.full((len(lens) * heads * chunk if segments else need,), float("nan"), device=DEV)
    ops.delta_chunked(proj, w2t, w0, a_b, decay, pack, state, seq_rows, seq_slot, out, len(lens), max(lens), heads, dim, scale, 1e-6)
    P = proj.double()
    r, k, v, _, a = (P[:, i * HD:(i + 1) * HD].view(rows, heads, dim) for i in range(5))
    w = torch.exp(-scale * torch.sigmoid(torch.tanh(P[:, 5 * HD:]) @ w2t.double() + w0.double())).view(rows, heads, dim)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    b = torch.sigmoid(a.reshape(rows, HD) + a_b.double()).view(rows, heads, dim) * u
    want, after, at = torch.full((rows, heads, dim), 7.0, dtype=torch.float64, device=DEV), before.double(), 0
    for n, slot in zip(lens, seq_slot.tolist()):
        for t in range(at, at + n if slot >= 0 else at):
            S = after[slot].transpose(1, 2)
            S = w[t][..., None] * S - b[t][..., None] * torch.bmm(u[t][:, None], S) + k[t][..., None] * v[t][:, None]
            want[t] = torch.bmm(r[t][:, None], S)[:, 0]
            after[slot] = S.transpose(1, 2)
        at += n
    close(out, want.view(rows, HD), "outputs")
    close(state, after, "states")
    assert torch.equal(state[0], before[0]) and bool((out[rows - lens[-1]:] == 7.0).all()), "what belongs to no sequence was touched"


@pytest.mark.parametrize("lens,heads,keys,values,rank,tau,segments", [
    ([1, 15, 16, 17, 5], 2, 128, 64, 16, 16.0, False), ([33, 47, 3], 3, 24, 12, 4, 16.0, True), ([130, 2], 1, 256, 36, 20, 0.05, False),
    ([70, 64, 9], 2, 64, 32, 1, 1.0, True)])
def test_gated_linear_attention_in_chunks(lens, heads, keys, values, rank, tau, segments):
    from borrowed_compute_b200 import ops

    rnd, hd, hp = draw(keys), heads * keys, heads * values
    rows, seq_rows, seq_slot = batch(lens)
    inner_at = 2 * hd + 2 * hp
    proj, w2t, bias = rnd(rows, -(-(inner_at + rank) // 4) * 4), 0.5 * rnd(rank, hd), rnd(hd) - (2.0 if tau < 1 else 0.0)
    before = 0.3 * rnd(len(lens) + 1, heads, values, keys)
    state, out, f = before.clone(), torch.full((rows, hp), 7.0, device=DEV), keys ** -0.5
    need = ops.gla_chunked_scratch(proj, 2 * hd, len(lens), heads, keys, values, rank)
    assert need > 0
    wide = 64 if keys <= 64 else 128 if keys <= 128 else 256
    pack = torch.full((len(lens) * heads * (2 * 16 * wide + 16 * 20 + wide) if segments else need,), float("nan"), device=DEV)
    ops.gla_chunked(proj, 0, hd, 2 * hd, inner_at, w2t, bias, tau, f, pack, state, seq_rows, seq_slot, out, len(lens), max(lens), heads, keys, values)
    P = proj.double()
    q, k, v = f * P[:, :hd].view(rows, heads, keys), P[:, hd:2 * hd].view(rows, heads, keys), P[:, 2 * hd:2 * hd + hp].view(rows, heads, values)
    z = P[:, inner_at:inner_at + rank] @ w2t.double() + bias.double()
    a = torch.exp(torch.nn.functional.logsigmoid(z) / tau).view(rows, heads, keys)        # down to exp(-100) a row at tau 0.05
    want, after, at = torch.full((rows, heads, values), 7.0, dtype=torch.float64, device=DEV), before.double(), 0
    for n, slot in zip(lens, seq_slot.tolist()):
        for t in range(at, at + n if slot >= 0 else at):
            S = a[t][..., None] * after[slot].transpose(1, 2) + k[t][..., None] * v[t][:, None]
            want[t] = torch.bmm(q[t][:, None], S)[:, 0]
            after[slot] = S.transpose(1, 2)
        at += n
    close(out, want.view(rows, hp), "outputs")
    close(state, after, "states")
    assert torch.equal(state[0], before[0]) and bool((out[rows - lens[-1]:] == 7.0).all()), "what belongs to no sequence was touched"


def test_what_the_chunks_do_not_take_and_what_is_too_small():
    from borrowed_compute_b200 import ops

    assert ops.delta_chunked_scratch(64, 1, 2, 68, 8, 0.6) == 0 and ops.delta_chunked_scratch(64, 1, 2, 64, 8, 4.5) == 0        # wide heads, small decays
    assert ops.delta_chunked_scratch(64, 1, 2, 24, 5, 0.6) == 0                                                               # rows off a 16-byte border
    proj = torch.zeros((64, 5 * 128 + 8), device=DEV)
    state, out = torch.zeros((1, 2, 64, 64), device=DEV), torch.zeros((64, 128), device=DEV)
    with pytest.raises(ops.KernelError):
        ops.delta_chunked(proj, torch.zeros((8, 128), device=DEV), torch.zeros(128, device=DEV), torch.zeros(128, device=DEV), torch.empty_like(out),
                          torch.empty(64, device=DEV), state, i32([0, 64]), i32([0]), out, 1, 64, 2, 64, 0.6, 1e-6)


@pytest.mark.parametrize("kind", ["delta", "linear"])
def test_an_infinity_reaches_no_earlier_row(kind):
    from borrowed_compute_b200 import ops

    rnd, H, D, rows, bad = draw(3), 2, 64, 40, 21
    HD = H * D
    seq_rows, seq_slot = i32([0, rows]), i32([0])
    clean, poisoned = torch.zeros((rows, HD), device=DEV), torch.zeros((rows, HD), device=DEV)
    proj = rnd(rows, 5 * HD + 8)
    for out, value in ((clean, None), (poisoned, float("inf"))):
        p, state = proj.clone(), torch.zeros((1, H, D, D), device=DEV)
        if value is not None:
            p[bad, 2 * HD:3 * HD] = value                   # a row of values
        if kind == "delta":
            w2t, zero = 0.5 * draw(4)(8, HD), torch.zeros(HD, device=DEV)
            pack = torch.empty((ops.delta_chunked_scratch(rows, 1, H, D, 8, 0.6),), device=DEV)
            ops.delta_chunked(p, w2t, zero, zero, torch.empty_like(out), pack, state, seq_rows, seq_slot, out, 1, rows, H, D, 0.6, 1e-6)
        else:
            w2t, zero = 0.5 * draw(4)(8, HD), torch.zeros(HD, device=DEV)
            pack = torch.empty((ops.gla_chunked_scratch(p, 2 * HD, 1, H, D, D, 8),), device=DEV)
            ops.gla_chunked(p, 0, HD, 2 * HD, 5 * HD, w2t, zero, 16.0, 0.125, pack, state, seq_rows, seq_slot, out, 1, rows, H, D, D)
    assert torch.equal(clean[:bad], poisoned[:bad])
    assert not bool(torch.isfinite(poisoned[bad:]).all(-1).any())
