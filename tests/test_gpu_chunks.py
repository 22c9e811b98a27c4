"""The recurrences that take sixteen rows at a time (csrc/delta_chunks.cu, csrc/linear_chunks.cu) against float64 sums and against the row-by-row
scans they stand in for: sequences around the edges of a chunk, several beside one another and one of no slot, states that are not
zero, channel counts that fill a tile and that do not, scratch for the whole step and for one chunk a sequence at a time, decays at the
ends of their range, an infinity that may reach later rows but no earlier one, and steps in which short sequences go row by row beside long
ones in chunks.

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


MIXED = [[1, 40, 3, 16, 15, 2, 100, 1, 9], [33, 1], [1] * 40 + [16, 17] + [2] * 30 + [50, 4]]      # (the last: more sequences than places by sequence are worth)


def delta_args(lens, seed, H=2, D=64, inner=8):
    rnd, HD = draw(seed), H * D
    rows, seq_rows, seq_slot = batch(lens)
    return dict(rows=rows, H=H, D=D, HD=HD, inner=inner, seq_rows=seq_rows, seq_slot=seq_slot, seqs=len(lens), longest=max(lens), proj=1.2 * rnd(rows, 5 * HD + inner),
                w2t=0.5 * rnd(inner, HD), w0=rnd(HD), a_b=0.5 * rnd(HD), state=0.3 * rnd(len(lens) + 1, H, D, D))


def delta_run(a, chunks=None, below=None, pack_chunks=None, write_state=True):
    """(outputs, states) of the chunked path over sequences of at least ``chunks`` rows, the row by row path over those below ``below``."""
    from borrowed_compute_b200 import ops

    state, out = a["state"].clone(), torch.full((a["rows"], a["HD"]), 7.0, device=DEV)
    decay, unit, removal = (torch.full((a["rows"], a["HD"]), float("nan"), device=DEV) for _ in range(3))
    dots = torch.full((a["rows"], a["H"], 2), float("nan"), device=DEV)
    if chunks is not None:
        need = ops.delta_chunked_scratch(a["rows"], a["seqs"], a["H"], a["D"], a["inner"], 0.6, write_state, min_rows=chunks)
        assert need > 0
        if pack_chunks is not None:
            need = pack_chunks * a["seqs"] * a["H"] * (4 * 16 * 64 + 16 * 20 + 64)
        pack = torch.full((need,), float("nan"), device=DEV)
        ops.delta_chunked(a["proj"], a["w2t"], a["w0"], a["a_b"], decay, pack, state, a["seq_rows"], a["seq_slot"], out, a["seqs"], a["longest"], a["H"], a["D"],
                          0.6, 1e-6, write_state=write_state, min_rows=chunks)
    if below is not None:
        ops.delta_prepare(a["proj"], a["w2t"], a["w0"], a["a_b"], decay, unit, removal, dots, a["H"], a["D"], 0.6, 1e-6, a["seq_rows"], a["seqs"], below)
        ops.delta_scan(a["proj"], decay, unit, removal, dots, state, a["seq_rows"], a["seq_slot"], out, a["seqs"], a["H"], a["D"], write_state=write_state, below=below)
    return out, state


def linear_args(lens, seed, H=2, N=24, P=36, rank=8):
    rnd, hd, hp = draw(seed), H * N, H * P
    rows, seq_rows, seq_slot = batch(lens)
    return dict(rows=rows, H=H, N=N, P=P, hd=hd, hp=hp, rank=rank, seq_rows=seq_rows, seq_slot=seq_slot, seqs=len(lens), longest=max(lens),
                proj=rnd(rows, 2 * hd + 2 * hp + rank), w2t=0.5 * rnd(rank, hd), bias=rnd(hd), state=0.3 * rnd(len(lens) + 1, H, P, N))


def linear_run(a, chunks=None, below=None, pack_chunks=None, write_state=True):
    from borrowed_compute_b200 import ops

    H, N, P, hd, hp = (a[k] for k in ("H", "N", "P", "hd", "hp"))
    state, out, decay = a["state"].clone(), torch.full((a["rows"], hp), 7.0, device=DEV), torch.full((a["rows"], hd), float("nan"), device=DEV)
    proj, inner_at = a["proj"], 2 * hd + 2 * hp
    if chunks is not None:
        need = ops.gla_chunked_scratch(proj, 2 * hd, a["seqs"], H, N, P, a["rank"], write_state, min_rows=chunks)
        assert need > 0
        if pack_chunks is not None:
            need = pack_chunks * a["seqs"] * H * (2 * 16 * 64 + 16 * 20 + 64)
        pack = torch.full((need,), float("nan"), device=DEV)
        ops.gla_chunked(proj, 0, hd, 2 * hd, inner_at, a["w2t"], a["bias"], 16.0, 0.2, pack, state, a["seq_rows"], a["seq_slot"], out, a["seqs"], a["longest"], H, N, P,
                        write_state=write_state, min_rows=chunks)
    if below is not None:
        ops.gla_decay(proj, inner_at, a["w2t"], a["bias"], decay, 16.0, a["seq_rows"], a["seqs"], below)
        ops.linear_scan(proj, 0, 1, proj, hd, 1, proj, 2 * hd, decay, 0, True, None, 0, None, 0.2, state, a["seq_rows"], a["seq_slot"], out, a["seqs"], H, N, P,
                        write_state=write_state, below=below)
    return out, state


@pytest.mark.parametrize("kind", ["delta", "linear"])
@pytest.mark.parametrize("lens", MIXED, ids=["few", "two", "many"])
def test_each_sequence_goes_by_its_own_rows(lens, kind):
    args, run = (delta_args, delta_run) if kind == "delta" else (linear_args, linear_run)
    a = args(lens, 11)
    chunked, scanned, nothing = run(a, chunks=0), run(a, below=10 ** 9), a["state"]
    both, long, short = run(a, chunks=16, below=16), run(a, chunks=16), run(a, below=16)
    small = run(a, chunks=16, below=16, pack_chunks=2)             # two chunks a sequence at a time
    at = 0
    for n, slot in zip(lens, a["seq_slot"].tolist()):
        rows = slice(at, at + n)
        at += n
        if slot < 0:
            assert all(bool((o[rows] == 7.0).all()) for o, _ in (both, long, short, small))
            continue
        want = chunked if n >= 16 else scanned
        for got in (both, small, long if n >= 16 else short):
            assert torch.equal(got[0][rows], want[0][rows]) and torch.equal(got[1][slot], want[1][slot]), (n, slot)
        other = short if n >= 16 else long
        assert bool((other[0][rows] == 7.0).all()) and torch.equal(other[1][slot], nothing[slot]), (n, slot)


@pytest.mark.parametrize("kind", ["delta", "linear"])
def test_a_short_sequence_beside_a_long_one_has_the_bits_it_has_alone(kind):
    """A part on bfloat16 rows.  Its matrices hold small whole numbers and its last one is the identity, so that the products are exact
    however many rows share them."""
    from borrowed_compute_b200.cache import PagedCache
    from borrowed_compute_b200.engine import StepEntry, plan_step
    from borrowed_compute_b200.parts import MIXERS, Runtime, StepContext

    H, D, E, rank = 2, 64, 128, 8
    part = MIXERS.get("generalized_delta")(hidden_size=E, heads=H, head_dim=D, decay_rank=rank, norm_eps=1e-5) if kind == "delta" else \
        MIXERS.get("gated_linear_attention")(hidden_size=E, heads=H, head_dim=D, value_dim=D, decay_rank=rank, tau=16.0, norm_eps=1e-5)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(5)
    weights = {}
    for name, spec in part.tensors().items():
        t = torch.randint(-1, 2, spec.shape, generator=gen, device=DEV).float() / 8.0
        weights[name] = torch.eye(E, device=DEV).bfloat16() if name == "o" else t if spec.role == "vector" else t.bfloat16()
    lens = [5, 70, 1, 16, 15]
    x = torch.randint(-1, 2, (sum(lens), E), generator=gen, device=DEV).bfloat16()
    rt = Runtime(torch.device(DEV), torch.bfloat16, max_positions=128)
    part.load(weights, rt)

    def run(which):
        n = [lens[i] for i in which]
        cache = PagedCache(rt, [part.cache_need()], [part.state_need()], [None], max_tokens=64 * 2 * len(n), n_slots=len(n), max_seq=128)
        slots = [cache.acquire() for _ in n]
        cache.slots.reserve_many([(slot, k, k) for slot, k in zip(slots, n)])
        cache.sync_tables()
        plan = plan_step([StepEntry(slot, [0] * k) for slot, k in zip(slots, n)], [0] * len(n))
        dev = lambda v: torch.from_numpy(v).to(DEV)       # noqa: E731
        ctx = StepContext(rows=plan.rows, seqs=plan.seqs, tokens=dev(plan.tokens), row_pos=dev(plan.row_pos), row_slot=dev(plan.row_slot), seq_rows=dev(plan.seq_rows),
                          seq_slot=dev(plan.seq_slot), seq_start=dev(plan.seq_start), max_new=plan.max_new, max_total=plan.max_total, decode=plan.decode,
                          host_seq_rows=tuple(int(v) for v in plan.seq_rows), host_seq_slot=tuple(int(v) for v in plan.seq_slot),
                          host_seq_start=tuple(int(v) for v in plan.seq_start))
        at = [sum(lens[:i]) for i in which]
        rows = torch.cat([x[a:a + k] for a, k in zip(at, n)])
        out, mem = torch.zeros(rows.shape, device=DEV), cache.memory(0)
        mem.state.zero_()
        part.forward(rows, out, ctx, mem)
        return list(out.split(n)), [mem.state[slot].clone() for slot in slots]

    outs, states = run(range(len(lens)))
    for i in range(len(lens)):
        (out,), (state,) = run([i])
        assert torch.equal(out, outs[i]) and torch.equal(state, states[i]), lens[i]


def test_an_infinity_leaves_with_its_own_chunk():
    """A last chunk of four rows takes the place of an earlier one that held an infinite value: the state keeps the sign it gave."""
    a = linear_args([52, 1], 14)
    a["proj"][8, 2 * a["hd"] + 3] = float("inf")                    # value channel 3 of head 0
    (_, chunked), (_, scanned) = linear_run(a, chunks=0), linear_run(a, below=10 ** 9)
    assert bool(torch.isinf(scanned[2, 0, 3]).all())
    assert torch.equal(chunked[2, 0, 3], scanned[2, 0, 3])
    chunked[2, 0, 3] = scanned[2, 0, 3] = 0.0
    assert torch.allclose(chunked, scanned, rtol=1e-4, atol=1e-5)


def distance(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("scale", [0.1, math.exp(-0.5), 4.0])
def test_delta_chunks_are_no_further_from_64_bit_sums_than_the_scan(scale):
    """Four seeds of 256 rows of eight heads; 5 % is left to chance."""
    from borrowed_compute_b200 import ops

    T, H, D, inner = 256, 8, 64, 32
    HD, sums = H * D, {}
    for seed in range(4):
        rnd = draw(100 + seed)
        proj, w2t, w0, a_b, before = rnd(T, 5 * HD + inner), rnd(inner, HD) / inner ** 0.5, rnd(HD), 0.5 * rnd(HD), 0.3 * rnd(1, H, D, D)
        P = proj.double()
        r, k, v, _, a = (P[:, i * HD:(i + 1) * HD].view(T, H, D) for i in range(5))
        w = torch.exp(-scale * torch.sigmoid(torch.tanh(P[:, 5 * HD:]) @ w2t.double() + w0.double())).view(T, H, D)
        u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        b = torch.sigmoid(a.reshape(T, HD) + a_b.double()).view(T, H, D) * u
        want, S = torch.empty(T, H, D, dtype=torch.float64, device=DEV), before[0].double().transpose(1, 2)
        for t in range(T):
            S = w[t][..., None] * S - b[t][..., None] * torch.bmm(u[t][:, None], S) + k[t][..., None] * v[t][:, None]
            want[t] = torch.bmm(r[t][:, None], S)[:, 0]
        for way in ("scan", "chunks"):
            state, out, decay, unit, removal = before.clone(), *(torch.empty((T, HD), device=DEV) for _ in range(4))
            if way == "scan":
                dots = torch.empty((T, H, 2), device=DEV)
                ops.delta_prepare(proj, w2t, w0, a_b, decay, unit, removal, dots, H, D, scale, 1e-6)
                ops.delta_scan(proj, decay, unit, removal, dots, state, i32([0, T]), i32([0]), out, 1, H, D)
            else:
                pack = torch.empty((ops.delta_chunked_scratch(T, 1, H, D, inner, scale),), device=DEV)
                ops.delta_chunked(proj, w2t, w0, a_b, decay, pack, state, i32([0, T]), i32([0]), out, 1, T, H, D, scale, 1e-6)
            for what, value in (("outputs", distance(out, want.view(T, HD))), ("state", distance(state[0], S.transpose(1, 2)))):
                sums[way, what] = sums.get((way, what), 0.0) + value ** 2
    for what in ("outputs", "state"):
        assert sums["chunks", what] <= 1.05 ** 2 * sums["scan", what], (what, sums)


@pytest.mark.parametrize("tau", [1.0, 16.0, 100.0])
def test_linear_chunks_are_no_further_from_64_bit_sums_than_the_scan(tau):
    from borrowed_compute_b200 import ops

    T, H, N, P, rank = 256, 4, 128, 64, 16
    hd, hp, f, sums = H * N, H * P, N ** -0.5, {}
    for seed in range(4):
        rnd = draw(200 + seed)
        proj, w2t, bias, before = rnd(T, 2 * hd + 2 * hp + rank), rnd(rank, hd) / rank ** 0.5, rnd(hd), 0.3 * rnd(1, H, P, N)
        p = proj.double()
        q, k, v = f * p[:, :hd].view(T, H, N), p[:, hd:2 * hd].view(T, H, N), p[:, 2 * hd:2 * hd + hp].view(T, H, P)
        a = torch.exp(torch.nn.functional.logsigmoid(p[:, 2 * hd + 2 * hp:] @ w2t.double() + bias.double()) / tau).view(T, H, N)
        want, S = torch.empty(T, H, P, dtype=torch.float64, device=DEV), before[0].double().transpose(1, 2)
        for t in range(T):
            S = a[t][..., None] * S + k[t][..., None] * v[t][:, None]
            want[t] = torch.bmm(q[t][:, None], S)[:, 0]
        for way in ("scan", "chunks"):
            state, out = before.clone(), torch.empty((T, hp), device=DEV)
            if way == "scan":
                decay = torch.empty((T, hd), device=DEV)
                ops.gla_decay(proj, 2 * hd + 2 * hp, w2t, bias, decay, tau)
                ops.linear_scan(proj, 0, 1, proj, hd, 1, proj, 2 * hd, decay, 0, True, None, 0, None, f, state, i32([0, T]), i32([0]), out, 1, H, N, P)
            else:
                pack = torch.empty((ops.gla_chunked_scratch(proj, 2 * hd, 1, H, N, P, rank),), device=DEV)
                ops.gla_chunked(proj, 0, hd, 2 * hd, 2 * hd + 2 * hp, w2t, bias, tau, f, pack, state, i32([0, T]), i32([0]), out, 1, T, H, N, P)
            for what, value in (("outputs", distance(out, want.view(T, hp))), ("state", distance(state[0], S.transpose(1, 2)))):
                sums[way, what] = sums.get((way, what), 0.0) + value ** 2
    for what in ("outputs", "state"):
        assert sums["chunks", what] <= 1.05 ** 2 * sums["scan", what], (what, sums)


@pytest.mark.parametrize("kind", ["delta", "linear"])
@pytest.mark.parametrize("pack_chunks", [None, 4, 5])
def test_segments_of_several_chunks(kind, pack_chunks):
    """A pack that holds four or five chunks a sequence: the same bits as with all of them at once."""
    args, run = (delta_args, delta_run) if kind == "delta" else (linear_args, linear_run)
    a = args([150, 64, 65, 3], 12)
    whole, got = run(a, chunks=0), run(a, chunks=0, pack_chunks=pack_chunks)
    assert all(torch.equal(x, y) for x, y in zip(whole, got))


@pytest.mark.parametrize("kind", ["delta", "linear"])
def test_a_state_that_is_only_read(kind):
    from borrowed_compute_b200 import ops

    args, run = (delta_args, delta_run) if kind == "delta" else (linear_args, linear_run)
    a = args([50, 17, 16, 3], 13)
    writing, reading = run(a, chunks=16, below=16), run(a, chunks=16, below=16, write_state=False)
    assert torch.equal(writing[0], reading[0]) and torch.equal(reading[1], a["state"]) and not torch.equal(writing[1], a["state"])
    with pytest.raises(ops.KernelError):             # segments hand the state on through memory
        run(a, chunks=0, pack_chunks=1, write_state=False)
    many = 10 ** 6                                   # rows whose packs are past what a step is given
    if kind == "delta":
        assert ops.delta_chunked_scratch(many, 1, 64, 64, 64, 0.6, False) == 0 < ops.delta_chunked_scratch(many, 1, 64, 64, 64, 0.6, True) <= 2 ** 28
    else:
        proj = torch.empty((0, 64), device=DEV).expand(0, 64)
        big = torch.empty((1, 64), device=DEV).expand(many, 64)
        assert ops.gla_chunked_scratch(proj, 0, 1, 64, 256, 4, 4, False) > 0
        assert ops.gla_chunked_scratch(big, 0, 1, 64, 256, 4, 4, False) == 0 < ops.gla_chunked_scratch(big, 0, 1, 64, 256, 4, 4, True) <= 2 ** 28
