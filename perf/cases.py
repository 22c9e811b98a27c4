"""The work that programs have this framework do, as cases to be timed and compared.

Whole calls go through ``Engine``: token ids in, scores out.  Everything else is one mixer or one feed-forward of a layer, through the
interface that every part has (``forward`` on the rows of a step, with the cache's memory for that layer), the same call that the
engine's blocks make.  A case is a dict of plain values; ``kind`` says which path it takes:

    replay     Engine: prompts of unequal lengths in one step, then single tokens; scores of every step (a whole request)
    decode     Engine: single tokens of several sequences whose prompts are already in the cache, then cut back to where they were
    attention  grouped-query attention of the Llama decoder on prompts (rotation, cache, causal attention, both products)
    mlp        the gated feed-forward of the Llama decoder
    experts    a feed-forward of routed experts beside a shared one
    delta      the generalized delta rule on prompts
    linear     gated linear attention on prompts
    talking    attention whose heads talk, with a window that keeps the first positions, on prompts
    latent     latent attention with sinks and a rotated part, on prompts

Weights, activations and token ids are drawn on the device from the seed.  Matrices have rows of norm about one, so that what leaves a
product is about as large as what entered it; inputs of parts are what a norm leaves, about one a value.  Prompts of unequal lengths
are spread over ``shortest`` to ``longest``.  ``exact`` computes the same in float64 with plain torch.
"""

import dataclasses
import math
import random

import torch

from borrowed_compute_b200.cache import PagedCache
from borrowed_compute_b200.engine import Engine, StepEntry, plan_step
from borrowed_compute_b200.parts import FEED_FORWARDS, MIXERS, Runtime, StepContext

DEV = "cuda:0"
EPS = 1e-5
TYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
LLAMA3 = {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}


def listed():
    return [
        # A few requests to a tiny model in true 32-bit arithmetic, prompts and then tokens one by one: the smallest whole call, all
        # latency and launches.  (The first of the two tiny configurations that the benchmark and the tests have.)
        dict(name="replay_tiny_float32", kind="replay", dtype="float32", layers=2, width=64, heads=4, kv_heads=2, dim=16, ff=176, vocab=256,
             prompts=3, shortest=1, longest=17, tokens=8),
        # Serving: eight sequences of about 2,000 positions decode together, on layers of the 8B shape.
        dict(name="decode_batch8", kind="decode", dtype="bfloat16", layers=4, width=4096, heads=32, kv_heads=8, dim=128, ff=14336, vocab=32000,
             prompts=8, shortest=1500, longest=2040, tokens=8),
        # A batch of prompts of very unequal lengths through one attention layer of the 8B shape.
        dict(name="attention_ragged", kind="attention", dtype="bfloat16", width=4096, heads=32, kv_heads=8, dim=128, prompts=16, shortest=64,
             longest=2048),
        # One long prompt through the same layer.
        dict(name="attention_long", kind="attention", dtype="bfloat16", width=4096, heads=32, kv_heads=8, dim=128, prompts=1, shortest=16384,
             longest=16384),
        # The feed-forward of the 8B shape on a prompt of 2,048 tokens.
        dict(name="mlp_prompt", kind="mlp", dtype="bfloat16", rows=2048, width=4096, ff=14336),
        # The true 32-bit path on a short prompt: scores to compare other precisions with.
        dict(name="mlp_float32", kind="mlp", dtype="float32", rows=300, width=2048, ff=8192),
        # Many small experts of which a row uses six, on a prompt.
        dict(name="experts_prompt", kind="experts", dtype="bfloat16", rows=2048, width=2048, experts=64, top=6, ff=1408, shared=2816),
        # A decode batch of 64 through a layer whose every expert is then touched by a few rows.
        dict(name="experts_batch64", kind="experts", dtype="bfloat16", rows=64, width=4096, experts=32, top=4, ff=2048, shared=4096),
        # Recurrent mixers on prompts: one prompt, and three of unequal lengths.
        dict(name="delta_prompt", kind="delta", dtype="bfloat16", width=4096, heads=64, dim=64, rank=64, prompts=1, shortest=2048, longest=2048),
        dict(name="linear_prompts", kind="linear", dtype="bfloat16", width=4096, heads=16, dim=128, vdim=256, rank=16, prompts=3, shortest=400,
             longest=1800),
        # Two further ways to attend, on a prompt each.
        dict(name="talking_prompt", kind="talking", dtype="bfloat16", width=4096, heads=32, kv_heads=8, dim=128, window=1024, keep=4, prompts=1,
             shortest=2048, longest=2048),
        dict(name="latent_prompt", kind="latent", dtype="bfloat16", width=4096, heads=32, dim=64, rot=64, vdim=128, q_rank=1536, kv_rank=512,
             prompts=1, shortest=2048, longest=2048),
    ]


# --------------------------------------------------------------------------------------------- drawn cases

def _spread(rng, lo, hi):
    """A whole number between lo and hi, its logarithm spread evenly."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lengths_of(rng, most):
    """Prompts whose tokens add up to at most ``most``: how many, the shortest, the longest."""
    n = rng.choice([1, 1, 2, 3, 5, 8])
    longest = _spread(rng, 24, most // n)
    return dict(prompts=n, shortest=longest if n == 1 else _spread(rng, 1, longest), longest=longest)


def draw(rng):
    kind = rng.choice(["replay", "decode", "attention", "attention", "mlp", "mlp", "experts", "experts", "delta", "linear", "talking", "latent"])
    wide = rng.random() < 0.5
    if kind == "replay":
        c = rng.choice([dict(layers=2, width=64, heads=4, kv_heads=2, dim=16, ff=176, vocab=256),
                        dict(layers=3, width=96, heads=4, kv_heads=1, dim=32, ff=256, vocab=320)])
        longest = rng.randint(2, 100)
        return dict(kind=kind, dtype=rng.choice(["bfloat16", "float32"]), prompts=rng.randint(1, 6), shortest=rng.randint(1, longest), longest=longest,
                    tokens=rng.randint(1, 16), **c)
    if kind == "decode":
        c = dict(width=4096, heads=32, kv_heads=8, dim=128, ff=14336) if wide else dict(width=2048, heads=16, kv_heads=4, dim=128, ff=8192)
        n = rng.choice([1, 2, 5, 8, 24, 64])
        longest = _spread(rng, 64, 16384 // n if n > 5 else 3000)
        return dict(kind=kind, dtype="bfloat16", layers=rng.choice([2, 3, 4]), vocab=32000, prompts=n, shortest=max(1, longest - rng.randint(0, 200)),
                    longest=longest, tokens=8, **c)
    if kind == "attention":
        c = rng.choice([dict(width=4096, heads=32, kv_heads=8, dim=128), dict(width=5120, heads=40, kv_heads=40, dim=128),
                        dict(width=3072, heads=24, kv_heads=8, dim=128), dict(width=2048, heads=16, kv_heads=4, dim=128),
                        dict(width=2048, heads=32, kv_heads=8, dim=64)])
        return dict(kind=kind, dtype="bfloat16", **c, **_lengths_of(rng, 12000))
    if kind == "mlp":
        if rng.random() < 0.25:
            return dict(kind=kind, dtype="float32", rows=_spread(rng, 3, 600), width=rng.choice([1024, 2048]), ff=rng.choice([2816, 8192]))
        return dict(kind=kind, dtype="bfloat16", rows=_spread(rng, 1, 6000), **rng.choice([dict(width=4096, ff=14336), dict(width=2048, ff=8192),
                                                                                        dict(width=3072, ff=8192), dict(width=5120, ff=13824)]))
    if kind == "experts":
        c = dict(width=4096, experts=32, top=4, ff=2048, shared=4096) if wide else dict(width=2048, experts=64, top=6, ff=1408, shared=2816)
        return dict(kind=kind, dtype="bfloat16", rows=_spread(rng, 8, 4096), **c)
    lengths = _lengths_of(rng, 4096)
    if kind == "delta":
        return dict(kind=kind, dtype="bfloat16", dim=64, **(dict(width=4096, heads=64, rank=64) if wide else dict(width=2048, heads=32, rank=32)), **lengths)
    if kind == "linear":
        return dict(kind=kind, dtype="bfloat16", dim=128, vdim=256, rank=16, **(dict(width=4096, heads=16) if wide else dict(width=2048, heads=8)), **lengths)
    if kind == "talking":
        c = dict(width=4096, heads=32, kv_heads=8, window=1024) if wide else dict(width=2048, heads=16, kv_heads=4, window=512)
        return dict(kind=kind, dtype="bfloat16", dim=128, keep=4, **c, **lengths)
    c = dict(width=4096, heads=32, rot=64, vdim=128, q_rank=1536, kv_rank=512) if wide else \
        dict(width=2048, heads=16, rot=32, vdim=64, q_rank=768, kv_rank=256)
    return dict(kind=kind, dtype="bfloat16", dim=64, **c, **lengths)


def lengths(c):
    """The lengths of a case's prompts, spread evenly over their range, no two neighbours in order of size."""
    n = c["prompts"]
    if n == 1:
        return [c["longest"]]
    even = [c["shortest"] + (c["longest"] - c["shortest"]) * i // (n - 1) for i in range(n)]
    return even[::2][::-1] + even[1::2]


# ------------------------------------------------------------------------------------------------- inputs

class Drawn:
    """Tensors from a seed, in the order in which they are asked for."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(1_000_003 * (int(seed) + 1))

    def normal(self, shape, spread, dtype=torch.bfloat16):
        """Normal numbers, rounded to bfloat16 whatever type they are kept in (what a folder stores)."""
        return (torch.randn(shape, generator=self.gen, device=DEV, dtype=torch.float32) * spread).to(torch.bfloat16).to(dtype)

    def matrix(self, rows, cols, dtype=torch.bfloat16, gain=1.0):
        return self.normal((rows, cols), gain / cols ** 0.5, dtype)

    def vector(self, n, centre=1.0, spread=0.1):
        return centre + self.normal((n,), spread, torch.float32)


def engine_config(c):
    return {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": c["layers"], "hidden_size": c["width"], "num_attention_heads": c["heads"],
            "num_key_value_heads": c["kv_heads"], "head_dim": c["dim"], "intermediate_size": c["ff"], "vocab_size": c["vocab"],
            "rope_theta": 500000.0, "rope_scaling": LLAMA3, "rms_norm_eps": EPS, "tie_word_embeddings": False, "max_position_embeddings": 8192}


def engine_inputs(c, seed):
    """(weights by name, token ids of every prompt, token ids that follow [tokens, prompts])."""
    d, dt = Drawn(seed), TYPES[c["dtype"]]
    E, F, q, kv = c["width"], c["ff"], c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
    w = {"model.embed_tokens.weight": d.normal((c["vocab"], E), 1.0, dt), "model.norm.weight": d.vector(E),
         "lm_head.weight": d.matrix(c["vocab"], E, dt)}
    for i in range(c["layers"]):
        p = f"model.layers.{i}."
        w.update({p + "input_layernorm.weight": d.vector(E), p + "post_attention_layernorm.weight": d.vector(E),
                  p + "self_attn.q_proj.weight": d.matrix(q, E, dt), p + "self_attn.k_proj.weight": d.matrix(kv, E, dt),
                  p + "self_attn.v_proj.weight": d.matrix(kv, E, dt), p + "self_attn.o_proj.weight": d.matrix(E, q, dt),
                  p + "mlp.gate_proj.weight": d.matrix(F, E, dt), p + "mlp.up_proj.weight": d.matrix(F, E, dt),
                  p + "mlp.down_proj.weight": d.matrix(E, F, dt)})
    rng = random.Random(seed)
    prompts = [[rng.randrange(c["vocab"]) for _ in range(n)] for n in lengths(c)]
    return w, prompts, [[rng.randrange(c["vocab"]) for _ in prompts] for _ in range(c["tokens"])]


def part_inputs(c, seed):
    """(weights by their names inside the part, input rows)."""
    d, dt = Drawn(seed), TYPES[c["dtype"]]
    kind, E = c["kind"], c["width"]
    x = d.normal((c["rows"] if "rows" in c else sum(lengths(c)), E), 1.0, dt)
    if kind == "attention":
        q, kv = c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
        w = {"q_proj.weight": d.matrix(q, E, dt), "k_proj.weight": d.matrix(kv, E, dt), "v_proj.weight": d.matrix(kv, E, dt),
             "o_proj.weight": d.matrix(E, q, dt)}
    elif kind == "mlp":
        w = {"gate_proj.weight": d.matrix(c["ff"], E, dt), "up_proj.weight": d.matrix(c["ff"], E, dt), "down_proj.weight": d.matrix(E, c["ff"], dt)}
    elif kind == "experts":
        w = {"router": d.matrix(c["experts"], E, torch.float32)}
        for name, f in [(f"e{i}.", c["ff"]) for i in range(c["experts"])] + [("shared.", c["shared"])]:
            w.update({name + "gate": d.matrix(f, E, dt), name + "up": d.matrix(f, E, dt), name + "down": d.matrix(E, f, dt)})
    elif kind == "delta":
        hd = c["heads"] * c["dim"]
        w = {n: d.matrix(hd, E, dt) for n in ("r", "k", "v", "g", "a")}
        w.update({"a.b": d.vector(hd, 0.0, 0.5), "w1": d.matrix(c["rank"], E, dt), "w2": d.matrix(hd, c["rank"], torch.float32, 2.0),
                  "w0": d.vector(hd, 0.0, 1.0), "norm": d.vector(hd), "o": d.matrix(E, hd, dt)})
    elif kind == "linear":
        hd, hp = c["heads"] * c["dim"], c["heads"] * c["vdim"]
        w = {"q": d.matrix(hd, E, dt), "k": d.matrix(hd, E, dt), "v": d.matrix(hp, E, dt), "g": d.matrix(hp, E, dt), "a1": d.matrix(c["rank"], E, dt),
             "a2": d.matrix(hd, c["rank"], torch.float32, 2.0), "a2.b": d.vector(hd, 0.0, 1.0), "norm": d.vector(c["vdim"]), "o": d.matrix(E, hp, dt)}
    elif kind == "talking":
        q, kv, H = c["heads"] * c["dim"], c["kv_heads"] * c["dim"], c["heads"]
        w = {"q": d.matrix(q, E, dt), "k": d.matrix(kv, E, dt), "g": d.matrix(q, E, dt), "o": d.matrix(E, q, dt), "temp": d.vector(H),
             "talk": torch.eye(H, device=DEV) + d.normal((H, H), 0.5 / H ** 0.5, torch.float32), "q.b": d.vector(q, 0.0, 0.3), "k.b": d.vector(kv, 0.0, 0.3),
             "o.b": d.vector(E, 0.0, 0.3)}
    elif kind == "latent":
        H, R, Q = c["heads"], c["kv_rank"], c["q_rank"]
        w = {"dq": d.matrix(Q, E, dt), "dq.norm": d.vector(Q), "uq": d.matrix(H * (c["dim"] + c["rot"]), Q, dt), "uk": d.matrix(H * c["dim"], R, dt),
             "uv": d.matrix(H * c["vdim"], R, dt), "g": d.matrix(H, E, dt), "o": d.matrix(E, H * c["vdim"], dt),
             "dkv": d.matrix(R + c["rot"], E, dt), "dkv.norm": d.vector(R), "sink": d.vector(H, 0.0, 1.0)}
    return w, x


def rotary(dims, pairing="half", scaling=None):
    return {"kind": "rotary", "head_dim": dims, "theta": 500000.0, "pairing": pairing, "scaling": scaling, "max_positions": 32768}


def build(c):
    """The part of a case, without its weights."""
    kind, E = c["kind"], c["width"]
    if kind == "attention":
        return MIXERS.get("gqa_attention")(hidden_size=E, heads=c["heads"], kv_heads=c["kv_heads"], head_dim=c["dim"],
                                           position=rotary(c["dim"], scaling=LLAMA3))
    if kind == "mlp":
        return FEED_FORWARDS.get("swiglu")(hidden_size=E, intermediate_size=c["ff"])
    if kind == "experts":
        return FEED_FORWARDS.get("routed_experts")(hidden_size=E, experts=c["experts"], top=c["top"], intermediate_size=c["ff"], shared_size=c["shared"])
    if kind == "delta":
        return MIXERS.get("generalized_delta")(hidden_size=E, heads=c["heads"], head_dim=c["dim"], decay_rank=c["rank"], norm_eps=EPS)
    if kind == "linear":
        return MIXERS.get("gated_linear_attention")(hidden_size=E, heads=c["heads"], head_dim=c["dim"], value_dim=c["vdim"], decay_rank=c["rank"],
                                                    tau=16.0, norm_eps=EPS)
    if kind == "talking":
        return MIXERS.get("talking_attention")(hidden_size=E, heads=c["heads"], kv_heads=c["kv_heads"], head_dim=c["dim"], norm_eps=EPS,
                                               position=rotary(c["dim"] // 2), softcap=30.0, window=c["window"], keep_first=c["keep"])
    return MIXERS.get("latent_attention")(hidden_size=E, heads=c["heads"], head_dim=c["dim"], value_dim=c["vdim"], q_rank=c["q_rank"],
                                          kv_rank=c["kv_rank"], norm_eps=EPS, rot_dim=c["rot"], position=rotary(c["rot"], "adjacent"), sink=True)


def prepare(case, seed):
    c = case
    if c["kind"] in ("replay", "decode"):
        w, prompts, after = engine_inputs(c, seed)
        longest = max(len(p) for p in prompts) + c["tokens"]
        eng = Engine.from_tensors(engine_config(c), w, dtype=c["dtype"], device=DEV, max_slots=len(prompts), max_seq=longest,
                                  max_tokens=sum(-(-(len(p) + c["tokens"] + 1) // 64) * 64 for p in prompts))
        s = {"case": c, "engine": eng, "prompts": prompts, "after": after}
        if c["kind"] == "decode":
            s["slots"] = [eng.acquire() for _ in prompts]
            eng.step([StepEntry(slot, p, (len(p) - 1,)) for slot, p in zip(s["slots"], prompts)])
        return s
    w, x = part_inputs(c, seed)
    part = build(c)
    rt = Runtime(torch.device(DEV), TYPES[c["dtype"]], max_positions=max(lengths(c)) if "prompts" in c else c["rows"])
    part.load(w, rt)
    s = {"case": c, "part": part, "x": x}
    if "prompts" in c:
        n = lengths(c)
        cache = PagedCache(rt, [part.cache_need()], [part.state_need()], [None], max_tokens=sum(-(-k // 64) * 64 for k in n), n_slots=len(n), max_seq=max(n))
        slots = [cache.acquire() for _ in n]
        cache.slots.reserve_many([(slot, k, k) for slot, k in zip(slots, n)])
        cache.sync_tables()
        s["memory"] = cache.memory(0)
        plan = plan_step([StepEntry(slot, [0] * k) for slot, k in zip(slots, n)], [0] * len(n))
    else:
        plan = plan_step([StepEntry(i, [0]) for i in range(c["rows"])], [0] * c["rows"])

    def dev(a):
        return torch.from_numpy(a).to(DEV)

    s["context"] = StepContext(rows=plan.rows, seqs=plan.seqs, tokens=dev(plan.tokens), row_pos=dev(plan.row_pos), row_slot=dev(plan.row_slot),
                               seq_rows=dev(plan.seq_rows), seq_slot=dev(plan.seq_slot), seq_start=dev(plan.seq_start), max_new=plan.max_new,
                               max_total=plan.max_total, decode=plan.decode, host_seq_rows=tuple(int(v) for v in plan.seq_rows),
                               host_seq_slot=tuple(int(v) for v in plan.seq_slot), host_seq_start=tuple(int(v) for v in plan.seq_start))
    return s


def run(state):
    c = state["case"]
    if c["kind"] == "replay":
        eng = state["engine"]
        slots = [eng.acquire() for _ in state["prompts"]]
        out = [eng.step([StepEntry(slot, p, (len(p) - 1,)) for slot, p in zip(slots, state["prompts"])])]
        out += [eng.step([StepEntry(slot, (t,), (0,)) for slot, t in zip(slots, ids)]) for ids in state["after"]]
        for slot in slots:
            eng.release(slot)
        return out
    if c["kind"] == "decode":
        eng, slots = state["engine"], state["slots"]
        out = [eng.step([StepEntry(slot, (t,), (0,)) for slot, t in zip(slots, ids)]) for ids in state["after"]]
        for slot, p in zip(slots, state["prompts"]):
            eng.rollback(slot, len(p))
        return out
    x, context = state["x"], dataclasses.replace(state["context"], extras={})     # a step's context is its own
    result = torch.zeros(x.shape, dtype=torch.float32, device=x.device)
    if "memory" not in state:
        state["part"].forward(x, result, context)
        return [result]
    memory = state["memory"]
    if memory.state is not None:
        memory.state.zero_()                                                       # new sequences begin with an empty state
    state["part"].forward(x, result, context, memory)
    return [result] + ([memory.state] if memory.state is not None else list(memory.planes))


# ---------------------------------------------------------------------------------- what a pass cannot do without

def work(case):
    c = case
    kind, b = c["kind"], 4 if c["dtype"] == "float32" else 2
    E = c["width"]
    if kind in ("replay", "decode"):
        q, kv = c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
        matrices = c["layers"] * (E * (2 * q + 2 * kv) + 3 * E * c["ff"])
        head, n, T = c["vocab"] * E, lengths(c), c["tokens"]
        flops, nbytes = 0.0, 0.0
        if kind == "replay":
            flops += 2.0 * matrices * sum(n) + 2.0 * head * len(n) + c["layers"] * 4.0 * q * sum(k * (k + 1) / 2 for k in n)
            nbytes += b * (matrices + head + E * sum(n)) + 4 * c["vocab"] * len(n) + b * c["layers"] * 2 * kv * sum(n)
        for t in range(T):
            seen = sum(k + t + 1 for k in n)
            flops += 2.0 * (matrices + head) * len(n) + c["layers"] * 4.0 * q * seen
            nbytes += b * (matrices + head + E * len(n)) + 4 * c["vocab"] * len(n) + b * c["layers"] * 2 * kv * (seen + len(n))
        return {"bytes": nbytes, "flops": flops}
    rows = c["rows"] if "rows" in c else sum(lengths(c))
    io = rows * E * (b + 4.0)                                   # the input rows, and the float result

    def pairs(window=0, keep=0):
        """How many (row, position) pairs a row sees, over all prompts."""
        total = 0
        for n in lengths(c):
            total += n * (n + 1) // 2
            if window and n > window:
                out = n - window
                total -= out * (out + 1) // 2 - sum(min(keep, k) for k in range(1, out + 1))
        return total

    if kind == "attention":
        q, kv = c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
        m = E * (2 * q + 2 * kv)
        return {"bytes": io + b * m + b * 2 * kv * rows, "flops": 2.0 * m * rows + 4.0 * q * pairs()}
    if kind == "mlp":
        return {"bytes": io + b * 3 * E * c["ff"], "flops": 6.0 * E * c["ff"] * rows}
    if kind == "experts":
        touched = c["experts"] * (1.0 - (1.0 - c["top"] / c["experts"]) ** rows)
        return {"bytes": io + 4 * c["experts"] * E + b * 3 * E * (touched * c["ff"] + c["shared"]),
                "flops": rows * (6.0 * E * (c["top"] * c["ff"] + c["shared"]) + 2.0 * E * c["experts"])}
    if kind == "delta":
        hd = c["heads"] * c["dim"]
        m = E * (6 * hd + c["rank"])
        return {"bytes": io + b * m + 8.0 * hd * c["dim"] * c["prompts"], "flops": rows * (2.0 * m + 2.0 * c["rank"] * hd + 9.0 * hd * c["dim"])}
    if kind == "linear":
        hd, hp = c["heads"] * c["dim"], c["heads"] * c["vdim"]
        m = E * (2 * hd + 3 * hp + c["rank"])
        return {"bytes": io + b * m + 8.0 * hd * c["vdim"] * c["prompts"], "flops": rows * (2.0 * m + 2.0 * c["rank"] * hd + 5.0 * hd * c["vdim"])}
    if kind == "talking":
        q, kv = c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
        m = E * (3 * q + kv)
        return {"bytes": io + b * m + b * 2 * kv * rows, "flops": 2.0 * m * rows + (4.0 * q + 2.0 * c["heads"] ** 2) * pairs(c["window"], c["keep"])}
    H, R, Q, w = c["heads"], c["kv_rank"], c["q_rank"], c["dim"] + c["rot"]
    m = E * (Q + R + c["rot"] + H + H * c["vdim"]) + Q * H * w + R * H * (c["dim"] + c["vdim"])
    return {"bytes": io + b * m + b * (R + c["rot"]) * rows, "flops": 2.0 * m * rows + 2.0 * H * (w + c["vdim"]) * pairs()}


def tolerance(case):
    """About four times the distance measured from float64 sums on the same inputs: what rounding activations to bfloat16 between the
    products of a path leaves, or the order of 32-bit sums."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5}                      # measured: 4e-7 a whole tiny model, 1.7e-6 the feed-forward
    return {"rel": {"replay": 2e-2, "decode": 1.5e-2, "attention": 1.5e-2, "latent": 1.8e-2, "talking": 5e-3}.get(case["kind"], 1e-2)}


# ------------------------------------------------------------------------------------- the same in 64-bit arithmetic

def _norm(x, weight):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * weight


def _silu(x):
    return x * torch.sigmoid(x)


def _frequencies(dims, scaling):
    f = []
    for i in range(dims // 2):
        v = 500000.0 ** (-2.0 * i / dims)
        if scaling is not None:
            wave, orig = 2.0 * math.pi / v, float(scaling["original_max_position_embeddings"])
            lo, hi = scaling["low_freq_factor"], scaling["high_freq_factor"]
            if wave > orig / lo:
                v = v / scaling["factor"]
            elif wave >= orig / hi:
                t = (orig / wave - lo) / (hi - lo)
                v = (1.0 - t) * v / scaling["factor"] + t * v
        f.append(v)
    return torch.tensor(f, dtype=torch.float64, device=DEV)


def _rotate(x, dims, scaling=None, adjacent=False):
    """x [T, heads, d] at positions 0 .. T - 1: the first ``dims`` dimensions turn."""
    a = torch.arange(x.shape[0], device=DEV, dtype=torch.float64)[:, None] * _frequencies(dims, scaling)
    cos, sin = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if adjacent else (x[..., :dims // 2], x[..., dims // 2:dims])
    nu, nv = u * cos - v * sin, v * cos + u * sin
    turned = torch.stack([nu, nv], -1).flatten(-2) if adjacent else torch.cat([nu, nv], -1)
    return torch.cat([turned, x[..., dims:]], -1)


def _attend(q, k, v, scale, sink=None):
    """Causal softmax attention of one sequence, head by head: q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H * dv]."""
    T, H = q.shape[:2]
    group, out = H // k.shape[1], []
    for h in range(H):
        rows = []
        for at in range(0, T, 4096):                                          # a stretch of rows at a time: [4096, T] scores
            end = min(at + 4096, T)
            s = q[at:end, h] @ k[:end, h // group].T * scale
            s = s.masked_fill(torch.arange(end, device=DEV)[None] > torch.arange(at, end, device=DEV)[:, None], -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(end - at, 1)], 1)
            p = torch.softmax(s, -1)
            rows.append(p[:, :end] @ v[:end, h // group])
        out.append(torch.cat(rows))
    return torch.cat(out, -1)


def _llama_attention(x, w, c):
    T = x.shape[0]
    q = _rotate((x @ w["q_proj.weight"].T).view(T, c["heads"], -1), c["dim"], LLAMA3)
    k = _rotate((x @ w["k_proj.weight"].T).view(T, c["kv_heads"], -1), c["dim"], LLAMA3)
    v = (x @ w["v_proj.weight"].T).view(T, c["kv_heads"], -1)
    return _attend(q, k, v, c["dim"] ** -0.5) @ w["o_proj.weight"].T


def _glu(x, gate, up, down):
    return (_silu(x @ gate.T) * (x @ up.T)) @ down.T


def _experts(x, w, c):
    s = torch.sigmoid(x @ w["router"].T)
    weight, choice = torch.topk(s, c["top"], dim=-1)
    out = _glu(x, w["shared.gate"], w["shared.up"], w["shared.down"])
    for e in range(c["experts"]):
        rows, col = torch.nonzero(choice == e, as_tuple=True)
        if len(rows):
            out[rows] += _glu(weight[rows, col][:, None] * x[rows], *(w[f"e{e}.{n}"].double() for n in ("gate", "up", "down")))
    return out


def _delta(x, w, c):
    T, H, D = x.shape[0], c["heads"], c["dim"]
    r, k, v = ((x @ w[n].T).view(T, H, D) for n in ("r", "k", "v"))
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(x @ w["w1"].T) @ w["w2"].T + w["w0"])).view(T, H, D)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    au = torch.sigmoid(x @ w["a"].T + w["a.b"]).view(T, H, D) * u
    S, o = torch.zeros(H, D, D, dtype=torch.float64, device=DEV), torch.empty(T, H, D, dtype=torch.float64, device=DEV)
    for t in range(T):
        removed = torch.bmm(u[t][:, None], S)
        S = decay[t][..., None] * S - au[t][..., None] * removed + k[t][..., None] * v[t][:, None]
        o[t] = torch.bmm(r[t][:, None], S)[:, 0]
    y = _norm(o, 1.0).view(T, H * D) * w["norm"] * torch.sigmoid(x @ w["g"].T)
    return y @ w["o"].T, S.transpose(1, 2)


def _linear(x, w, c):
    T, H, D, P = x.shape[0], c["heads"], c["dim"], c["vdim"]
    q, k, v = (x @ w["q"].T).view(T, H, D) * D ** -0.5, (x @ w["k"].T).view(T, H, D), (x @ w["v"].T).view(T, H, P)
    decay = torch.exp(torch.nn.functional.logsigmoid((x @ w["a1"].T) @ w["a2"].T + w["a2.b"]) / 16.0).view(T, H, D)
    S, o = torch.zeros(H, D, P, dtype=torch.float64, device=DEV), torch.empty(T, H, P, dtype=torch.float64, device=DEV)
    for t in range(T):
        S = decay[t][..., None] * S + k[t][..., None] * v[t][:, None]
        o[t] = torch.bmm(q[t][:, None], S)[:, 0]
    y = _norm(o, w["norm"]).view(T, H * P) * _silu(x @ w["g"].T)
    return y @ w["o"].T, S.transpose(1, 2)


def _talking(x, w, c):
    T, H, G, d = x.shape[0], c["heads"], c["kv_heads"], c["dim"]
    q, v = (x @ w["q"].T + w["q.b"]).view(T, H, d), (x @ w["k"].T + w["k.b"]).view(T, G, d)
    q, k = _norm(_rotate(q, d // 2), 1.0), _norm(_rotate(v, d // 2), 1.0)
    j, out = torch.arange(T, device=DEV), []
    for at in range(0, T, 512):
        i = torch.arange(at, min(at + 512, T), device=DEV)[:, None]
        raw = torch.stack([q[at:at + 512, h] @ k[:, h * G // H].T * (d ** -0.5 * w["temp"][h]) for h in range(H)])
        s = torch.einsum("hm,mij->hij", w["talk"], 30.0 * torch.tanh(raw / 30.0))
        p = torch.softmax(s.masked_fill(~((j <= i) & ((i - j < c["window"]) | (j < c["keep"]))), -math.inf), -1)
        out.append(torch.cat([p[h] @ v[:, h * G // H] for h in range(H)], -1))
    return (torch.cat(out) * torch.sigmoid(x @ w["g"].T)) @ w["o"].T + w["o.b"]


def _latent(x, w, c):
    T, H, R, w_ = x.shape[0], c["heads"], c["kv_rank"], c["dim"] + c["rot"]
    q = (_norm(x @ w["dq"].T, w["dq.norm"]) @ w["uq"].T).view(T, H, w_)
    z = x @ w["dkv"].T
    lat = _norm(z[:, :R], w["dkv.norm"])
    q = torch.cat([q[..., :c["dim"]], _rotate(q[..., c["dim"]:], c["rot"], adjacent=True)], -1)
    kr = _rotate(z[:, None, R:], c["rot"], adjacent=True).expand(T, H, c["rot"])
    k = torch.cat([(lat @ w["uk"].T).view(T, H, -1), kr], -1)
    o = _attend(q, k, (lat @ w["uv"].T).view(T, H, -1), w_ ** -0.5, w["sink"]).view(T, H, -1)
    return (o * torch.sigmoid(x @ w["g"].T)[..., None]).view(T, -1) @ w["o"].T


def _llama(c, w, ids):
    """Scores of every row that a step returns: after the prompt (replay), and after every further token."""
    x = w["model.embed_tokens.weight"][torch.tensor(ids, device=DEV)].double()
    for i in range(c["layers"]):
        p = f"model.layers.{i}."
        part = {n: w[p + "self_attn." + n].double() for n in ("q_proj.weight", "k_proj.weight", "v_proj.weight", "o_proj.weight")}
        x = x + _llama_attention(_norm(x, w[p + "input_layernorm.weight"].double()), part, c)
        x = x + _glu(_norm(x, w[p + "post_attention_layernorm.weight"].double()),
                     *(w[p + f"mlp.{n}_proj.weight"].double() for n in ("gate", "up", "down")))
    last = x[-c["tokens"] - (c["kind"] == "replay"):]
    return _norm(last, w["model.norm.weight"].double()) @ w["lm_head.weight"].double().T


def exact(case, seed):
    c = case
    if c["kind"] in ("replay", "decode"):
        w, prompts, after = engine_inputs(c, seed)
        scores = torch.stack([_llama(c, w, p + [ids[i] for ids in after]) for i, p in enumerate(prompts)], 1)
        return list(scores)
    w, x = part_inputs(c, seed)
    w = {n: t.double() for n, t in w.items()} if c["kind"] != "experts" else \
        {n: t if n[0] == "e" else t.double() for n, t in w.items()}                # (an expert's matrices where they are used)
    x = x.double()
    if c["kind"] == "mlp":
        return [_glu(x, w["gate_proj.weight"], w["up_proj.weight"], w["down_proj.weight"])]
    if c["kind"] == "experts":
        return [_experts(x, w, c)]
    of = {"attention": _llama_attention, "delta": _delta, "linear": _linear, "talking": _talking, "latent": _latent}[c["kind"]]
    each = [of(part, w, c) for part in x.split(lengths(c))]
    if c["kind"] in ("delta", "linear"):
        return [torch.cat([o for o, _ in each]), torch.stack([s for _, s in each])]
    return [torch.cat(each), None, None]                                            # (pages of the cache are a layout of the framework's own)
