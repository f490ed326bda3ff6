"""The work this framework is used for, as cases that can be timed and checked: engine steps of the five model families (prompts and
decoding), and the calls a speculative verification round makes through the attention, cache, activation and acceptance interfaces.

A model case serves random bfloat16 weights of a published layer shape through `Engine.step`; a layer or two of every kind stand for the
whole depth.  `exact` restates each path in plain float64 tensors."""

from __future__ import annotations

import math

import torch

import vllm_rlt_b200 as rlt
from vllm_rlt_b200 import hybrid_lm, looped_lm, postnorm_lm, sandwich_lm, stream_lm

DEVICE = "cuda"
VOCAB = 49152
HEAD = 128
BLOCK = 16                # tokens of a page of the verification cases
ROOM = 2048               # tokens a decoding sequence may grow by before it starts over
EXACT = 8                 # sequences (or requests) of a case that are also computed in 64 bits

# Layer shapes by model width: heads, key/value heads, feed-forward widths, Mamba-2 (heads, head size, state, groups), experts (count, used, widths).
SHAPES = {
    2048: dict(heads=16, grouped=4, ff=5632, hybrid_kv=16, hybrid_ff=8448, mamba=(64, 64, 128, 1), experts=64, top=8, stream_ff=1024, postnorm_ff=704),
    4096: dict(heads=32, grouped=8, ff=9600, hybrid_kv=8, hybrid_ff=14336, mamba=(128, 64, 128, 8), experts=32, top=4, stream_ff=3584, postnorm_ff=2400),
}
FAMILIES = ("looped", "hybrid", "stream", "sandwich", "postnorm")


def listed():
    prefill = lambda name, family, width, count, shortest, longest: dict(
        name=name, kind="prefill", family=family, width=width, count=count, shortest=shortest, longest=longest)
    decode = lambda name, family, width, count, context: dict(name=name, kind="decode", family=family, width=width, count=count, context=context)
    return [
        # Prompts of a looped model's serving batch: U[128, 1024] tokens, four loops over the same layers.
        prefill("looped-prefill", "looped", 2048, 16, 128, 1024),
        # A few long conversations of a looped model: every loop reads a cache of its own.
        decode("looped-decode", "looped", 2048, 8, 4096),
        # An offline batch: equal prompts that fill a step.
        prefill("hybrid-prefill", "hybrid", 2048, 8, 2048, 2048),
        # A full serving batch of recurrent layers with some attention.
        decode("hybrid-decode", "hybrid", 2048, 64, 2048),
        # One long document, of odd length.
        prefill("stream-prefill", "stream", 2048, 1, 8191, 8191),
        # A medium batch over long contexts.
        decode("stream-decode", "stream", 2048, 16, 4096),
        # Interactive prompts of very different lengths in one step of a wide model.
        prefill("sandwich-prefill", "sandwich", 4096, 5, 37, 3001),
        # One user: launches and latency are what counts.
        decode("sandwich-decode", "sandwich", 2048, 1, 4095),
        # Equal prompts again, through recurrent layers with large states and experts.
        prefill("postnorm-prefill", "postnorm", 2048, 8, 2048, 2048),
        # A full serving batch.
        decode("postnorm-decode", "postnorm", 2048, 64, 2048),
        # The attention half of a speculative verification round, called the way an engine with models of its own calls it: four rows at
        # four loop depths for each of 64 requests.
        dict(name="verify", kind="verify", requests=64, rows=16, shortest=512, longest=4096, heads=16, kv_heads=16, ff=5632, layers=4, dtype="bfloat16"),
        # Its acceptance half: target and proposal distributions of every row, filtered as requests ask, accepted tokens, a residual draw.
        dict(name="accept", kind="accept", requests=128, rows=5, vocab=VOCAB, top_k=50, top_p=0.95, filtered=0.5, dtype="float32"),
    ]


def draw(rng):
    spread = lambda low, high: int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    kind = rng.choice(["prefill"] * 5 + ["decode"] * 5 + ["verify", "accept"])
    if kind == "verify":
        heads = rng.choice([16, 16, 32])
        requests = spread(1, 64)
        longest = spread(64, 4096)
        return dict(kind=kind, requests=requests, rows=rng.randint(2, 16), shortest=spread(17, longest), longest=longest, heads=heads,
                    kv_heads=rng.choice([16, heads // 4]), ff=rng.choice([5632, 9600, 5633]), layers=rng.randint(1, 4), dtype=rng.choice(["bfloat16", "bfloat16", "float16"]))
    if kind == "accept":
        return dict(kind=kind, requests=spread(1, 128), rows=rng.randint(2, 5), vocab=rng.choice([VOCAB, 32000, 50257]), top_k=rng.choice([0, 20, 50]),
                    top_p=rng.choice([1.0, 0.95, 0.8]), filtered=rng.choice([0.0, 0.5, 1.0]), dtype=rng.choice(["float32", "bfloat16"]))
    family = rng.choice(FAMILIES)
    width = rng.choice([2048, 2048, 4096])
    if kind == "decode":
        context = spread(100, 4096)
        most = min(64, 131072 // context) if family != "looped" else min(32, 32768 // context)
        return dict(kind=kind, family=family, width=width, count=spread(1, most), context=context)
    most = {2048: 16384, 4096: 6144}[width] // (2 if family == "looped" else 1)
    count = spread(1, 16)
    longest = spread(17, most // count)
    return dict(kind=kind, family=family, width=width, count=count, shortest=spread(max(1, longest // 20), longest), longest=longest)


# ---- models ------------------------------------------------------------------------------------
def configuration(family, width):
    """The config.json of a small stack with the family's layer kinds."""
    s = SHAPES[width]
    heads = s["heads"]
    top = {"vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}}
    dense = {"kind": "dense", "ff": s["ff"]}
    decays = [1 - 2.0 ** -(2 + 8 * h / heads) for h in range(heads)]
    if family == "looped":
        return dict(vocab_size=VOCAB, hidden_size=width, intermediate_size=s["ff"], num_hidden_layers=4, num_attention_heads=heads,
                    num_key_value_heads=heads, head_dim=HEAD, total_ut_steps=4)
    if family == "hybrid":
        m, size, state, groups = s["mamba"]
        mlp = {"kind": "dense", "ff": s["hybrid_ff"]}
        recurrent = {"type": "mamba2", "mlp": mlp, "mixer": {"heads": m, "vdim": size, "state": state, "groups": groups, "conv": 4, "norm_groups": groups}}
        attention = {"type": "attention", "mlp": mlp, "mixer": {"heads": heads, "kv_heads": s["hybrid_kv"], "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5,
                                                                "q_temp": {"coef": 0.1, "every": 2048}}}
        return dict(top, layers=[recurrent, attention, recurrent, recurrent])
    latent = {"heads": heads, "dim": HEAD, "rot_dim": 64, "vdim": HEAD, "q_rank": 1536, "kv_rank": 512, "scale": (HEAD + 64) ** -0.5,
              "rot": {"base": 10000.0, "dims": 64}}
    if family == "stream":
        clamped = dict(dense, limit=7.0)
        experts = {"kind": "moe", "router": {"experts": s["experts"], "top": s["top"]}, "expert": {"ff": s["stream_ff"]}}
        attention = {"type": "latent_attention", "mixer": dict(latent, mask={"size": 1024})}
        lightning = {"type": "lightning", "mixer": {"heads": heads, "dim": HEAD, "vdim": HEAD, "decay": decays}}
        return dict(top, streams=4, embedding={"bigram": {"buckets": 65521, "mul_prev": 8191, "mul_cur": 131}},
                    layers=[dict(attention, mlp=experts), dict(lightning, mlp=experts), dict(lightning, mlp=clamped), dict(attention, mlp=clamped)])
    if family == "sandwich":
        scaled = dict(latent, rot={"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}})
        windowed = {"heads": heads, "kv_heads": s["grouped"], "dim": HEAD, "vdim": HEAD, "conv": 4, "mask": {"size": 1024}, "scale": 2 * HEAD ** -0.5}
        return dict(top, residual_mult=0.5, logit_softcap=30.0,
                    layers=[{"type": t, "mixer": m, "mlp": dense} for t, m in (("attention", windowed), ("latent_attention_2", scaled),
                                                                              ("latent_attention", latent), ("attention", windowed))])
    experts = {"kind": "moe", "router": {"experts": s["experts"], "top": s["top"]}, "expert": {"ff": s["postnorm_ff"]}, "shared": {"ff": s["postnorm_ff"]}}
    delta = {"type": "channel_delta", "mixer": {"heads": heads, "kv_heads": heads, "dim": HEAD, "vdim": HEAD, "conv": 4}}
    talking = {"type": "attention", "mixer": {"heads": heads, "kv_heads": s["grouped"], "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5, "softcap": 20.0,
                                              "rot": {"base": 10000.0, "dims": HEAD // 2}, "mask": {"size": 1024, "keep_first": 4}}}
    keeping = {"type": "retention", "mixer": {"heads": heads, "dim": HEAD, "vdim": HEAD, "rot": {"base": 10000.0, "dims": HEAD}, "decay": decays}}
    return dict(top, layers=[dict(delta, mlp=dense), dict(talking, mlp=experts), dict(delta, mlp=experts), dict(keeping, mlp=dense)])


PARTS = {
    "looped": (rlt.LoopedLMConfig.from_json, looped_lm.parameter_shapes, rlt.LoopedLM),
    "hybrid": (rlt.HybridLMConfig.from_json, hybrid_lm.parameter_shapes, rlt.HybridLM),
    "stream": (rlt.StreamLMConfig.from_json, stream_lm.parameter_shapes, rlt.StreamLM),
    "sandwich": (rlt.SandwichLMConfig.from_json, sandwich_lm.parameter_shapes, rlt.SandwichLM),
    "postnorm": (rlt.PostNormLMConfig.from_json, lambda config: postnorm_lm.parameter_shapes(config, lambda name: 128), rlt.PostNormLM),
}


def shapes_of(family, width):
    return PARTS[family][1](PARTS[family][0](configuration(family, width)))


def weights(family, width, seed):
    """Weights at a trained model's scales: attention that prefers some keys, decays from a few tokens to thousands, routers that prefer some
    experts clearly."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    out = {}
    for name, shape in shapes_of(family, width).items():
        r = torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32 if len(shape) == 1 else torch.bfloat16)
        last = name.rsplit(".", 1)[-1]
        if family == "looped" and "norm" in name or name.startswith("final") or "norm" in last:
            r = 0.2 * r if family == "hybrid" and not name.endswith("mix.norm") else 1 + 0.2 * r
        elif "embed" in name or name == "bigram":
            r = 0.1 * r if family == "sandwich" else r               # there the table is the head too
        elif last in ("in", "out") and "hc" in name:
            r = 0.7 + 0.3 * r.abs()
        elif last == "mix":
            r = 0.6 * torch.eye(shape[0], device=DEVICE) + 0.1 * r.abs()
        elif last == "conv":
            r = 0.3 * r
            r[:, -1] += 0.6
        elif last == "A_log":
            r = torch.linspace(-2.0, 1.0, shape[0], device=DEVICE) + 0.1 * r
        elif last == "dt_bias":
            r = -3.0 + r
        elif last == "D":
            r = 0.5 + 0.5 * r
        elif last == "temp":
            r = 1 + 0.2 * r
        elif last == "talk":
            r = torch.eye(shape[0], device=DEVICE) + 0.1 * r
        elif last == "sink":
            r = 2.0 + r
        elif last == "router":
            r = 5.0 * r * shape[1] ** -0.5
        elif last == "correction":
            r = 1e-3 * r
        elif len(shape) == 1:
            r = 0.1 * r
        else:
            r = r * shape[-1] ** -0.5
        out[name] = r.to(torch.bfloat16)
    return out


def lengths_of(case, seed):
    if case["kind"] == "decode":
        return [case["context"]] * case["count"]
    g = torch.Generator().manual_seed(case["count"] * 1000003 + case["longest"])          # a case's lengths are its own: its work is the same for all seeds
    return torch.randint(case["shortest"], case["longest"] + 1, (case["count"],), generator=g).tolist()


def prompts_of(case, seed):
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, VOCAB, (n,), generator=g).tolist() for n in lengths_of(case, seed)]


def next_tokens(case, seed):
    g = torch.Generator().manual_seed(seed + 7919)
    return torch.randint(0, VOCAB, (64, case["count"]), generator=g).tolist()


class Serving:
    """A model behind the engine with a case's sequences."""

    def __init__(self, case, seed):
        self.decoding = case["kind"] == "decode"
        parse, _, model_class = PARTS[case["family"]]
        model = model_class(parse(configuration(case["family"], case["width"])), weights(case["family"], case["width"], seed), DEVICE, torch.bfloat16)
        self.prompts = prompts_of(case, seed)
        longest = max(map(len, self.prompts)) + (ROOM if self.decoding else 0)
        self.engine = rlt.Engine(model, max_tokens=len(self.prompts) * (-(-longest // 64) * 64), max_sequences=len(self.prompts), max_sequence_tokens=longest,
                                 capture_sizes=[len(self.prompts)])
        if self.decoding:
            self.next, self.at = next_tokens(case, seed), 0
            self.engine.prepare()
            self.start()

    def start(self):
        """The prompts, in steps of up to 16384 tokens."""
        entries, tokens = [], 0
        for name, prompt in enumerate(self.prompts):
            if tokens + len(prompt) > 16384 and entries:
                self.engine.step(entries)
                entries, tokens = [], 0
            entries.append(rlt.StepEntry(name, prompt))
            tokens += len(prompt)
        self.engine.step(entries)
        self.stored = len(self.prompts[0])

    def prefill(self):
        logits = self.engine.step([rlt.StepEntry(name, prompt, [len(prompt) - 1]) for name, prompt in enumerate(self.prompts)])
        for name in range(len(self.prompts)):
            self.engine.release(name)
        return logits

    def decode(self):
        if self.stored == self.engine.max_sequence_tokens:           # the conversations end and others of their length begin
            for name in range(len(self.prompts)):
                self.engine.release(name)
            self.start()
        tokens, self.at = self.next[self.at % len(self.next)], self.at + 1
        self.stored += 1
        return self.engine.step([rlt.StepEntry(name, [token], [0]) for name, token in enumerate(tokens)])


# ---- the verification round of an engine with models of its own ----------------------------------
class Verification:
    """Paged caches of a batch of requests, the rows that are verified, and one plan's metadata for all layers."""

    def __init__(self, case, seed):
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        dtype = getattr(torch, case["dtype"])
        n, rows, layers, heads, kv = case["requests"], case["rows"], case["layers"], case["heads"], case["kv_heads"]
        normal = lambda *shape: torch.randn(shape, generator=g, device=DEVICE, dtype=dtype)
        self.contexts = contexts_of(case)
        pages = [-(-c // BLOCK) for c in self.contexts]
        order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(seed)).to(torch.int32)
        tables = torch.full((n, max(pages)), -1, dtype=torch.int32)
        at = 0
        for i, count in enumerate(pages):
            tables[i, :count] = order[at:at + count]
            at += count
        lengths = torch.tensor(self.contexts)[:, None] - rows + 1 + torch.arange(rows)
        position = (lengths - 1).reshape(-1)
        request = torch.arange(n).repeat_interleave(rows)
        self.blocks = tables[request, position // BLOCK].long().to(DEVICE)
        self.offsets = (position % BLOCK).to(DEVICE)
        self.host_tables = tables
        self.tables = tables[request].contiguous().to(DEVICE)
        self.lengths = lengths.reshape(-1).to(torch.int32).to(DEVICE)
        self.keys, self.values = (normal(sum(pages), layers, BLOCK, kv, HEAD) for _ in range(2))
        self.rows = [dict(q=2 * normal(n * rows, heads, HEAD), k=normal(n * rows, kv, HEAD), v=normal(n * rows, kv, HEAD),
                          gate=normal(n * rows, case["ff"]), up=normal(n * rows, case["ff"])) for _ in range(layers)]
        self.backend = rlt.create_backend(DEVICE, dtype, HEAD, BLOCK)

    def run(self):
        outs = []
        with self.backend.kernel.shared_plan():
            for layer, r in enumerate(self.rows):
                keys, values = self.keys[:, layer], self.values[:, layer]
                rlt.kv_write(keys, values, r["k"], r["v"], self.blocks, self.offsets)
                outs.append((self.backend(r["q"], keys, values, self.tables, self.lengths), rlt.silu_and_mul(r["gate"], r["up"])))
        return outs


def contexts_of(case):
    g = torch.Generator().manual_seed(case["requests"])
    shortest = max(case["shortest"], case["rows"])
    return torch.randint(shortest, max(case["longest"], shortest) + 1, (case["requests"],), generator=g).tolist()


class Acceptance:
    """Logits of a round's rows, the drafts drawn from the proposals, and what the requests ask for."""

    def __init__(self, case, seed):
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        n, rows = case["requests"], case["rows"]
        uniform = lambda *shape: torch.rand(shape, generator=g, device=DEVICE)
        dtype = getattr(torch, case["dtype"])
        target = 2.5 * torch.randn(n * rows, case["vocab"], generator=g, device=DEVICE)
        self.target, self.draft = target.to(dtype), (target + 0.7 * torch.randn(target.shape, generator=g, device=DEVICE)).to(dtype)
        self.temperature = torch.full((n,), 0.8, device=DEVICE)
        self.temperature[::8] = 0.0                                   # some requests are greedy
        asked = torch.arange(n, device=DEVICE) < round(case["filtered"] * n)
        self.filters = dict(top_k=torch.where(asked, case["top_k"], 0).to(torch.int32), top_p=torch.where(asked, case["top_p"], 1.0).float()) \
            if case["filtered"] else {}
        self.cu = torch.arange(0, n * rows + 1, rows, dtype=torch.int32, device=DEVICE)
        self.starts = torch.randint(1, 4096, (n,), generator=g, device=DEVICE)
        self.u_accept, self.u_final, self.u_next = uniform(n * rows), uniform(n), uniform(n)
        every = {name: t.repeat_interleave(rows) for name, t in self.filters.items()}
        drafts, _ = rlt.sample_rows(self.draft, self.temperature.repeat_interleave(rows), uniform(n * rows), **every)
        self.tokens = torch.cat([torch.zeros(n, 1, dtype=torch.int64, device=DEVICE), drafts.view(n, rows)[:, :-1]], 1).contiguous()
        self.slots, self.slot_values = torch.randperm(n, generator=g, device=DEVICE), torch.zeros(n, 2, dtype=torch.int64, device=DEVICE)
        self.first = self.draft.view(n, rows, -1)[:, 0]

    def run(self):
        result, status = rlt.accept_rejection(self.target, self.draft, self.cu, self.tokens, self.starts, self.temperature, self.u_accept, self.u_final,
                                              slots=self.slots, slot_values=self.slot_values, **self.filters)
        proposals, drawn = rlt.sample_rows(self.first, self.temperature, self.u_next, **self.filters)
        return result, status, self.slot_values, proposals, drawn


# ---- what is measured ----------------------------------------------------------------------------
@torch.no_grad()
def prepare(case, seed):
    return {"verify": Verification, "accept": Acceptance}.get(case["kind"], Serving)(case, seed)


@torch.no_grad()
def run(state):
    if not isinstance(state, Serving):
        return state.run()
    logits = state.decode() if state.decoding else state.prefill()
    states = {name: t[:len(state.prompts)] for name, t in state.engine.cache.state.items()}
    return {"logits": logits[:EXACT], "states": {name: t[:EXACT] for name, t in states.items()},
            "rest": [logits[EXACT:], {name: t[EXACT:] for name, t in states.items()}]}


def work(case):
    if case["kind"] == "accept":
        rows = case["requests"] * (2 * case["rows"] + 1)
        return {"bytes": rows * case["vocab"] * (4 if case["dtype"] == "float32" else 2), "flops": rows * case["vocab"] * 4}
    if case["kind"] == "verify":
        contexts, rows, heads, kv = contexts_of(case), case["requests"] * case["rows"], case["heads"], case["kv_heads"]
        visible = sum(c * case["rows"] - case["rows"] * (case["rows"] - 1) // 2 for c in contexts)
        a_layer = 2 * (2 * sum(contexts) * kv * HEAD + 2 * rows * heads * HEAD + 4 * rows * kv * HEAD + 3 * rows * case["ff"])
        return {"bytes": case["layers"] * a_layer, "flops": case["layers"] * 4 * HEAD * heads * visible}
    family, width = case["family"], case["width"]
    config, s = configuration(family, width), SHAPES[width]
    lengths, decoding = lengths_of(case, 0), case["kind"] == "decode"
    tokens = len(lengths) if decoding else sum(lengths)
    portions = [(n, 1) if decoding else (0, n) for n in lengths]                         # (stored before, new)
    seen = lambda window, keep=0: sum(sum(min(p + 1, window + keep) for p in range(a, a + n)) if window else n * a + n * (n + 1) // 2 for a, n in portions)
    loops = config.get("total_ut_steps", 1)
    share = s["top"] / s["experts"]
    touched = min(1.0, 1 - (1 - share) ** tokens)
    flops = bytes_ = 0.0
    for name, shape in shapes_of(family, width).items():
        if len(shape) < 2 or name in ("bigram",) or "embed" in name and family != "sandwich":
            continue
        size = shape[0] * shape[1]
        routed = ".mlp.e" in name
        if "head" in name or "embed" in name:
            flops, bytes_ = flops + 2 * size * len(lengths), bytes_ + 2 * size
        else:
            flops, bytes_ = flops + 2 * size * tokens * loops * (share if routed else 1), bytes_ + 2 * size * (touched if routed else 1) * loops
    bytes_ += 2 * tokens * width + 4 * len(lengths) * VOCAB
    for layer in config.get("layers", [{"type": "looped"}] * 4 * loops):
        kind, m = layer["type"], layer.get("mixer", {})
        heads, window = m.get("heads", s["heads"]), (m.get("mask") or {}).get("size", 0)
        if kind.startswith("latent"):
            key, value, stored = HEAD + 64, HEAD, 512 + 64
        elif kind in ("looped", "attention"):
            key, value, stored = HEAD, HEAD, 2 * HEAD * m.get("kv_heads", s["heads"])
        else:                                                                          # a state per sequence, read and written
            inner = (m.get("state", HEAD)) * m["vdim"] * heads
            flops, bytes_ = flops + 4 * inner * tokens, bytes_ + 4 * inner * len(lengths) * (2 if decoding else 1)
            continue
        flops += 2 * heads * (key + value) * seen(window)
        bytes_ += 2 * stored * (sum(min(a, window or a) for a, _ in portions) + tokens)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # Acceptance is defined to the bit.  Verification: outputs are 16-bit, and probabilities pass through 16 bits (0.0018 and, of the activation
    # that is rounded twice, 0.0024 from 64 bits).  Models: about a hundred roundings to bfloat16 lie between a token and its logits, and an
    # expert chosen by a hair changes; 0.006 to 0.018 from 64 bits, and 0.0055 between two runs whose experts get their rows in another order.
    if case["kind"] == "accept":
        return "exact"
    if case["kind"] == "verify":
        return {"rel": 0.01 if case["dtype"] == "bfloat16" else 0.002}
    return {"rel": 0.03}


# ---- the same in 64 bits -------------------------------------------------------------------------
def rms(x, eps, weight=1.0):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * weight


def centred(x, eps, weight):
    return rms(x - x.mean(-1, keepdim=True), eps, weight)


def rotated(x, dims, base, halves, scaling=None):
    """x [n, .., d]: pairs of its first `dims` dimensions turned by position times frequency."""
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    turns, amplitude = base ** (-2 * i / dims), 1.0
    if scaling:
        pair = lambda t: dims * math.log(scaling["original"] / (2 * math.pi * t)) / (2 * math.log(base))
        low, high = max(math.floor(pair(scaling["fast"])), 0), min(math.ceil(pair(scaling["slow"])), dims - 1)
        slow = ((i - low) / max(high - low, 0.001)).clamp(0, 1)
        turns, amplitude = turns / scaling["factor"] * slow + turns * (1 - slow), 0.1 * math.log(scaling["factor"]) + 1
    angle = torch.arange(x.shape[0], device=x.device)[:, None] * turns
    c, s = (amplitude * f(angle).reshape(x.shape[0], *[1] * (x.dim() - 2), -1) for f in (torch.cos, torch.sin))
    y = x.clone()
    first, second = (slice(0, dims // 2), slice(dims // 2, dims)) if halves else (slice(0, dims, 2), slice(1, dims, 2))
    u, v = x[..., first], x[..., second]
    y[..., first], y[..., second] = u * c - v * s, v * c + u * s
    return y


def convolved(u, weight):
    taps = weight.shape[1]
    padded = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u])
    return sum(weight[:, j] * padded[j:j + u.shape[0]] for j in range(taps))


def seen_keys(q, k, v, weigh, first=0, rows=256):
    """Blocks of query rows over all keys: weigh(scores [H, rows, T], distances [rows, T]) gives weights; q [n, H, d], k [T, G, d], v [T, G, e]."""
    share, out = q.shape[1] // k.shape[1], []
    k, v = (x.repeat_interleave(share, 1) for x in (k, v))
    for at in range(0, q.shape[0], rows):
        part = q[at:at + rows]
        last = first + at + part.shape[0]
        distance = torch.arange(first + at, last, device=q.device)[:, None] - torch.arange(last, device=q.device)
        out.append(torch.einsum("hnt,the->nhe", weigh(torch.einsum("nhd,thd->hnt", part, k[:last]), distance), v[:last]))
    return torch.cat(out)


def softmaxed(scale, window=0, keep=0, sink=None, cap=0.0, talk=None):
    def weigh(scores, distance):
        keys = torch.arange(distance.shape[1], device=distance.device)
        scores = scores * scale
        scores = cap * torch.tanh(scores / cap) if cap else scores
        hidden = (distance < 0) | ((distance >= window) & (keys >= keep) if window else False)
        scores = scores.masked_fill(hidden, -math.inf)
        if sink is not None:
            scores = torch.cat([scores, sink[:, None, None].expand(-1, scores.shape[1], 1)], -1)
        probabilities = torch.softmax(scores, -1)
        probabilities = probabilities[..., :-1] if sink is not None else probabilities
        return torch.einsum("hg,gnt->hnt", talk, probabilities) if talk is not None else probabilities
    return weigh


def decayed(decay):
    return lambda scores, distance: scores * torch.where(distance < 0, 0.0, decay[:, None, None] ** distance.clamp_min(0))


silu, sigmoid = torch.nn.functional.silu, torch.sigmoid


class Exact:
    """A family's model over one token sequence, in float64."""

    def __init__(self, family, width, seed):
        self.family, self.config = family, configuration(family, width)
        self.w = {name: t.double() for name, t in weights(family, width, seed).items()}
        self.eps = self.config["norm"]["eps"] if "norm" in self.config else 1e-6

    def last(self, tokens):
        """Logits of the last token, and the recurrent states behind it."""
        self.states = {}
        return getattr(self, self.family)(tokens), self.states

    def looped(self, tokens):
        w, c = self.w, self.config
        x = w["model.embed_tokens.weight"][tokens]
        for _ in range(c["total_ut_steps"]):
            for i in range(c["num_hidden_layers"]):
                get = lambda name: w[f"model.layers.{i}.{name}.weight"]
                h = rms(x, self.eps, get("input_layernorm"))
                q, k, v = ((h @ get(f"self_attn.{n}_proj").T).unflatten(1, (-1, HEAD)) for n in "qkv")
                q, k = (rotated(t, HEAD, 1e6, True) for t in (q, k))
                o = seen_keys(q, k, v, softmaxed(HEAD ** -0.5)).flatten(1) @ get("self_attn.o_proj").T
                x = x + rms(o, self.eps, get("input_layernorm_2"))
                h = rms(x, self.eps, get("post_attention_layernorm"))
                h = (silu(h @ get("mlp.gate_proj").T) * (h @ get("mlp.up_proj").T)) @ get("mlp.down_proj").T
                x = x + rms(h, self.eps, get("post_attention_layernorm_2"))
            x = rms(x, self.eps, w["model.norm.weight"])
        return x[-1] @ w["lm_head.weight"].T

    def hybrid(self, tokens):
        w, x = self.w, self.w["embed"][tokens]
        for i, layer in enumerate(self.config["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            h = rms(x, self.eps, 1 + w[p + "norm1"])
            y = torch.nn.functional.gelu(h @ w[p + "mlp.up"].T) @ w[p + "mlp.down"].T
            x = x + y + getattr(self, "hybrid_" + layer["type"])(p, m, h) @ w[p + "mix.o"].T
        return rms(x[-1], self.eps, 1 + w["final.norm"]) @ w["head"].T

    def hybrid_attention(self, p, m, h):
        q, k, v = ((h @ self.w[f"{p}mix.{n}"].T).unflatten(1, (-1, HEAD)) for n in "qkv")
        at = torch.arange(h.shape[0], device=h.device)
        temperature = 1 + m["q_temp"]["coef"] * torch.log((at + 1) // m["q_temp"]["every"] + 1.0)
        slope = 2.0 ** (-8.0 * (torch.arange(m["heads"], device=h.device, dtype=torch.float64) + 1) / m["heads"])
        weigh = softmaxed(1.0)
        scored = lambda scores, distance: weigh(scores * m["scale"] - slope[:, None, None] * distance, distance)
        return seen_keys(q * temperature[:, None, None], k, v, scored).flatten(1)

    def hybrid_mamba2(self, layer, m, h):
        w, p, heads, gn = self.w, layer + "mix.", m["heads"], m["groups"] * m["state"]
        inner = heads * m["vdim"]
        z, xbc, dt = (h @ w[p + "in"].T).split((inner, inner + 2 * gn, heads), 1)
        x, b, c = silu(convolved(xbc, w[p + "conv"]) + w[p + "conv.b"]).split((inner, gn, gn), 1)
        x, b, c = x.unflatten(1, (heads, -1)), b.unflatten(1, (m["groups"], -1)), c.unflatten(1, (m["groups"], -1))
        dt = torch.nn.functional.softplus(dt + w[p + "dt_bias"])
        total = torch.cumsum(-torch.exp(w[p + "A_log"]) * dt, 0)
        out, share = [], heads // m["groups"]
        for at in range(0, h.shape[0], 128):
            last = min(at + 128, h.shape[0])
            hidden = torch.arange(at, last, device=h.device)[:, None] < torch.arange(last, device=h.device)
            fade = torch.exp((total[at:last, None] - total[None, :last]).masked_fill(hidden[..., None], -math.inf))
            scores = torch.einsum("ngs,tgs->ntg", c[at:last], b[:last]).repeat_interleave(share, 2)
            out.append(torch.einsum("nth,thp->nhp", fade * scores * dt[:last], x[:last]))
        self.states[layer + "ssm"] = torch.einsum("th,thn,thp->hnp", torch.exp(total[-1] - total) * dt, b.repeat_interleave(share, 1), x)
        y = (torch.cat(out) + w[p + "D"][:, None] * x).flatten(1) * silu(z)
        return rms(y.unflatten(1, (m["norm_groups"], -1)), self.eps).flatten(1) * w[p + "norm"]

    def latent(self, p, m, h, halves, sink=None, scaling=None, window=0):
        w, n = self.w, h.shape[0]
        turn = lambda t: rotated(t, m["rot"]["dims"], m["rot"]["base"], halves, scaling)
        q = (rms(h @ w[p + "dq"].T, self.eps, w[p + "dq.norm"]) @ w[p + "uq"].T).unflatten(1, (m["heads"], -1))
        down = h @ w[p + "dkv"].T
        c = rms(down[:, :m["kv_rank"]], self.eps, w[p + "dkv.norm"])
        shared = turn(down[:, m["kv_rank"]:])[:, None].expand(n, m["heads"], -1)
        k = torch.cat([(c @ w[p + "uk"].T).unflatten(1, (m["heads"], -1)), shared], -1)
        q = torch.cat([q[..., :HEAD], turn(q[..., HEAD:])], -1)
        return seen_keys(q, k, (c @ w[p + "uv"].T).unflatten(1, (m["heads"], -1)), softmaxed(m["scale"], window, sink=sink)).flatten(1)

    def stream(self, tokens):
        w, c = self.w, self.config
        b = c["embedding"]["bigram"]
        rows = torch.cat([tokens.new_full((1,), b["buckets"]), (tokens[:-1] * b["mul_prev"] + tokens[1:] * b["mul_cur"]) % b["buckets"]])
        streams = [rms(w["embed"][tokens] + w["bigram"][rows], self.eps, w["embed.norm"])] * c["streams"]
        for i, layer in enumerate(c["layers"]):
            for q in (1, 2):
                p, hc, m = f"l{i}.", f"l{i}.hc{q}.", layer["mixer"]
                h = rms(sum(a * x for a, x in zip(w[hc + "in"], streams)), self.eps, w[f"{p}norm{q}"])
                if q == 2:
                    y = self.stream_feed(p + "mlp.", layer["mlp"], h)
                elif layer["type"] == "lightning":
                    a, k, v = (silu(h @ w[f"{p}mix.{n}"].T).unflatten(1, (m["heads"], -1)) for n in "qkv")
                    y = self.linear(f"r{i}.state", a, k, v, m["decay"]).flatten(1)
                    y = (rms(y, self.eps, w[p + "mix.norm"]) * sigmoid(h @ w[p + "mix.g"].T)) @ w[p + "mix.o"].T
                else:
                    y = self.latent(p + "mix.", m, h, False, window=m["mask"]["size"]) @ w[p + "mix.o"].T
                mix, out = w[hc + "mix"], w[hc + "out"]
                streams = [sum(mix[s, t] * streams[s] for s in range(len(streams))) + out[t] * y for t in range(len(streams))]
        return rms(sum(streams)[-1], self.eps, w["final.norm"]) @ w["head"].T

    def linear(self, name, q, k, v, decay):
        """Attention that fades by a constant per head; its state after the last token."""
        decay = torch.tensor(decay, dtype=torch.float64, device=q.device)
        left = torch.arange(q.shape[0] - 1, -1, -1, device=q.device)
        self.states[name] = torch.einsum("th,thd,the->hde", decay ** left[:, None], k, v)
        return seen_keys(q, k, v, decayed(decay))

    def stream_feed(self, p, f, h):
        w = self.w
        if f["kind"] == "dense":
            g, u = (h @ w[p + "gate"].T).clamp(max=f["limit"]), (h @ w[p + "up"].T).clamp(-f["limit"], f["limit"])
            return (g * sigmoid(1.702 * g) * (u + 1)) @ w[p + "down"].T
        scores = torch.softmax(h @ w[p + "router"].T, -1)
        chosen = torch.topk(scores + w[p + "correction"], f["router"]["top"], -1).indices
        picked = scores.gather(1, chosen)
        expert = lambda e, x: torch.relu(x @ w[f"{p}e{e}.up"].T) ** 2 @ w[f"{p}e{e}.down"].T
        return self.routed(h, chosen, picked / (picked.sum(1, keepdim=True) + 1e-20), f["router"]["experts"], expert)

    @staticmethod
    def routed(h, chosen, shares, experts, expert):
        y = torch.zeros_like(h)
        for e in range(experts):
            row, place = torch.nonzero(chosen == e, as_tuple=True)
            if len(row):
                y[row] += shares[row, place][:, None] * expert(e, h[row])
        return y

    def sandwich(self, tokens):
        w, c, x = self.w, self.config, self.w["embed"][tokens]
        for i, layer in enumerate(c["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            h = centred(x, self.eps, w[p + "norm1"])
            if layer["type"] == "attention":
                q, k, v = (convolved(h @ w[f"{p}mix.{n}"].T + w[f"{p}mix.{n}.b"], w[f"{p}mix.{n}.conv"]).unflatten(1, (-1, HEAD)) for n in "qkv")
                y = seen_keys(rms(q, self.eps), rms(k, self.eps), v, softmaxed(m["scale"], m["mask"]["size"])).flatten(1)
            else:
                second = layer["type"] == "latent_attention_2"
                y = self.latent(p + "mix.", m, h, True, w[p + "mix.sink"] if second else None, m["rot"].get("scaling"))
            gate = sigmoid(h @ w[p + "mix.g"].T).unflatten(1, (m["heads"], -1))
            y = (y.unflatten(1, (m["heads"], -1)) * gate).flatten(1) @ w[p + "mix.o"].T
            x = x + c["residual_mult"] * centred(y, self.eps, w[p + "norm1b"])
            h = centred(x, self.eps, w[p + "norm2"])
            y = (torch.nn.functional.gelu(h @ w[p + "mlp.gate"].T, approximate="tanh") * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
            x = x + c["residual_mult"] * centred(y, self.eps, w[p + "norm2b"])
        cap = c["logit_softcap"]
        return cap * torch.tanh(centred(x[-1], self.eps, w["final.norm"]) @ w["embed"].T / cap)

    def postnorm(self, tokens):
        w, x = self.w, self.w["embed"][tokens]
        for i, layer in enumerate(self.config["layers"]):
            p = f"l{i}."
            x = x + rms(getattr(self, "postnorm_" + layer["type"])(p, layer["mixer"], x) @ w[p + "mix.o"].T, self.eps, w[p + "norm1"])
            x = x + rms(self.postnorm_feed(p + "mlp", layer["mlp"], x), self.eps, w[p + "norm2"])
        return rms(x[-1], self.eps, w["final.norm"]) @ w["head"].T

    def postnorm_channel_delta(self, layer, m, h):
        p, w, heads = layer + "mix.", self.w, m["heads"]
        q, k, v = (silu(convolved(h @ w[p + n].T, w[f"{p}{n}.conv"])).unflatten(1, (heads, -1)) for n in "qkv")
        q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, beta = q * HEAD ** -0.5, sigmoid(h @ w[p + "b"].T)
        low = (h @ w[p + "a1"].T @ w[p + "a2"].T + w[p + "dt_bias"]).unflatten(1, (heads, -1))
        fade = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * torch.nn.functional.softplus(low))[..., None]
        state, out = h.new_zeros(heads, HEAD, HEAD), []
        for t in range(h.shape[0]):
            state = fade[t] * state
            change = beta[t][:, None, None] * (v[t][:, None] - k[t][:, None] @ state)
            state = torch.baddbmm(state, k[t][:, :, None], change)
            out.append(q[t][:, None] @ state)
        self.states[layer + "state"] = state
        y = rms(torch.stack(out).squeeze(2), self.eps, w[p + "norm"]).flatten(1)
        return y * sigmoid(h @ w[p + "g1"].T @ w[p + "g2"].T)

    def postnorm_attention(self, layer, m, h):
        p, w = layer + "mix.", self.w
        q, k, v = ((h @ w[p + n].T).unflatten(1, (-1, HEAD)) for n in "qkv")
        q, k = (rotated(rms(t, self.eps, w[f"{p}{n}.norm"]), m["rot"]["dims"], m["rot"]["base"], False) for n, t in (("q", q), ("k", k)))
        weigh = softmaxed(m["scale"], m["mask"]["size"], m["mask"]["keep_first"], cap=m["softcap"], talk=w[p + "talk"])
        return seen_keys(q * w[p + "temp"][:, None], k, v, weigh).flatten(1)

    def postnorm_retention(self, layer, m, h):
        p, w = layer + "mix.", self.w
        q, k, v = ((h @ w[p + n].T).unflatten(1, (m["heads"], -1)) for n in "qkv")
        q, k = (rotated(t, m["rot"]["dims"], m["rot"]["base"], True) for t in (q, k))
        y = self.linear(layer + "state", q, k * HEAD ** -0.5, v, m["decay"])
        return rms(y, self.eps).flatten(1) * silu(h @ w[p + "g"].T)

    def postnorm_feed(self, p, f, h):
        w = self.w
        unit = lambda name, x: (silu(x @ w[name + ".gate"].T) * (x @ w[name + ".up"].T)) @ w[name + ".down"].T
        if f["kind"] == "dense":
            return unit(p, h)
        picked, chosen = torch.topk(h @ w[p + ".router"].T + w[p + ".router.b"], f["router"]["top"], -1)
        return unit(p + ".shared", h) + self.routed(h, chosen, torch.softmax(picked, -1), f["router"]["experts"], lambda e, x: unit(f"{p}.e{e}", x))


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "accept":
        return None
    if case["kind"] == "verify":
        return exact_verification(case, seed)
    model, prompts = Exact(case["family"], case["width"], seed), prompts_of(case, seed)
    first = next_tokens(case, seed)[0] if case["kind"] == "decode" else [None] * len(prompts)
    done = [model.last(torch.tensor(p if t is None else [*p, t], device=DEVICE)) for p, t in list(zip(prompts, first))[:EXACT]]
    logits, states = zip(*done)
    return {"logits": torch.stack(logits), "states": {name: torch.stack([s[name] for s in states]) for name in states[0]}, "rest": None}


def exact_verification(case, seed):
    state, rows, outs = Verification(case, seed), case["rows"], []
    for layer, r in enumerate(state.rows):
        attended = []
        for i, context in enumerate(state.contexts):
            pages = state.host_tables[i, :-(-context // BLOCK)].long().to(DEVICE)
            own = slice(i * rows, (i + 1) * rows)
            keys, values = (pool[pages, layer].flatten(0, 1)[:context].double() for pool in (state.keys, state.values))
            keys[-rows:], values[-rows:] = r["k"][own].double(), r["v"][own].double()
            attended.append(seen_keys(r["q"][own].double(), keys, values, softmaxed(HEAD ** -0.5), first=context - rows))
        outs.append((torch.cat(attended), silu(r["gate"].double()) * r["up"].double()))
    return outs
