"""What the framework's speed is measured on: its mixers, experts and whole steps at the sizes that its benchmark and its
configurations have, each through the entry points that a program calls (`build_model`, `ModelRunner.build_context` and `.step`, a
part's `forward`).  Prompts run eagerly, as the engine runs them; decoding replays a CUDA graph, as the engine's decode steps do.

A case is a dict: `kind` (what runs), `requests`, `tokens` (the most that a request brings; 1: it decodes), `context` (the most positions
that it held before), and the layer's sizes.  The requests of a case are ragged: `lengths` draws theirs below those two numbers.
"""

from __future__ import annotations

import math
import random

import torch

PAGE = 16
VOCAB = 1024          # of the models that are built for one layer; whole models say theirs
F64 = torch.float64
YARN = {"factor": 8.0, "original": 8192, "fast": 16.0, "slow": 2.0}
EPS = 1e-6
TAPS = 4


# ---- the cases ------------------------------------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # one person's chat: a token of one request through one attention layer of the 1B shape, launch and latency alone
        dict(name="attend_decode_1", kind="attention", requests=1, tokens=1, context=1000, width=2048, heads=32, kv_heads=8, dim=64),
        # a busy server: 64 requests of unlike lengths through an attention layer of the 8B shape
        dict(name="attend_decode_64", kind="attention", requests=64, tokens=1, context=2300, width=4096, heads=32, kv_heads=8, dim=128),
        # chunked prefill: portions of up to 512 tokens on contexts of up to 3,000, an attention layer of the 3B shape
        dict(name="attend_prefill", kind="attention", requests=8, tokens=512, context=3000, width=3072, heads=24, kv_heads=8, dim=128),
        # two long prompts through Dezolorn's attention: a window, kept first keys, weights of 16 bits
        dict(name="window_prefill", kind="window", requests=2, tokens=2048, context=0, width=2048, heads=32, kv_heads=8, dim=64, window=1024, keep=8),
        # the second portion of a prompt through Sorizen's attention on a cached latent, heads gated
        dict(name="latent_prefill", kind="latent", requests=1, tokens=1500, context=1200, width=2048, heads=16, dim=128, rot=64, rank=512, window=1024),
        # a prompt through Dezolorn's gated delta rule
        dict(name="delta_prefill", kind="delta", requests=1, tokens=2048, context=0, width=2048, heads=16, kv_heads=8, dim=128),
        # three prompts through Rasezen's state space
        dict(name="mamba2_prefill", kind="mamba2", requests=3, tokens=1000, context=0, width=2048, heads=64, dim=64, state=128, groups=8),
        # and 64 requests that decode with it: the state read and written
        dict(name="mamba2_decode_64", kind="mamba2", requests=64, tokens=1, context=8, width=2048, heads=64, dim=64, state=128, groups=8),
        # Rasezen's routed experts for a prompt, a shared one and experts that return their input among them
        dict(name="experts_prefill", kind="experts", requests=1, tokens=2048, context=0, width=2048, experts=32, identity=4, top=4, inter=1024, shared=2048),
        # and for 24 requests that decode
        dict(name="experts_decode", kind="experts", requests=24, tokens=1, context=8, width=2048, experts=32, identity=4, top=4, inter=1024, shared=2048),
        # the headline: a whole decode step of 8 requests (the 8B shape, two of its layers), embedding to greedy tokens
        dict(name="llama_decode_8", kind="llama", requests=8, tokens=1, context=1024, width=4096, ff=14336, heads=32, kv_heads=8, dim=128, layers=2,
             vocab=128256, dtype="bf16"),
        # the exact mode: prompts admitted together through a whole float32 model of the 1B shape (two of its layers)
        dict(name="llama_float32", kind="llama", requests=3, tokens=300, context=0, width=2048, ff=8192, heads=32, kv_heads=8, dim=64, layers=2,
             vocab=32768, dtype="float32"),
    ]


def _between(rng: random.Random, lo: int, hi: int, step: int = 1) -> int:
    """Spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["attention", "attention", "window", "latent", "delta", "mamba2", "experts", "llama"])
    decode = rng.random() < 0.4 and kind not in ("llama",)
    requests = _between(rng, 1, 64) if decode else rng.choice([1, 1, 2, 3, 5, 8])
    tokens = 1 if decode else max(2, _between(rng, 16, 2048) // (requests if requests > 3 else 1))
    width = rng.choice([1024, 2048, 3072, 4096])
    case = dict(kind=kind, requests=requests, tokens=tokens, context=8 if decode else 0, width=width)
    if kind in ("attention", "window"):
        dim = rng.choice([64, 128])
        case.update(context=_between(rng, 16, 3000), kv_heads=8, heads=8 * rng.choice([1, 2, 3, 4]), dim=dim)
        if kind == "window":
            case.update(window=_between(rng, 100, 1500), keep=rng.choice([0, 1, 4, 8, 17]), context=case["context"] if decode else 0)
    elif kind == "latent":
        case.update(context=_between(rng, 16, 1500), heads=rng.choice([8, 16, 32]), dim=128, rot=64, rank=512, window=_between(rng, 200, 4000))
    elif kind == "delta":
        case.update(heads=rng.choice([8, 16, 32]), kv_heads=8, dim=128)
    elif kind == "mamba2":
        case.update(heads=rng.choice([32, 64, 128]), dim=64, state=rng.choice([64, 128]), groups=rng.choice([1, 4, 8]))
    elif kind == "experts":
        case.update(experts=rng.choice([16, 32]), identity=rng.choice([0, 4]), top=rng.choice([2, 4, 6]), inter=rng.choice([512, 1024]), shared=2048)
    else:
        case.update(requests=rng.choice([1, 2, 3]), tokens=_between(rng, 8, 250), width=1024, ff=4096, heads=16, kv_heads=8, dim=64, layers=2,
                    vocab=16384, dtype=rng.choice(["bf16", "float32"]))
    return case


def lengths(case: dict) -> list[tuple[int, int]]:
    """(positions held before, tokens brought) of every request: ragged, the same for every seed."""
    rng = random.Random(case["requests"] * 1000003 + case["tokens"] * 1009 + case["context"])
    out = []
    for i in range(case["requests"]):
        full = i == 0  # one request is as large as the case says
        take = case["tokens"] if full or case["tokens"] == 1 else max(2, int(case["tokens"] * rng.uniform(0.3, 1.0)))
        held = case["context"] if full or case["context"] <= 8 else int(case["context"] * rng.uniform(0.2, 1.0))
        out.append((held, take))
    return out


# ---- configurations and weights ----------------------------------------------------------------------------------------------
def config(case: dict) -> dict:
    """The config.json of the model whose first layer the case runs (of the whole model for `llama`)."""
    kind, width = case["kind"], case["width"]
    if kind in ("attention", "llama"):
        return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": case.get("vocab", VOCAB), "hidden_size": width,
                "intermediate_size": case.get("ff", 256), "num_hidden_layers": case.get("layers", 1), "num_attention_heads": case["heads"],
                "num_key_value_heads": case["kv_heads"], "head_dim": case["dim"], "rms_norm_eps": EPS, "rope_theta": 500000.0,
                "max_position_embeddings": 8192, "hidden_act": "silu", "tie_word_embeddings": False}
    base = {"vocab": VOCAB, "width": width, "norm": {"eps": EPS}}
    if kind == "window":
        mixer = {"heads": case["heads"], "kv_heads": case["kv_heads"], "dim": case["dim"], "vdim": case["dim"], "scale": case["dim"] ** -0.5,
                 "mask": {"size": case["window"], "keep_first": case["keep"]}, "rot": {"dims": case["dim"], "base": 1e6, "scaling": YARN}}
        layer = {"type": "attention", "mixer": mixer, "mlp": None}
    elif kind == "delta":
        layer = {"type": "delta", "mlp": None, "mixer": {"heads": case["heads"], "kv_heads": case["kv_heads"], "dim": case["dim"], "vdim": case["dim"], "conv": TAPS}}
    if kind in ("window", "delta"):
        return {"architecture": "Dezolorn", **base, "layers": [layer], "loop": {"start": 0, "stop": 0, "times": 1}, "logit_scale": 1.0, "logit_softcap": 0.0}
    if kind == "latent":
        mixer = {"heads": case["heads"], "dim": case["dim"], "rot_dim": case["rot"], "vdim": case["dim"], "kv_rank": case["rank"],
                 "scale": (case["dim"] + case["rot"]) ** -0.5, "mask": {"size": case["window"]}, "rot": {"dims": case["rot"], "base": 1e6, "scaling": YARN}}
        return {"architecture": "Sorizen", **base, "embedding": {"scale": 1.0}, "layers": [{"type": "latent_attention_2", "mixer": mixer, "mlp": None}]}
    state = {"heads": case.get("heads", 8), "vdim": case.get("dim", 64), "state": case.get("state", 64), "groups": case.get("groups", 1), "conv": TAPS,
             "norm_groups": case.get("groups", 1)}
    mlp = None
    if kind == "experts":
        mlp = {"kind": "moe", "expert": {"ff": case["inter"]}, "shared": {"ff": case["shared"]},
               "router": {"experts": case["experts"], "identity": case["identity"], "top": case["top"], "scale": 2.0}}
    return {"architecture": "Rasezen", **base, "layers": [{"type": "mamba2", "mixer": state, "mlp": mlp}]}


def shapes(case: dict) -> dict[str, tuple]:
    """Checkpoint name -> (shape, standard deviation, mean, float32 in every mode?) of the layer under test (of all, for `llama`)."""
    kind, W = case["kind"], case["width"]
    fan = lambda *s: (s, s[-1] ** -0.5, 0.0, False)  # noqa: E731
    gain = lambda *s: (s, 0.1, 1.0, True)  # noqa: E731
    small = lambda std, *s: (s, std, 0.0, True)  # noqa: E731
    if kind in ("attention", "llama"):
        q, kv = case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
        out = {"model.embed_tokens.weight": ((case.get("vocab", VOCAB), W), 1.0, 0.0, False), "lm_head.weight": fan(case.get("vocab", VOCAB), W),
               "model.norm.weight": gain(W)}
        for i in range(case.get("layers", 1)):
            p, ff = f"model.layers.{i}.", case.get("ff", 256)
            out |= {p + "self_attn.q_proj.weight": fan(q, W), p + "self_attn.k_proj.weight": fan(kv, W), p + "self_attn.v_proj.weight": fan(kv, W),
                    p + "self_attn.o_proj.weight": fan(W, q), p + "mlp.gate_proj.weight": fan(ff, W), p + "mlp.up_proj.weight": fan(ff, W),
                    p + "mlp.down_proj.weight": fan(W, ff), p + "input_layernorm.weight": gain(W), p + "post_attention_layernorm.weight": gain(W)}
        return out
    m = "l0.mix."
    if kind == "window":
        q, kv = case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
        return {m + "q": fan(q, W), m + "k": fan(kv, W), m + "v": fan(kv, W), m + "o": fan(W, q), m + "q.norm": gain(q), m + "k.norm": gain(kv)}
    if kind == "latent":
        H, d, r, R = case["heads"], case["dim"], case["rot"], case["rank"]
        return {m + "q": fan(H * (d + r), W), m + "dkv": fan(R + r, W), m + "dkv.norm": gain(R), m + "uk": fan(H * d, R), m + "uv": fan(H * d, R),
                m + "g": fan(H, W), m + "o": fan(W, H * d)}
    if kind == "delta":
        qk, v, H = case["kv_heads"] * case["dim"], case["heads"] * case["dim"], case["heads"]
        return {m + "q": fan(qk, W), m + "k": fan(qk, W), m + "v": fan(v, W), m + "g": fan(v, W), m + "b": fan(H, W), m + "a": fan(H, W), m + "o": fan(W, v),
                m + "q.conv": small(0.5, qk, TAPS), m + "k.conv": small(0.5, qk, TAPS), m + "v.conv": small(0.5, v, TAPS), m + "A_log": small(0.5, H),
                m + "dt_bias": small(0.5, H), m + "norm": gain(case["dim"])}
    if kind == "mamba2":
        inner, gn, H = case["heads"] * case["dim"], 2 * case["groups"] * case["state"], case["heads"]
        return {m + "in": fan(2 * inner + gn + H, W), m + "conv": small(0.5, inner + gn, TAPS), m + "conv.b": small(0.1, inner + gn), m + "dt_bias": small(0.5, H),
                m + "A_log": small(0.5, H), m + "D": gain(H), m + "norm": gain(inner), m + "o": fan(W, inner)}
    p, E, f = "l0.mlp.", case["experts"], case["inter"]
    out = {p + "router": (((E + case["identity"]), W), W ** -0.5, 0.0, True), p + "correction": small(0.01, E + case["identity"]),
           p + "shared.gate": fan(case["shared"], W), p + "shared.up": fan(case["shared"], W), p + "shared.down": fan(W, case["shared"])}
    for e in range(E):
        out |= {f"{p}e{e}.gate": fan(f, W), f"{p}e{e}.up": fan(f, W), f"{p}e{e}.down": fan(W, f)}
    return out


def _dtype(case: dict) -> torch.dtype:
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _gen(seed: int, salt: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed * 1009 + salt)


def weights(case: dict, seed: int) -> dict[str, torch.Tensor]:
    """As a checkpoint holds them: rounded to bfloat16, then in the run's type (gains and small tensors in float32)."""
    g, out = _gen(seed, 1), {}
    for name, (shape, std, mean, f32) in sorted(shapes(case).items()):
        t = (torch.empty(shape, device="cuda").normal_(mean, std, generator=g)).to(torch.bfloat16)
        out[name] = t.float() if f32 else t.to(_dtype(case))
    return out


def activations(case: dict, seed: int, rows: int, salt: int) -> torch.Tensor:
    """Normed activations: about unit variance."""
    return torch.empty((rows, case["width"]), device="cuda").normal_(0.0, 1.0, generator=_gen(seed, salt)).to(_dtype(case))


def held(case: dict, seed: int, layer: int) -> list[tuple[torch.Tensor, ...]]:
    """What every request's earlier positions left in the cache: keys and values [positions, kv heads, dim], or latents."""
    g, out = _gen(seed, 7 + layer), []
    if case["kind"] == "latent":
        widths = [(1, case["rank"] + case["rot"])]
    else:
        widths = [(case["kv_heads"], case["dim"])] * 2
    for before, _ in lengths(case):
        out.append(tuple(torch.empty((before, *w), device="cuda").normal_(0.0, 1.0, generator=g).to(_dtype(case)) for w in widths))
    return out


def token_ids(case: dict, seed: int) -> list[list[int]]:
    rng = random.Random(seed)
    return [[rng.randrange(case.get("vocab", VOCAB)) for _ in range(n)] for _, n in lengths(case)]


# ---- what a program has in hand before the call ------------------------------------------------------------------------------------
class State:
    """The model, its runner with the cache, the step's context, its inputs, and for decoding the captured graph."""


def _has_cache(case: dict) -> bool:
    return case["kind"] in ("attention", "window", "latent", "llama")


def prepare(case: dict, seed: int) -> State:
    from nanospec_b200.engine import ModelRunner, StepEntry
    from nanospec_b200.weights import build_model

    s = State()
    s.case = case
    dtype = _dtype(case)
    s.model, _ = build_model(config(case), None, dtype, "cuda")
    w = weights(case, seed)
    for name, spec in s.model.weight_specs().items():  # parts of the model that the case does not run
        if name not in w:
            w[name] = torch.zeros(spec.shape, device="cuda", dtype=torch.float32 if spec.rule == "float32" else dtype)
    s.model.bind(w)
    del w
    lens = lengths(case)
    pages = sum(-(-(a + b + 1) // PAGE) + 1 for a, b in lens) + 8
    s.runner = ModelRunner(s.model, pages, PAGE, len(lens))
    s.ids = token_ids(case, seed)
    whole_prompt = case["kind"] == "llama" and case["tokens"] > 1
    if whole_prompt:
        s.entries = [StepEntry(i, ids, [len(ids) - 1]) for i, ids in enumerate(s.ids)]
        return s
    decode = case["tokens"] == 1
    for i in range(len(lens)):
        s.runner.begin(i)
    before = [StepEntry(i, [1] * a, []) for i, (a, _) in enumerate(lens) if a]
    part = s.model.blocks[0].feed_forward if case["kind"] == "experts" else s.model.blocks[0].mixer
    if before and case["kind"] != "experts":
        ctx, _, _ = s.runner.build_context(before)
        if _has_cache(case):  # earlier positions' keys and values, where the block tables say
            for layer in range(case.get("layers", 1)):
                lane, row = ctx.lanes[layer], 0
                table = lane.block_table.long()
                for (a, _), kept in zip(lens, held(case, seed, layer)):
                    if a == 0:
                        continue
                    at = torch.arange(a, device="cuda")
                    for store, values in zip((lane.k, lane.v), kept):
                        store[table[row, at // PAGE], :, at % PAGE] = values
                    row += 1
        else:             # a state is what walking the earlier positions leaves
            part.forward(activations(case, seed, ctx.n_tokens, 3), ctx, ctx.lanes[0])
    entries = [StepEntry(i, ids, [0] if case["kind"] == "llama" else []) for i, ids in enumerate(s.ids)]
    s.ctx, s.want, _ = s.runner.build_context(entries)
    s.x = activations(case, seed, s.ctx.n_tokens, 2) if case["kind"] != "llama" else None
    if case["kind"] == "llama":
        from nanospec_b200 import ops
        n = len(lens)
        s.logits = torch.empty((n, case["vocab"]), device="cuda")
        s.options = (torch.zeros(n, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda"), torch.ones(n, device="cuda"), torch.zeros(n, device="cuda"))

        def forward():
            hidden = s.model.forward(s.ctx, s.want)
            s.model.logits(hidden, s.logits)
            _, raw, _ = ops.sample_rows(s.logits, *s.options)
            return {"logits": s.logits, "log_probability": raw}
    elif case["kind"] == "experts":
        def forward():
            return {"y": part.forward(s.x, s.ctx)}
    elif _has_cache(case):
        def forward():
            y, lane = part.forward(s.x, s.ctx, s.ctx.lanes[0]), s.ctx.lanes[0]
            return {"y": y, "keys": lane.k, "values": lane.v}
    else:
        def forward():
            return {"y": part.forward(s.x, s.ctx, s.ctx.lanes[0]), "state": s.ctx.lanes[0].state}
    s.forward, s.graph = forward, None
    if decode:
        lane = s.ctx.lanes[0]
        kept = lane.state.clone() if lane.state is not None else None
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                forward()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            s.out = forward()
        if kept is not None:
            lane.state.copy_(kept)
    return s


def run(s: State):
    if s.case["kind"] == "llama" and s.case["tokens"] > 1:  # prompts come, run and go
        for e in s.entries:
            s.runner.begin(e.req_id)
        logits = s.runner.step(s.entries)
        for e in s.entries:
            s.runner.end(e.req_id)
        return {"logits": logits}
    if s.graph is not None:
        s.graph.replay()
        return s.out
    return s.forward()


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------------------
def _pairs(case: dict) -> tuple[int, int]:
    """(query-key pairs under the mask, positions of the cache that the step reads or writes)"""
    window, keep = case.get("window", 1 << 30), case.get("keep", 0)
    pairs = seen = 0
    for a, n in lengths(case):
        for p in range(a, a + n):
            pairs += min(p + 1, window) + max(0, min(keep, p + 1 - window))
        seen += min(a + n, window + n - 1 + keep)
    return pairs, seen


def work(case: dict) -> dict:
    kind, W = case["kind"], case["width"]
    size = 4 if case.get("dtype") == "float32" else 2
    N = sum(n for _, n in lengths(case))
    params = {k: math.prod(v[0]) for k, v in shapes(case).items()}
    if kind == "attention":
        params = {k: v for k, v in params.items() if "self_attn" in k}
    if kind in ("attention", "window", "llama"):
        pairs, seen = _pairs(case)
        L, per = case.get("layers", 1), case["kv_heads"] * case["dim"]
        read = size * 2 * per * seen * L
        flops = 4.0 * case["heads"] * case["dim"] * pairs * L
        if kind == "llama":
            R, V = case["requests"], case["vocab"]
            matrices = sum(v for k, v in params.items() if "embed" not in k and "lm_head" not in k and "norm" not in k)
            return {"bytes": size * (matrices + V * W + N * W) + read + 4.0 * R * V, "flops": flops + 2.0 * N * matrices + 2.0 * R * V * W}
        return {"bytes": size * (sum(params.values()) + 2 * N * W) + read, "flops": flops + 2.0 * N * sum(params.values())}
    if kind == "latent":
        pairs, seen = _pairs(case)
        H, d, r, R = case["heads"], case["dim"], case["rot"], case["rank"]
        unfold = params["l0.mix.uk"] + params["l0.mix.uv"]
        return {"bytes": size * (sum(params.values()) + 2 * N * W + seen * (R + r)),
                "flops": 2.0 * N * (sum(params.values()) - unfold) + 2.0 * seen * unfold + 2.0 * H * (2 * d + r) * pairs}
    if kind in ("delta", "mamba2"):
        entries = case["heads"] * case["dim"] * (case["dim"] if kind == "delta" else case["state"])
        return {"bytes": size * (sum(params.values()) + 2 * N * W) + 8.0 * case["requests"] * entries,
                "flops": 2.0 * N * sum(params.values()) + (7.0 if kind == "delta" else 5.0) * N * entries}
    E, f, top = case["experts"], case["inter"], case["top"]
    share = E / (E + case["identity"])  # of the choices that fall on experts with tensors
    chosen = E * (1.0 - (1.0 - top / (E + case["identity"])) ** N)
    return {"bytes": size * (3.0 * chosen * f * W + 3.0 * case["shared"] * W + 2 * N * W) + 4.0 * params["l0.mlp.router"],
            "flops": 2.0 * N * (3.0 * top * share * f * W + 3.0 * case["shared"] * W + params["l0.mlp.router"])}


def tolerance(case: dict) -> dict:
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 1e-4}  # measured against 64 bits: 1.2e-6 to 1.7e-6
    # bfloat16 activations between the products: about 2^-9 of each value, and 8 bits of the softmax weights
    # (measured against 64 bits: 0.003 to 0.005)
    return {"rel": 1.5e-2, "max": 0.3}


# ---- the same in 64 bits, in plain torch --------------------------------------------------------------------------------------------------
def _frequencies(dims: int, base: float, scaling: dict | None) -> tuple[torch.Tensor, float]:
    i = torch.arange(dims // 2, dtype=F64)
    f = base ** (-2.0 * i / dims)
    if scaling is None:
        return f.cuda(), 1.0
    turn = lambda n: dims * math.log(scaling["original"] / (2 * math.pi * n)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(turn(scaling["fast"])), 0), min(math.ceil(turn(scaling["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return (f / scaling["factor"] * ramp + f * (1 - ramp)).cuda(), 0.1 * math.log(scaling["factor"]) + 1.0


def _rotate(x: torch.Tensor, positions: torch.Tensor, base: float, scaling: dict | None, halves: bool) -> torch.Tensor:
    """x [T, heads, dim], every feature rotated: pairs (i, i + dim / 2) or (2i, 2i + 1)."""
    dims = x.shape[-1]
    f, mag = _frequencies(dims, base, scaling)
    a = (positions.double()[:, None] * f[None, :])[:, None, :]
    cos, sin = torch.cos(a) * mag, torch.sin(a) * mag
    out = torch.empty_like(x)
    first, second = (slice(0, dims // 2), slice(dims // 2, dims)) if halves else (slice(0, dims, 2), slice(1, dims, 2))
    out[..., first] = x[..., first] * cos - x[..., second] * sin
    out[..., second] = x[..., second] * cos + x[..., first] * sin
    return out


def _attend(q, k, v, first: int, scale: float, window: int = 1 << 30, keep: int = 0) -> torch.Tensor:
    """q [T, H, d] at positions from `first` on, k [S, G, d], v [S, G, dv] -> [T, H * dv]."""
    T, H, _ = q.shape
    S, G, _ = k.shape
    i, j = torch.arange(first, first + T, device="cuda")[:, None], torch.arange(S, device="cuda")[None, :]
    mask = (j <= i) & ((i - j < window) | (j < keep))
    out = torch.empty((T, H, v.shape[2]), dtype=F64, device="cuda")
    for h in range(H):
        g = h // (H // G)
        out[:, h] = torch.softmax(((q[:, h] @ k[:, g].T) * scale).masked_fill(~mask, -math.inf), dim=-1) @ v[:, g]
    return out.reshape(T, -1)


def _rms(x: torch.Tensor) -> torch.Tensor:
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _silu(x: torch.Tensor) -> torch.Tensor:
    return x * torch.sigmoid(x)


def _conv(x: torch.Tensor, taps: torch.Tensor) -> torch.Tensor:
    n = taps.shape[1]
    padded = torch.cat([torch.zeros((n - 1, x.shape[1]), dtype=F64, device="cuda"), x])
    return sum(padded[j: j + x.shape[0]] * taps[:, j] for j in range(n))


def _llama_attention(x, w, p, case, first, k0, v0):
    T, H, G, d = x.shape[0], case["heads"], case["kv_heads"], case["dim"]
    at = torch.arange(first, first + T, device="cuda")
    q = _rotate((x @ w[p + "q_proj.weight"].T).view(T, H, d), at, 500000.0, None, True)
    k = _rotate((x @ w[p + "k_proj.weight"].T).view(T, G, d), at, 500000.0, None, True)
    k, v = torch.cat([k0, k]), torch.cat([v0, (x @ w[p + "v_proj.weight"].T).view(T, G, d)])
    return _attend(q, k, v, first, d ** -0.5) @ w[p + "o_proj.weight"].T


def _window(x, w, case, first, k0, v0):
    T, H, G, d, m = x.shape[0], case["heads"], case["kv_heads"], case["dim"], "l0.mix."
    at = torch.arange(first, first + T, device="cuda")
    q = _rotate((_rms(x @ w[m + "q"].T) * w[m + "q.norm"]).view(T, H, d), at, 1e6, YARN, False)
    k = _rotate((_rms(x @ w[m + "k"].T) * w[m + "k.norm"]).view(T, G, d), at, 1e6, YARN, False)
    k, v = torch.cat([k0, k]), torch.cat([v0, (x @ w[m + "v"].T).view(T, G, d)])
    return _attend(q, k, v, first, d ** -0.5, case["window"], case["keep"]) @ w[m + "o"].T


def _latent(x, w, case, first, c0):
    T, H, d, r, R, m = x.shape[0], case["heads"], case["dim"], case["rot"], case["rank"], "l0.mix."
    at = torch.arange(first, first + T, device="cuda")
    q = (x @ w[m + "q"].T).view(T, H, d + r)
    dkv = x @ w[m + "dkv"].T
    c = torch.cat([c0[:, 0, :R], _rms(dkv[:, :R]) * w[m + "dkv.norm"]])
    kr = torch.cat([c0[:, 0, R:], _rotate(dkv[:, None, R:], at, 1e6, YARN, False)[:, 0]])
    k = torch.cat([(c @ w[m + "uk"].T).view(-1, H, d), kr[:, None, :].expand(-1, H, r)], dim=-1)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], at, 1e6, YARN, False)], dim=-1)
    out = _attend(q, k, (c @ w[m + "uv"].T).view(-1, H, d), first, (d + r) ** -0.5, case["window"]).view(T, H, d)
    return (out * torch.sigmoid(x @ w[m + "g"].T)[:, :, None]).reshape(T, H * d) @ w[m + "o"].T


def _delta(x, w, case):
    """x: every position from the sequence's start."""
    T, H, G, d, m = x.shape[0], case["heads"], case["kv_heads"], case["dim"], "l0.mix."
    q, k, v = (_silu(_conv(x @ w[m + n].T, w[m + n + ".conv"])).view(T, -1, d) for n in ("q", "k", "v"))
    q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5).repeat_interleave(H // G, dim=1)
    k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1)
    beta = torch.sigmoid(x @ w[m + "b"].T)
    g = torch.exp(-torch.exp(w[m + "A_log"]) * torch.nn.functional.softplus(x @ w[m + "a"].T + w[m + "dt_bias"]))
    S, out = torch.zeros((H, d, d), dtype=F64, device="cuda"), torch.empty((T, H, d), dtype=F64, device="cuda")
    for t in range(T):
        S = g[t][:, None, None] * S
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None, :], S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.bmm(q[t][:, None, :], S)[:, 0]
    return ((_rms(out) * w[m + "norm"]).reshape(T, H * d) * _silu(x @ w[m + "g"].T)) @ w[m + "o"].T


def _mamba2(x, w, case):
    T, H, V, n, G, m = x.shape[0], case["heads"], case["dim"], case["state"], case["groups"], "l0.mix."
    inner = H * V
    p = x @ w[m + "in"].T
    z, xbc, dt = p[:, :inner], p[:, inner: 2 * inner + 2 * G * n], p[:, 2 * inner + 2 * G * n: 2 * inner + 2 * G * n + H]
    xbc = _silu(_conv(xbc, w[m + "conv"]) + w[m + "conv.b"])
    u = xbc[:, :inner].reshape(T, H, V)
    B = xbc[:, inner: inner + G * n].reshape(T, G, n).repeat_interleave(H // G, dim=1)
    C = xbc[:, inner + G * n:].reshape(T, G, n).repeat_interleave(H // G, dim=1)
    dt = torch.nn.functional.softplus(dt + w[m + "dt_bias"])
    decay = torch.exp(-torch.exp(w[m + "A_log"]) * dt)
    S, y = torch.zeros((H, n, V), dtype=F64, device="cuda"), torch.empty((T, H, V), dtype=F64, device="cuda")
    for t in range(T):
        S = decay[t][:, None, None] * S + (dt[t][:, None] * B[t])[:, :, None] * u[t][:, None, :]
        y[t] = torch.bmm(C[t][:, None, :], S)[:, 0] + w[m + "D"][:, None] * u[t]
    y = (y.reshape(T, inner) * _silu(z)).view(T, G, inner // G)
    return (_rms(y).reshape(T, inner) * w[m + "norm"]) @ w[m + "o"].T


def _experts(x, w, case):
    p, E = "l0.mlp.", case["experts"]
    unit = lambda h, name: (_silu(h @ w[name + "gate"].T) * (h @ w[name + "up"].T)) @ w[name + "down"].T  # noqa: E731
    score = torch.softmax(x @ w[p + "router"].T, dim=-1)
    chosen = torch.topk(score + w[p + "correction"], case["top"], dim=-1).indices
    weight = torch.zeros_like(score).scatter(1, chosen, score.gather(1, chosen) * 2.0)
    y = unit(x, p + "shared.") + weight[:, E:].sum(1, keepdim=True) * x
    for e in range(E):
        rows = weight[:, e].nonzero()[:, 0]
        if rows.numel():
            y[rows] += weight[rows, e, None] * unit(x[rows], f"{p}e{e}.")
    return y


def _llama(case, seed, w):
    per = [held(case, seed, layer) for layer in range(case["layers"])]
    rows = []
    for r, ((first, _), ids) in enumerate(zip(lengths(case), token_ids(case, seed))):
        x = w["model.embed_tokens.weight"][torch.tensor(ids, device="cuda")].double()
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            k0, v0 = (t.double() for t in per[i][r])
            x = x + _llama_attention(_rms(x) * w[p + "input_layernorm.weight"], w, p + "self_attn.", case, first, k0, v0)
            h = _rms(x) * w[p + "post_attention_layernorm.weight"]
            x = x + (_silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
        rows.append((_rms(x[-1:]) * w["model.norm.weight"]) @ w["lm_head.weight"].T)
    return torch.cat(rows)


def exact(case: dict, seed: int):
    w = {k: v if k == "model.embed_tokens.weight" else v.double() for k, v in weights(case, seed).items()}
    kind, lens = case["kind"], lengths(case)
    if kind == "llama":
        logits = _llama(case, seed, w)
        return {"logits": logits} if case["tokens"] > 1 else {"logits": logits, "log_probability": logits.amax(-1) - torch.logsumexp(logits, dim=-1)}
    xs = activations(case, seed, sum(n for _, n in lens), 2).double().split([n for _, n in lens])
    if kind == "experts":
        return {"y": _experts(torch.cat(xs), w, case)}
    if kind in ("delta", "mamba2"):
        # (the state that a step leaves has the mixer's own layout and no counterpart here)
        walk = _delta if kind == "delta" else _mamba2
        early = activations(case, seed, sum(a for a, _ in lens), 3).double().split([a for a, _ in lens])
        return {"y": torch.cat([walk(torch.cat([e, x]), w, case)[-x.shape[0]:] for e, x in zip(early, xs)]), "state": None}
    ys = []
    for x, (first, _), kept in zip(xs, lens, held(case, seed, 0)):
        kept = [t.double() for t in kept]
        if kind == "attention":
            ys.append(_llama_attention(x, w, "model.layers.0.self_attn.", case, first, *kept))
        elif kind == "window":
            ys.append(_window(x, w, case, first, *kept))
        else:
            ys.append(_latent(x, w, case, first, *kept))
    # (the cache's pages are laid out by the manager and have no counterpart here; y is computed from them)
    return {"y": torch.cat(ys), "keys": None, "values": None}
