"""What the library is measured by: the calls a program that serves or scores with it makes.

A case is a dict of plain values with one of four kinds:

``step``   ``Engine.step`` with one token per sequence behind a filled cache (a decode step), logits for all;
``serve``  a whole request: slots taken, unequal prompts in one step, a few decode steps, slots given back;
``layer``  one mixer, or one whole pre-norm block, over prompts of unequal lengths, with a cache of its own;
``ffn``    one feed-forward over the tokens of a step.

Layer sizes are those of the benchmark's shapes and of the runs of one design beside another in
``bench.py``; sequence lengths are the ranges served there.  ``exact`` restates every part in plain torch at 64 bits.
"""
import math

import torch
import torch.nn.functional as F

DEV = torch.device("cuda:0")
EPS = 1e-6
THETA = 1e6
ROUTED = {"n_groups": 4, "keep_groups": 2}


# ---- the cases ---------------------------------------------------------------------------------------------------

def listed():
    return [
        # one user, one token at a time: launches and latency count, the weights are read once
        dict(name="qwen_step_b1", kind="step", mixer="attention", dtype="bf16", width=2560, heads=32, kv=8, dim=128, inner=9728,
             vocab=32768, layers=2, batch=1, lo=700, hi=700),
        # a full batch near the end of a 4,096-token context: reading keys and values
        dict(name="qwen_step_b64_long", kind="step", mixer="attention", dtype="bf16", width=2560, heads=32, kv=8, dim=128, inner=9728,
             vocab=32768, layers=1, batch=64, lo=3900, hi=4090),
        # requests as they arrive: prompts of 64 to 2,048 tokens, then single-token steps
        dict(name="qwen_serve_b16", kind="serve", mixer="attention", dtype="bf16", width=2560, heads=32, kv=8, dim=128, inner=9728,
             vocab=32768, layers=2, batch=16, lo=64, hi=2048, steps=8),
        # the benchmark's prompt, one block of it
        dict(name="qwen_block_prompt", kind="layer", part="block", mixer="attention", dtype="bf16", width=2560, heads=32, kv=8, dim=128,
             inner=9728, seqs=1, lo=2048, hi=2048),
        # the float32 run: what outputs are checked against, and what a user who needs the bits runs
        dict(name="qwen_block_float32", kind="layer", part="block", mixer="attention", dtype="fp32", width=2560, heads=32, kv=8, dim=128,
             inner=9728, seqs=4, lo=60, hi=507),
        # linear attention with a decay per head (Datasun), unequal prompts
        dict(name="lightning_prompts", kind="layer", part="mixer", mixer="lightning", dtype="bf16", width=2560, heads=32, dim=128, vdim=128,
             seqs=3, lo=301, hi=2048),
        # the state-space layer (Bepilorn), one long prompt
        dict(name="state_space_prompt", kind="layer", part="mixer", mixer="state_space", dtype="bf16", width=2560, heads=32, dim=128, vdim=128,
             kv=8, seqs=1, lo=2048, hi=2048),
        # gated linear attention (Bepilorn), unequal prompts
        dict(name="gated_linear_prompts", kind="layer", part="mixer", mixer="gated_linear", dtype="bf16", width=2048, heads=16, dim=128,
             vdim=128, seqs=4, lo=130, hi=1500),
        # latent attention (Munerax, and the layer kind of Kikelorn and Zitezen), the prompt
        dict(name="latent_prompt", kind="layer", part="mixer", mixer="latent", dtype="bf16", width=2048, heads=16, dim=64, rot=64, vdim=128,
             rank=512, seqs=1, lo=2048, hi=2048),
        # ... and single tokens of a full batch behind a long context
        dict(name="latent_step_b64", kind="step", mixer="latent", dtype="bf16", width=2048, heads=16, dim=64, rot=64, vdim=128, rank=512,
             inner=6144, vocab=32768, layers=1, batch=64, lo=3900, hi=4090),
        # the routed feed-forward (Bepilorn) over a prompt
        dict(name="experts_prompt", kind="ffn", part="ffn", dtype="bf16", width=2048, inner=1024, shared=2048, experts=16, top=4, tokens=2048),
        # a recurrent model served: short prompts, then single-token steps
        dict(name="state_space_serve_b8", kind="serve", mixer="state_space", dtype="bf16", width=2048, heads=16, dim=128, vdim=128, kv=4,
             inner=6144, vocab=32768, layers=2, batch=8, lo=33, hi=500, steps=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _span(rng, lo, hi):
    a, b = _log(rng, lo, hi), _log(rng, lo, hi)
    return min(a, b), max(a, b)


def draw(rng):
    """The kinds of the list at other sizes: the three widths of the design runs, whole and odd lengths, one sequence to a full batch."""
    width, heads, kv, inner = rng.choice([(2048, 16, 4, 6144), (2560, 32, 8, 9728), (1000, 12, 2, 2728)])
    what = rng.choice(["step", "step_latent", "serve", "block", "block32", "lightning", "state_space", "gated_linear", "latent", "ffn",
                       "serve_ssm"])
    base = dict(dtype="bf16", width=width, heads=heads)
    if what in ("step", "step_latent"):
        batch = _log(rng, 1, 64)
        lo, hi = _span(rng, 20, 4090)
        more = dict(base, kind="step", inner=inner, vocab=32768, layers=1, batch=batch, lo=lo, hi=hi)
        if what == "step":
            return dict(more, mixer="attention", kv=kv, dim=rng.choice([64, 128]))
        return dict(more, mixer="latent", dim=64, rot=64, vdim=128, rank=512)
    if what in ("serve", "serve_ssm"):
        lo, hi = _span(rng, 10, 1500)
        more = dict(base, kind="serve", inner=inner, vocab=32768, layers=1, batch=_log(rng, 1, 16), lo=lo, hi=hi, steps=8, kv=kv, dim=128)
        if what == "serve":
            return dict(more, mixer="attention")
        return dict(more, mixer="state_space", vdim=rng.choice([64, 128]))
    if what == "ffn":
        return dict(kind="ffn", part="ffn", dtype="bf16", width=width, inner=rng.choice([344, 1024]), shared=rng.choice([0, 1024]), experts=16,
                    top=4, tokens=_log(rng, 1, 2048))
    lo, hi = _span(rng, 10, 2000)
    more = dict(base, kind="layer", seqs=rng.randint(1, 3), lo=lo, hi=hi)
    if what == "block":
        return dict(more, part="block", mixer="attention", kv=kv, dim=rng.choice([64, 128]), inner=inner)
    if what == "block32":
        return dict(more, part="block", mixer="attention", kv=kv, dim=rng.choice([64, 128]), inner=inner, dtype="fp32", seqs=1)
    if what == "latent":
        return dict(more, part="mixer", mixer="latent", dim=64, rot=64, vdim=128, rank=rng.choice([256, 512]))
    return dict(more, part="mixer", mixer=what, dim=rng.choice([64, 128]), vdim=rng.choice([64, 128]), kv=kv)


# ---- sizes, weights and inputs -----------------------------------------------------------------------------------

def _lengths(case):
    n = case.get("batch", case.get("seqs", 1))
    lo, hi = case["lo"], case["hi"]
    return [hi - (hi - lo) * i // max(n - 1, 1) for i in range(n)]


def _mixer_shapes(c):
    """Name -> (shape, how it is filled)."""
    w, a = c["width"], c["heads"]
    if c["mixer"] == "attention":
        d, kv = c["dim"], c["kv"]
        return {"q_proj": ((a * d, w), "matrix"), "k_proj": ((kv * d, w), "matrix"), "v_proj": ((kv * d, w), "matrix"),
                "o_proj": ((w, a * d), "matrix"), "q_norm": ((d,), "norm"), "k_norm": ((d,), "norm")}
    if c["mixer"] == "latent":
        d, rd, dv, r = c["dim"], c["rot"], c["vdim"], c["rank"]
        return {"q_proj": ((a * (d + rd), w), "matrix"), "dkv_proj": ((r + rd, w), "matrix"), "dkv_norm": ((r,), "norm"),
                "uk_proj": ((a * d, r), "matrix"), "uv_proj": ((a * dv, r), "matrix"), "o_proj": ((w, a * dv), "matrix"),
                "sink": ((a,), "unit"), "g_proj": ((a, w), "matrix")}
    qk, vv = a * c["dim"], a * c["vdim"]
    if c["mixer"] == "lightning":
        return {"q_proj": ((qk, w), "matrix"), "k_proj": ((qk, w), "matrix"), "v_proj": ((vv, w), "matrix"), "g_proj": ((vv, w), "matrix"),
                "o_proj": ((w, vv), "matrix"), "norm": ((vv,), "norm")}
    if c["mixer"] == "gated_linear":
        return {"q_proj": ((qk, w), "matrix"), "k_proj": ((qk, w), "matrix"), "v_proj": ((vv, w), "matrix"), "g_proj": ((vv, w), "matrix"),
                "a1_proj": ((64, w), "matrix"), "a2_proj": ((qk, 64), "matrix"), "a2_proj.bias": ((qk,), "unit"),
                "o_proj": ((w, vv), "matrix"), "norm": ((c["vdim"],), "norm")}
    gn = c["kv"] * c["dim"]
    ch = vv + 2 * gn
    return {"in_proj": ((2 * vv + 2 * gn + a, w), "matrix"), "conv": ((ch, 4), "matrix"), "conv.bias": ((ch,), "small"),
            "dt_bias": ((a,), "dt"), "A_log": ((a,), "rate"), "D": ((a,), "norm"), "norm": ((vv,), "norm"), "o_proj": ((w, vv), "matrix")}


def _mlp_shapes(c):
    w, f = c["width"], c["inner"]
    return {"gate_proj": ((f, w), "matrix"), "up_proj": ((f, w), "matrix"), "down_proj": ((w, f), "matrix")}


def _ffn_shapes(c):
    w, f, s = c["width"], c["inner"], c["shared"]
    out = {"router": ((c["experts"], w), "matrix"), "correction": ((c["experts"],), "small")}
    for e in range(c["experts"]):
        out.update({f"experts.{e}.gate_proj": ((f, w), "matrix"), f"experts.{e}.up_proj": ((f, w), "matrix"),
                    f"experts.{e}.down_proj": ((w, f), "matrix")})
    if s:
        out.update({"shared.gate_proj": ((s, w), "matrix"), "shared.up_proj": ((s, w), "matrix"), "shared.down_proj": ((w, s), "matrix"),
                    "shared.gate": ((1, w), "matrix")})
    return out


def _block_shapes(c):
    out = {"norm1.weight": ((c["width"],), "norm"), "norm2.weight": ((c["width"],), "norm")}
    out.update({"mixer." + k: v for k, v in _mixer_shapes(c).items()})
    out.update({"ffn." + k: v for k, v in _mlp_shapes(c).items()})
    return out


def _dtype(c):
    return torch.float32 if c["dtype"] == "fp32" else torch.bfloat16


def _filled(shapes, dtype, g):
    out = {}
    for name, (shape, how) in shapes.items():
        t = torch.randn(shape, generator=g, device=DEV)
        if how == "matrix":
            t *= shape[1] ** -0.5
        elif how == "table":
            t *= 0.5
        elif how == "norm":
            t = 1 + 0.1 * t
        elif how == "small":
            t *= 0.1
        elif how in ("dt", "rate"):
            u = torch.rand(shape, generator=g, device=DEV)
            # Mamba-2's own starting values: steps of 0.001 to 0.1 spread over their logarithm, rates of 1 to 16
            t = torch.log(torch.expm1(torch.exp(math.log(1e-3) + u * math.log(100.0)))) if how == "dt" else torch.log(1 + 15 * u)
        out[name] = t.to(dtype)
    return out


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(1000 + seed)


def _weights(case, seed):
    """The tensors of a case and the generator that its inputs are drawn from next."""
    g = _generator(seed)
    if case["kind"] == "ffn":
        return _filled(_ffn_shapes(case), _dtype(case), g), g
    if case["kind"] == "layer":
        return _filled(_block_shapes(case) if case["part"] == "block" else _mixer_shapes(case), _dtype(case), g), g
    shapes = {"embed": ((case["vocab"], case["width"]), "table"), "final": ((case["width"],), "norm"),
              "head": ((case["vocab"], case["width"]), "matrix")}
    for i in range(case["layers"]):
        shapes.update({f"l{i}.{k}": v for k, v in _block_shapes(case).items()})
    return _filled(shapes, _dtype(case), g), g


def _tokens(case, g):
    """Every sequence's prompt and the tokens that follow it."""
    n = _lengths(case)
    more = case.get("steps", 1)
    ids = torch.randint(0, case["vocab"], (sum(n) + more * len(n),), generator=g, device=DEV).tolist()
    out, at = [], 0
    for k in n:
        out.append((ids[at:at + k], ids[at + k:at + k + more]))
        at += k + more
    return out


def _rows(case, g):
    """The input rows of a part alone: the residual stream for a block, a normed row for a mixer or a feed-forward."""
    n = case["tokens"] if case["kind"] == "ffn" else sum(_lengths(case))
    x = torch.randn((n, case["width"]), generator=g, device=DEV)
    return x if case["part"] == "block" else x.to(_dtype(case))


def _decays(heads):
    return [1.0 - 2.0 ** -(5.0 + 3.0 * i / max(heads - 1, 1)) for i in range(heads)]


# ---- what a program keeps, and the call ---------------------------------------------------------------------------

def _mixer_spec(c):
    from builderforce_inference_b200.parts import PartSpec
    w, a = c["width"], c["heads"]
    if c["mixer"] == "attention":
        return PartSpec("attention", {"width": w, "n_heads": a, "n_kv_heads": c["kv"], "head_dim": c["dim"], "qk_norm": True, "eps": EPS,
                                      "position": PartSpec("rotary", {"theta": THETA, "rot_dim": c["dim"]})})
    if c["mixer"] == "latent":
        return PartSpec("latent_attention", {"width": w, "n_heads": a, "dim": c["dim"], "rot_dim": c["rot"], "v_dim": c["vdim"],
                                             "kv_rank": c["rank"], "eps": EPS, "sink": "learned", "gate": True,
                                             "position": PartSpec("rotary", {"theta": THETA, "rot_dim": c["rot"]})})
    if c["mixer"] == "lightning":
        return PartSpec("lightning", {"width": w, "n_heads": a, "dim": c["dim"], "vdim": c["vdim"], "decay": _decays(a), "eps": EPS})
    if c["mixer"] == "gated_linear":
        return PartSpec("gated_linear", {"width": w, "n_heads": a, "dim": c["dim"], "vdim": c["vdim"], "tau": 8.0, "decay_rank": 64, "eps": EPS})
    return PartSpec("state_space", {"width": w, "n_heads": a, "vdim": c["vdim"], "state": c["dim"], "groups": c["kv"], "conv_taps": 4,
                                    "norm_groups": c["kv"], "eps": EPS})


def _block_spec(c):
    from builderforce_inference_b200.parts import PartSpec
    norm = PartSpec("rms", {"width": c["width"], "eps": EPS})
    return PartSpec("prenorm", {"norm1": norm, "mixer": _mixer_spec(c), "norm2": norm,
                                "ffn": PartSpec("gated_mlp", {"width": c["width"], "inner": c["inner"]})})


def _prepare_engine(case, seed):
    from builderforce_inference_b200.engine.engine import Engine, SequenceStep
    from builderforce_inference_b200.parts import LayerSpec, ModelSpec, PartSpec, RunSpec
    w, g = _weights(case, seed)
    n = _lengths(case)
    longest = max(n) + case.get("steps", 1)
    layers = [LayerSpec(_block_spec(case), {k: f"l{i}.{k}" for k in _block_shapes(case)}) for i in range(case["layers"])]
    spec = ModelSpec(vocab_size=case["vocab"], width=case["width"], embedding_name="embed", layers=layers,
                     schedule=[RunSpec(i) for i in range(case["layers"])], final_norm=PartSpec("rms", {"width": case["width"], "eps": EPS}),
                     final_norm_names={"weight": "final"}, head_name="head", max_positions=longest)
    eng = Engine(spec, w, _dtype(case), DEV, max_tokens=sum((k + case.get("steps", 1) + 63) // 64 * 64 for k in n))
    seqs = _tokens(case, g)
    state = {"kind": case["kind"], "engine": eng, "seqs": seqs, "Step": SequenceStep}
    if case["kind"] == "step":
        state["slots"] = [eng.acquire() for _ in n]
        eng.step([SequenceStep(s, p, ()) for s, (p, _) in zip(state["slots"], seqs)])
        state["lengths"] = n
    return state


def _prepare_layer(case, seed):
    from builderforce_inference_b200.cache import SequenceCache
    from builderforce_inference_b200.engine.context import Workspace, build_context
    from builderforce_inference_b200.engine.decoder import Runtime
    from builderforce_inference_b200.parts import BLOCKS, MIXERS
    dt, n = _dtype(case), _lengths(case)
    w, g = _weights(case, seed)
    rt, ws = Runtime(DEV, dt), Workspace(DEV)
    block = case["part"] == "block"
    part = BLOCKS.build(_block_spec(case)) if block else MIXERS.build(_mixer_spec(case))
    part.load_all(w, rt)
    (part.mixer() if block else part).prepare(rt, max(n))
    cache = SequenceCache([part.cache_need()], [None], sum((k + 63) // 64 * 64 for k in n), max(n), dt, DEV)
    slots = [cache.acquire() for _ in n]
    ctx = build_context([(s, 0, range(k)) for s, k in zip(slots, n)], dt, ws, DEV)      # the parts read no token ids
    for s in slots:
        cache.release(s)
    x = _rows(case, g)
    return {"kind": "layer", "block": block, "part": part, "cache": cache, "slots": slots, "counts": n, "ctx": ctx, "x": x,
            "out": torch.empty((sum(n), case["width"]), dtype=torch.float32, device=DEV)}


def _prepare_ffn(case, seed):
    from builderforce_inference_b200.engine.context import Workspace, build_context
    from builderforce_inference_b200.engine.decoder import Runtime
    from builderforce_inference_b200.parts import FEED_FORWARDS, PartSpec
    w, g = _weights(case, seed)
    part = FEED_FORWARDS.build(PartSpec("mixture_of_experts", dict(ROUTED, width=case["width"], n_experts=case["experts"], top=case["top"],
                                                                   inner=case["inner"], shared_inner=case["shared"] or None)))
    part.load_all(w, Runtime(DEV, _dtype(case)))
    x = _rows(case, g)
    ctx = build_context([(0, 0, range(case["tokens"]))], _dtype(case), Workspace(DEV), DEV)
    return {"kind": "ffn", "part": part, "ctx": ctx, "x": x, "out": torch.empty((case["tokens"], case["width"]), dtype=torch.float32, device=DEV)}


def prepare(case, seed):
    if case["kind"] == "ffn":
        return _prepare_ffn(case, seed)
    return _prepare_layer(case, seed) if case["kind"] == "layer" else _prepare_engine(case, seed)


def run(state):
    if state["kind"] == "ffn":
        state["part"].forward_store(state["ctx"], state["x"], state["out"])
        return state["out"]
    if state["kind"] == "layer":
        cache, slots = state["cache"], state["slots"]
        for _ in slots:
            cache.acquire()                       # lowest first: the slots that the context names
        cache.begin_step(slots, state["counts"])
        here = cache.run_cache(0)
        if state["block"]:
            state["out"].copy_(state["x"])        # the stream is renewed in place
            state["part"].forward(state["ctx"], state["out"], here)
        else:
            state["part"].forward_store(state["ctx"], state["x"], state["out"], here)
        cache.end_step(slots, state["counts"])
        for s in slots:
            cache.release(s)
        kept = [e[:len(slots)] for e in here.entries if isinstance(e, torch.Tensor)]     # a recurrence's state after the step
        return [state["out"]] + kept
    eng, Step = state["engine"], state["Step"]
    if state["kind"] == "step":
        out = eng.step([Step(s, t, (0,)) for s, (_, t) in zip(state["slots"], state["seqs"])], check=False)
        for s, n in zip(state["slots"], state["lengths"]):
            eng.rewind(s, n)                      # the next pass scores a token at the same place
        return out
    slots = [eng.acquire() for _ in state["seqs"]]
    got = [eng.step([Step(s, p, (len(p) - 1,)) for s, (p, _) in zip(slots, state["seqs"])], check=False).clone()]
    for i in range(len(state["seqs"][0][1])):
        got.append(eng.step([Step(s, (t[i],), (0,)) for s, (_, t) in zip(slots, state["seqs"])], check=False).clone())
    for s in slots:
        eng.release(s)
    return got


# ---- the work of a pass, and how far another correct implementation may be --------------------------------------

def _count(shapes):
    return sum(math.prod(s) for s, _ in shapes.values())


def _mixing(c, new, held):
    """Operations of the mixer beside its products for ``new`` tokens behind ``held`` earlier ones, and the cache's values read."""
    pairs = new * held + new * (new + 1) // 2
    if c["mixer"] == "attention":
        return 4 * c["heads"] * c["dim"] * pairs, 2 * c["kv"] * c["dim"] * (held + new)
    if c["mixer"] == "latent":
        return 2 * c["heads"] * (2 * c["rank"] + c["rot"]) * pairs, (c["rank"] + c["rot"]) * (held + new)
    return 6 * c["heads"] * c["dim"] * c["vdim"] * new, 0


def work(case):
    b = 4 if case["dtype"] == "fp32" else 2
    if case["kind"] == "ffn":
        n, w, f, s = case["tokens"], case["width"], case["inner"], case["shared"]
        used = min(case["experts"], n * case["top"])
        return {"bytes": b * (3 * w * (f * used + s) + case["experts"] * w) + (b + 4) * n * w,
                "flops": 2 * n * (3 * w * (f * case["top"] + s) + case["experts"] * w)}
    n = _lengths(case)
    state = 0 if case["mixer"] in ("attention", "latent") else 4 * case["heads"] * case["dim"] * case["vdim"]
    if case["kind"] == "layer":
        shapes = _block_shapes(case) if case["part"] == "block" else _mixer_shapes(case)
        return {"bytes": b * _count(shapes) + sum(n) * case["width"] * ((4 if case["part"] == "block" else b) + 4) + state * len(n),
                "flops": 2 * _count(shapes) * sum(n) + sum(_mixing(case, k, 0)[0] for k in n)}
    block = _count(_block_shapes(case)) * case["layers"]
    head = case["vocab"] * case["width"]
    steps = case.get("steps", 1)
    weights, cached, flops = 0, 0, 0
    if case["kind"] == "serve":
        weights += block + head
        flops += 2 * block * sum(n) + 2 * head * len(n) + case["layers"] * sum(_mixing(case, k, 0)[0] for k in n)
        cached += state * len(n) * case["layers"]
    for i in range(steps):
        weights += block + head
        flops += 2 * (block + head) * len(n)
        for k in n:
            f, v = _mixing(case, 1, k + i)
            flops += case["layers"] * f
            cached += case["layers"] * (b * v + 2 * state)
    passes = steps + (1 if case["kind"] == "serve" else 0)
    return {"bytes": b * weights + cached + 4 * passes * len(n) * case["vocab"], "flops": flops}


def tolerance(case):
    # four times the distance from exact(): 1.3e-6 in float32; in bfloat16 0.0016 to 0.0047 for one layer,
    # 0.0038 to 0.0069 for logits
    if case["dtype"] == "fp32":
        return {"rel": 5e-6, "max": 1e-3}
    return {"rel": 1.6e-2 if case["kind"] in ("layer", "ffn") else 2.5e-2, "max": 0.3}


# ---- the same in plain torch, 64 bits ---------------------------------------------------------------------------

def _rms(x, w=None):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _turn(x, first=0):
    """Rotate-half over the last dimension of ``[tokens, heads, d]``, positions from ``first``."""
    n, _, d = x.shape
    freq = THETA ** (-2.0 * torch.arange(d // 2, device=DEV, dtype=torch.float64) / d)
    ang = torch.arange(first, first + n, device=DEV, dtype=torch.float64)[:, None] * freq
    cos, sin = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    a, b = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _softmax_rows(q, k, v, scale, last, sink=None):
    """Causal attention of one head; ``last``: the number of final queries wanted."""
    n = k.shape[0]
    out = []
    for at in range(n - last, n, 1024):
        rows = q[at - (n - last):min(at + 1024, n) - (n - last)]
        s = rows @ k[:at + rows.shape[0]].T * scale
        mask = torch.arange(at + rows.shape[0], device=DEV)[None] > torch.arange(at, at + rows.shape[0], device=DEV)[:, None]
        s = s.masked_fill(mask, float("-inf"))
        m = s.amax(-1, keepdim=True)
        if sink is not None:
            m = torch.maximum(m, sink)
        e = torch.exp(s - m)
        z = e.sum(-1, keepdim=True)
        if sink is not None:
            z = z + torch.exp(sink - m)
        out.append(e @ v[:at + rows.shape[0]] / z)
    return torch.cat(out)


def _mix(c, w, h, last):
    """One sequence through a mixer: its output for the last ``last`` tokens, and what its state holds then."""
    n, a = h.shape[0], c["heads"]
    hq = h[n - last:]
    if c["mixer"] == "attention":
        d, kv = c["dim"], c["kv"]
        q = _turn(_rms((hq @ w["q_proj"].T).view(last, a, d), w["q_norm"]), n - last)
        k = _turn(_rms((h @ w["k_proj"].T).view(n, kv, d), w["k_norm"]))
        v = (h @ w["v_proj"].T).view(n, kv, d)
        o = torch.cat([_softmax_rows(q[:, i], k[:, i * kv // a], v[:, i * kv // a], d ** -0.5, last) for i in range(a)], dim=1)
        return o @ w["o_proj"].T, []
    if c["mixer"] == "latent":
        d, rd, dv, r = c["dim"], c["rot"], c["vdim"], c["rank"]
        q = (hq @ w["q_proj"].T).view(last, a, d + rd)
        qr = _turn(q[..., d:], n - last)
        down = h @ w["dkv_proj"].T
        lat, kr = _rms(down[:, :r], w["dkv_norm"]), _turn(down[:, None, r:])[:, 0]
        gate = torch.sigmoid(hq @ w["g_proj"].T)
        out = []
        for i in range(a):
            uk, uv = w["uk_proj"][i * d:(i + 1) * d], w["uv_proj"][i * dv:(i + 1) * dv]
            o = _softmax_rows(torch.cat([q[:, i, :d] @ uk, qr[:, i]], dim=1), torch.cat([lat, kr], dim=1), lat, (d + rd) ** -0.5, last,
                              w["sink"][i])
            out.append(o @ uv.T * gate[:, i:i + 1])
        return torch.cat(out, dim=1) @ w["o_proj"].T, []
    d, dv = c["dim"], c["vdim"]
    S = torch.zeros((a, d, dv), dtype=torch.float64, device=DEV)
    o = torch.empty((n, a, dv), dtype=torch.float64, device=DEV)
    if c["mixer"] == "lightning":
        q, k, v = (F.silu(h @ w[m].T).view(n, a, -1) for m in ("q_proj", "k_proj", "v_proj"))
        # the kernels hold the decay as a 32-bit number
        dec = torch.tensor(_decays(a), dtype=torch.float32, device=DEV).double()[:, None, None]
        for t in range(n):
            S = dec * S + k[t, :, :, None] * v[t, :, None, :]
            o[t] = (q[t, :, None, :] @ S)[:, 0]
        y = _rms(o.view(n, -1), w["norm"]) * torch.sigmoid(h @ w["g_proj"].T)
        return (y @ w["o_proj"].T)[n - last:], [S]
    if c["mixer"] == "gated_linear":
        q, k, v = ((h @ w[m].T).view(n, a, -1) for m in ("q_proj", "k_proj", "v_proj"))
        dec = torch.sigmoid(h @ w["a1_proj"].T @ w["a2_proj"].T + w["a2_proj.bias"]).pow(1.0 / 8.0).view(n, a, d)
        for t in range(n):
            S = dec[t, :, :, None] * S + k[t, :, :, None] * v[t, :, None, :]
            o[t] = (q[t, :, None, :] @ S)[:, 0] * d ** -0.5
        y = _rms(o, w["norm"]).reshape(n, -1) * F.silu(h @ w["g_proj"].T)
        return (y @ w["o_proj"].T)[n - last:], [S]
    g, inner = c["kv"], a * dv
    proj = h @ w["in_proj"].T
    z, u, dt = proj[:, :inner], proj[:, inner:2 * inner + 2 * g * d], proj[:, 2 * inner + 2 * g * d:]
    conv = F.conv1d(F.pad(u.T, (3, 0))[None], w["conv"][:, None], w["conv.bias"], groups=u.shape[1])[0].T
    conv = F.silu(conv)
    x = conv[:, :inner].view(n, a, dv)
    B = conv[:, inner:inner + g * d].view(n, g, d).repeat_interleave(a // g, dim=1)
    C = conv[:, inner + g * d:].view(n, g, d).repeat_interleave(a // g, dim=1)
    dt = F.softplus(dt + w["dt_bias"])
    dec = torch.exp(-torch.exp(w["A_log"]) * dt)
    for t in range(n):
        S = dec[t, :, None, None] * S + B[t, :, :, None] * (dt[t, :, None] * x[t])[:, None, :]
        o[t] = (C[t, :, None, :] @ S)[:, 0] + w["D"][:, None] * x[t]
    y = _rms((o.reshape(n, -1) * F.silu(z)).view(n, g, -1)).reshape(n, -1) * w["norm"]
    return (y @ w["o_proj"].T)[n - last:], [S, F.pad(u.T, (3, 0)).T[-3:]]


def _mlp(w, h):
    return (F.silu(h @ w["gate_proj"].T) * (h @ w["up_proj"].T)) @ w["down_proj"].T


def _block(c, w, x, last):
    """One sequence through a pre-norm block, its last ``last`` tokens."""
    part = lambda p: {k[len(p):]: v for k, v in w.items() if k.startswith(p)}  # noqa: E731
    y, _ = _mix(c, part("mixer."), _rms(x, w["norm1.weight"]), last)
    x = x[x.shape[0] - last:] + y
    return x + _mlp(part("ffn."), _rms(x, w["norm2.weight"]))


def _experts(c, w, h):
    z = h @ w["router"].T
    s = torch.softmax(z, -1)
    pick = s + w["correction"]
    per = c["experts"] // ROUTED["n_groups"]
    best = pick.view(-1, ROUTED["n_groups"], per).amax(-1)
    keep = torch.zeros_like(best).scatter(1, best.topk(ROUTED["keep_groups"], dim=1).indices, 1.0).repeat_interleave(per, dim=1)
    idx = pick.masked_fill(keep == 0, float("-inf")).topk(c["top"], dim=1).indices
    y = torch.zeros_like(h)
    for e in range(c["experts"]):
        rows, _ = torch.nonzero(idx == e, as_tuple=True)
        if rows.numel():
            one = {k: w[f"experts.{e}.{k}"] for k in ("gate_proj", "up_proj", "down_proj")}
            y[rows] += _mlp(one, h[rows]) * s[rows, e:e + 1]
    if c["shared"]:
        one = {k: w[f"shared.{k}"] for k in ("gate_proj", "up_proj", "down_proj")}
        y += _mlp(one, h) * torch.sigmoid(h @ w["shared.gate"].T)
    return y


def exact(case, seed):
    w, g = _weights(case, seed)
    if case["kind"] in ("layer", "ffn"):
        x = _rows(case, g).double()
        w = {k: v.double() for k, v in w.items()}
        if case["kind"] == "ffn":
            return _experts(case, w, x)
        outs, kept = [], []
        for one in x.split(_lengths(case)):
            if case["part"] == "block":
                outs.append(_block(case, w, one, one.shape[0]))
            else:
                y, state = _mix(case, w, one, one.shape[0])
                outs.append(y)
                kept.append(state)
        return [torch.cat(outs)] + ([torch.stack(list(s)) for s in zip(*kept)] if kept and kept[0] else [])
    embed = w.pop("embed")
    w = {k: v.double() for k, v in w.items()}
    logits = []
    for prompt, more in _tokens(case, g):
        x = embed[torch.tensor(prompt + more, device=DEV)].double()
        wanted = len(more) + (1 if case["kind"] == "serve" else 0)
        for i in range(case["layers"]):
            p = f"l{i}."
            x = _block(case, {k[len(p):]: v for k, v in w.items() if k.startswith(p)}, x, wanted if i == case["layers"] - 1 else x.shape[0])
        logits.append(_rms(x, w["final"]) @ w["head"].T)
    if case["kind"] == "step":
        return torch.cat(logits)
    return list(torch.stack(logits, dim=1))
