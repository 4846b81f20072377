"""What is timed: the layers that this framework's models are made of, and one whole call.

A layer is built from its part kind, given weights, emitted into a plan and compiled once, as a model does it when it is loaded;
a pass is one run of that plan for one step's batch.  The whole call serves a few prompts and some decoded tokens through
`Engine.step`.  Sizes are those of the benchmark's shapes (the 8B, 14B and 32B grouped-query models and the designs of width
2,048 and 4,096), with request counts, prompt lengths and contexts around them.
"""
import math

import numpy as np
import torch

from llmengine_b200.config import EngineConfig
from llmengine_b200.config.spec import PartSpec
from llmengine_b200.engine.batch import GroupView, StepBatch
from llmengine_b200.engine.engine import Engine, StepEntry
from llmengine_b200.engine.plan import Plan
from llmengine_b200.kernels.ops import CudaOps
from llmengine_b200.parts import Runtime, build_part

DEVICE = "cuda:0"
EPS = 1e-6
PAGE = 16
THETA = 1000000.0
F64 = torch.float64


# ----------------------------------------------------------------------------- the cases
def listed():
    return [
        # the feed-forward of a small model while a few requests decode: the shortest pass there is
        {"name": "mlp_few_tokens", "layer": "mlp", "dtype": "bfloat16", "tokens": 3, "hidden": 2048, "inter": 5504},
        # the feed-forward of the 8B shape in a decode step of 8 requests: weights streamed once
        {"name": "mlp_decode", "layer": "mlp", "dtype": "bfloat16", "tokens": 8, "hidden": 4096, "inter": 12288},
        # the 14B shape in a step that mixes a prompt portion with decoded tokens
        {"name": "mlp_mixed", "layer": "mlp", "dtype": "bfloat16", "tokens": 72, "hidden": 5120, "inter": 17408},
        # the 8B shape on one full prompt: the largest pass
        {"name": "mlp_prompt", "layer": "mlp", "dtype": "bfloat16", "tokens": 2048, "hidden": 4096, "inter": 12288},
        # the 32-bit engine on a short prompt
        {"name": "mlp_prompt_f32", "layer": "mlp", "dtype": "float32", "tokens": 300, "hidden": 2048, "inter": 5504},
        # attention of the 8B shape on two prompts of different lengths
        {"name": "gqa_prompt", "layer": "gqa", "requests": 2, "tokens": 2048, "cached": 0, "hidden": 4096, "heads": 32, "kv_heads": 8},
        # latent attention while 24 requests decode over long contexts
        {"name": "latent_decode", "layer": "latent", "requests": 24, "tokens": 24, "cached": 4000, "hidden": 2048, "heads": 16},
        # latent attention on one prompt
        {"name": "latent_prompt", "layer": "latent", "requests": 1, "tokens": 2000, "cached": 0, "hidden": 2048, "heads": 16},
        # window attention with kept first positions and a sink, a prompt's second portion beside a fresh one
        {"name": "window_prompt", "layer": "window", "requests": 2, "tokens": 1900, "cached": 700, "hidden": 2048, "heads": 16, "kv_heads": 4,
         "window": 1024},
        # routed experts with a shared one on a prompt portion
        {"name": "experts_prompt", "layer": "experts", "tokens": 700, "hidden": 2048, "experts": 32, "top": 4, "inter": 1024},
        # the gated delta memory on two prompts
        {"name": "delta_prompt", "layer": "delta", "requests": 2, "tokens": 1500, "fresh": True, "hidden": 2048, "heads": 16},
        # a whole call: four prompts, then sixteen decoded tokens each, through four layers of a width-2,048 model
        {"name": "engine_generate", "layer": "engine", "requests": 4, "prompt": 700, "steps": 16, "layers": 4, "hidden": 2048, "heads": 16,
         "kv_heads": 4, "inter": 5504, "vocab": 32768},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    layer = rng.choice(["mlp", "mlp", "gqa", "latent", "window", "experts", "delta", "engine"])
    prompt = rng.random() < 0.5
    if layer == "mlp":
        hidden, inter = rng.choice([(2048, 5504), (4096, 12288), (4096, 10944), (5120, 17408)])
        if rng.random() < 0.15:
            return {"layer": layer, "dtype": "float32", "tokens": _log(rng, 1, 400), "hidden": 2048, "inter": 5504}
        tokens = _log(rng, 1, 2048 if hidden * inter <= 4096 * 12288 else 1100)
        return {"layer": layer, "dtype": "bfloat16", "tokens": tokens, "hidden": hidden, "inter": inter}
    if layer == "engine":
        hidden, heads, inter = rng.choice([(2048, 16, 5504), (4096, 32, 10944)])
        return {"layer": layer, "requests": rng.randint(1, 12), "prompt": _log(rng, 20, 160), "steps": rng.randint(4, 12), "layers": rng.randint(2, 3),
                "hidden": hidden, "heads": heads, "kv_heads": heads // 4, "inter": inter, "vocab": 32768}
    hidden, heads = rng.choice([(2048, 16), (4096, 32)])
    if layer == "experts":
        tokens = _log(rng, 1, 1500)
        return {"layer": layer, "tokens": tokens, "hidden": 2048, "experts": 32, "top": 4, "inter": rng.choice([1024, 1536, 2048])}
    if layer == "delta":
        requests = rng.randint(1, 4) if prompt else _log(rng, 1, 64)
        return {"layer": layer, "requests": requests, "tokens": requests * _log(rng, 40, 1500 // requests) + 1 if prompt else requests,
                "fresh": prompt and rng.random() < 0.5, "hidden": hidden, "heads": heads}
    requests = rng.randint(1, 4) if prompt else _log(rng, 1, 64)
    tokens = _log(rng, 64, 2048 if hidden == 2048 else 1200) if prompt else requests
    cached = (rng.choice([0, _log(rng, 16, 1500)]) if prompt else _log(rng, 100, 6000))
    case = {"layer": layer, "requests": requests, "tokens": tokens, "cached": cached, "hidden": hidden, "heads": heads}
    if layer != "latent":
        case["kv_heads"] = heads // 4
    if layer == "window":
        case["window"] = rng.choice([256, 512, 1024])
    return case


# ----------------------------------------------------------------------------- inputs, the same for `prepare` and `exact`
HEAD = 128                                         # head size of the grouped-query and window layers, and of the delta memory
RANK, ROT, NOPE, VDIM = 512, 64, 128, 128          # latent attention
KEEP_FIRST, TAPS = 4, 4


def _shapes(c):
    """Tensor name -> (shape, kind): "m" a matrix of the products' type, "g" a gain, "u" a vector of ordinary numbers."""
    D, n = c["hidden"], "layer."
    if c["layer"] == "mlp":
        return {n + "gate_proj.weight": ((c["inter"], D), "m"), n + "up_proj.weight": ((c["inter"], D), "m"), n + "down_proj.weight": ((D, c["inter"]), "m")}
    if c["layer"] == "gqa":
        q, kv = c["heads"] * HEAD, c["kv_heads"] * HEAD
        return {n + "q_proj.weight": ((q, D), "m"), n + "k_proj.weight": ((kv, D), "m"), n + "v_proj.weight": ((kv, D), "m"),
                n + "o_proj.weight": ((D, q), "m"), n + "q_norm.weight": ((HEAD,), "g"), n + "k_norm.weight": ((HEAD,), "g")}
    if c["layer"] == "window":
        q, kv = c["heads"] * HEAD, c["kv_heads"] * HEAD
        return {n + "q": ((q, D), "m"), n + "k": ((kv, D), "m"), n + "v": ((kv, D), "m"), n + "o": ((D, q), "m"), n + "q.norm": ((q,), "g"),
                n + "k.norm": ((kv,), "g"), n + "sink": ((c["heads"],), "u")}
    if c["layer"] == "latent":
        H = c["heads"]
        return {n + "q": ((H * (NOPE + ROT), D), "m"), n + "dkv": ((RANK + ROT, D), "m"), n + "dkv.norm": ((RANK,), "g"),
                n + "uk": ((H * NOPE, RANK), "m"), n + "uv": ((H * VDIM, RANK), "m"), n + "g": ((H * VDIM, D), "m"), n + "o": ((D, H * VDIM), "m")}
    if c["layer"] == "experts":
        s = {n + "router": ((c["experts"], D), "m")}
        for e in [f"e{i}" for i in range(c["experts"])] + ["shared"]:
            s.update({f"{n}{e}.gate": ((c["inter"], D), "m"), f"{n}{e}.up": ((c["inter"], D), "m"), f"{n}{e}.down": ((D, c["inter"]), "m")})
        return s
    if c["layer"] == "delta":
        H, q, v = c["heads"], c["heads"] // 2 * HEAD, c["heads"] * HEAD
        return {n + "q": ((q, D), "m"), n + "q.conv": ((q, TAPS), "u"), n + "k": ((q, D), "m"), n + "k.conv": ((q, TAPS), "u"), n + "v": ((v, D), "m"),
                n + "v.conv": ((v, TAPS), "u"), n + "g": ((v, D), "m"), n + "b": ((H, D), "m"), n + "a": ((H, D), "m"), n + "A_log": ((H,), "u"),
                n + "dt_bias": ((H,), "u"), n + "norm": ((HEAD,), "g"), n + "o": ((D, v), "m")}
    s = {"model.embed_tokens.weight": ((c["vocab"], D), "m"), "model.norm.weight": ((D,), "g"), "lm_head.weight": ((c["vocab"], D), "m")}
    for i in range(c["layers"]):
        p, q, kv = f"model.layers.{i}.", c["heads"] * HEAD, c["kv_heads"] * HEAD
        s.update({p + "input_layernorm.weight": ((D,), "g"), p + "post_attention_layernorm.weight": ((D,), "g"),
                  p + "self_attn.q_proj.weight": ((q, D), "m"), p + "self_attn.k_proj.weight": ((kv, D), "m"), p + "self_attn.v_proj.weight": ((kv, D), "m"),
                  p + "self_attn.o_proj.weight": ((D, q), "m"), p + "self_attn.q_norm.weight": ((HEAD,), "g"), p + "self_attn.k_norm.weight": ((HEAD,), "g"),
                  p + "mlp.gate_proj.weight": ((c["inter"], D), "m"), p + "mlp.up_proj.weight": ((c["inter"], D), "m"),
                  p + "mlp.down_proj.weight": ((D, c["inter"]), "m")})
    return s


def _dtype(c):
    return torch.float32 if c.get("dtype") == "float32" else torch.bfloat16


def _generator(seed, salt):
    return torch.Generator(device=DEVICE).manual_seed(int(seed) * 16 + salt)


def _weights(c, seed):
    g = _generator(seed, 1)
    out = {}
    for name, (shape, kind) in _shapes(c).items():
        t = torch.randn(*shape, generator=g, device=DEVICE, dtype=torch.float32)
        out[name] = (t * 0.02).to(_dtype(c)) if kind == "m" else 1.0 + 0.1 * t if kind == "g" else t
    return out


def _input(c, seed):
    """What a norm hands to the layer: about one in size."""
    return torch.randn(c["tokens"], c["hidden"], generator=_generator(seed, 2), device=DEVICE, dtype=torch.float32).to(_dtype(c))


def _lens(c):
    """(new tokens, cached tokens) of each request: decode steps have one token each over contexts of different lengths, prompts
    are cut unevenly, and only the first request of several has a portion cached already."""
    R, T = c["requests"], c["tokens"]
    cached = c.get("cached", 0)
    if T == R:
        return [1] * R, [cached - (37 * i) % (cached // 2 + 1) for i in range(R)]
    share = [T * (2 + i) // sum(2 + j for j in range(R)) for i in range(R)]
    share[-1] += T - sum(share)
    return share, [cached if i == 0 else 0 for i in range(R)]


def _pages(c):
    """Each request's pages, in an order that a pool in use would give out: requests' pages lie between one another."""
    q, s = _lens(c)
    need = [-(-(a + b) // PAGE) for a, b in zip(q, s)]
    perm = np.random.RandomState(7).permutation(sum(need))
    ends = np.cumsum(need)
    return [perm[e - n:e].tolist() for e, n in zip(ends, need)], sum(need)


def _row_width(c):
    return RANK + ROT if c["layer"] == "latent" else 2 * c["kv_heads"] * HEAD


def _cache_values(c, seed):
    """What earlier steps left in the pages, one row a token: normed keys (about one in size) and values."""
    _, n = _pages(c)
    return torch.randn(n, PAGE * _row_width(c), generator=_generator(seed, 3), device=DEVICE, dtype=torch.float32).to(torch.bfloat16)


def _states(c, seed):
    """(conv, state) of the delta memory's slots: cleared for new requests, else what a memory holds after some tokens."""
    R, H = c["requests"], c["heads"]
    g = _generator(seed, 3)
    conv = torch.randn(R, TAPS - 1, 2 * H * HEAD, generator=g, device=DEVICE)
    state = torch.randn(R, H, HEAD, HEAD, generator=g, device=DEVICE) * 0.1
    return (torch.zeros_like(conv), torch.zeros_like(state)) if c["fresh"] else (conv, state)


# ----------------------------------------------------------------------------- a layer, ready to run
def _part(c, rt):
    D = c["hidden"]
    if c["layer"] == "mlp":
        return build_part("feed_forward", PartSpec("swiglu", {"hidden_size": D, "intermediate_size": c["inter"]}), rt, "layer")
    if c["layer"] == "gqa":
        return build_part("mixer", PartSpec("gqa_attention", {
            "hidden_size": D, "num_heads": c["heads"], "num_kv_heads": c["kv_heads"], "head_dim": HEAD, "qk_norm_eps": EPS,
            "position_encoding": PartSpec("rope", {"head_dim": HEAD, "theta": THETA, "max_positions": 16384})}), rt, "layer")
    if c["layer"] == "window":
        return build_part("mixer", PartSpec("gqa_window_sink", {
            "hidden_size": D, "num_heads": c["heads"], "num_kv_heads": c["kv_heads"], "qk_dim": HEAD, "v_dim": HEAD, "scale": HEAD ** -0.5,
            "norm_eps": EPS, "window": c["window"], "keep_first": KEEP_FIRST, "sink": True,
            "position_encoding": PartSpec("rotary_partial", {"dims": HEAD // 2, "base": THETA})}), rt, "layer")
    if c["layer"] == "latent":
        return build_part("mixer", PartSpec("latent_attention", {
            "hidden_size": D, "num_heads": c["heads"], "nope_dim": NOPE, "rot_dim": ROT, "v_dim": VDIM, "kv_rank": RANK,
            "scale": (NOPE + ROT) ** -0.5, "norm_eps": EPS, "output_gate": True,
            "position_encoding": PartSpec("rotary_partial", {"dims": ROT, "base": THETA})}), rt, "layer")
    if c["layer"] == "experts":
        return build_part("feed_forward", PartSpec("routed_experts", {
            "hidden_size": D, "num_experts": c["experts"], "top_k": c["top"], "expert_size": c["inter"], "route_scale": 2.5,
            "shared_size": c["inter"]}), rt, "layer")
    return build_part("mixer", PartSpec("gated_delta", {
        "hidden_size": D, "num_heads": c["heads"], "num_qk_heads": c["heads"] // 2, "qk_dim": HEAD, "v_dim": HEAD, "taps": TAPS, "norm_eps": EPS}),
        rt, "layer")


def _batch(c):
    """The step's batch: tokens, positions, lengths and block tables, as the engine lays them out."""
    q, s = _lens(c)
    R, T = c["requests"], c["tokens"]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEVICE)
    positions = [s[r] + i for r in range(R) for i in range(q[r])]
    groups = []
    if c["layer"] != "delta":
        pages, _ = _pages(c)
        widest = max(len(p) for p in pages)
        slots = [pages[r][p // PAGE] * PAGE + p % PAGE for r in range(R) for p in range(s[r], s[r] + q[r])]
        groups = [GroupView(PAGE, c.get("window", 0), i32([p + [-1] * (widest - len(p)) for p in pages]), i32(slots), widest)]
    empty = i32([])
    return StepBatch(
        num_tokens=T, num_requests=R, q_lens=q, start_positions=s, token_ids=torch.zeros(T, dtype=torch.int32, device=DEVICE),
        positions=i32(positions), token_request=i32([r for r in range(R) for _ in range(q[r])]), cu_q_lens=i32([0] + np.cumsum(q).tolist()),
        ctx_lens=i32([a + b for a, b in zip(q, s)]), state_slots=i32(list(range(R))), first_portion=i32([1 if b == 0 else 0 for b in s]),
        logit_rows=empty, decode_rows=i32([r for r in range(R) if q[r] == 1]), portion_rows=i32([r for r in range(R) if q[r] != 1]), groups=groups)


def _prepare_layer(c, seed):
    device = torch.device(DEVICE)
    T, R = c["tokens"], c.get("requests", 1)
    rt = Runtime(CudaOps(device), device, _dtype(c), T, max_requests=R)
    part = _part(c, rt)
    part.load_weights(_weights(c, seed))
    h, plan, kept = _input(c, seed), Plan(), {}
    if c["layer"] in ("mlp", "experts"):
        out, batch = part.emit(plan, h), StepBatch.bare(T, device)
    elif c["layer"] == "delta":
        spec = part.cache_spec()
        states = spec.allocate(R, PAGE, rt.dtype, device)
        view = spec.view(states, None, True)
        conv, state = _states(c, seed)
        view.states["conv"].copy_(conv)
        view.states["state"].copy_(state)
        out, batch, kept = part.emit(plan, h, view), _batch(c), {"conv": view.states["conv"], "state": view.states["state"]}
    else:
        spec = part.cache_spec()
        _, pages = _pages(c)
        cache = spec.allocate(pages, PAGE, rt.dtype, device)
        cache.copy_(_cache_values(c, seed).view(cache.shape))
        out, batch, kept = part.emit(plan, h, spec.view(cache, 0, True)), _batch(c), {"cache": cache}
    return {"rt": rt, "part": part, "batch": batch, "compiled": rt.ops.compile(plan), "outputs": {"out": out[:T], **kept}}


# ----------------------------------------------------------------------------- the whole call
def _config(c):
    return {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": c["layers"], "hidden_size": c["hidden"], "num_attention_heads": c["heads"],
            "num_key_value_heads": c["kv_heads"], "head_dim": HEAD, "intermediate_size": c["inter"], "vocab_size": c["vocab"], "rope_theta": THETA,
            "rms_norm_eps": EPS, "tie_word_embeddings": False, "max_position_embeddings": 4096, "hidden_act": "silu"}


def _prompts(c, seed):
    """Each request's tokens: its prompt (lengths differ) and the tokens that are decoded after it, given beforehand."""
    r = np.random.RandomState(int(seed) % (1 << 31))
    return [r.randint(0, c["vocab"], c["prompt"] - (13 * i) % (c["prompt"] // 2 + 1) + c["steps"]).tolist() for i in range(c["requests"])]


def _prepare_engine(c, seed):
    room = c["requests"] * (c["prompt"] + c["steps"] + PAGE)
    ec = EngineConfig(dtype="bfloat16", page_size=PAGE, max_cached_tokens=-(-room // PAGE) * PAGE, max_num_seqs=c["requests"],
                      max_num_batched_tokens=c["requests"] * c["prompt"], max_model_len=c["prompt"] + c["steps"])
    engine = Engine(config=_config(c), random_seed=0, engine_config=ec)
    engine.model.load_weights(_weights(c, seed))
    tokens = _prompts(c, seed)
    n = c["steps"]
    return {"engine": engine, "prompts": [StepEntry(i, t[:-n], [len(t) - n - 1]) for i, t in enumerate(tokens)],
            "decode": [[StepEntry(i, [t[len(t) - n + k]], [0]) for i, t in enumerate(tokens)] for k in range(n)]}


def prepare(case, seed):
    return _prepare_engine(case, seed) if case["layer"] == "engine" else _prepare_layer(case, seed)


def run(state):
    if "engine" not in state:
        state["compiled"].run(state["batch"])
        return state["outputs"]
    engine, last = state["engine"], len(state["decode"]) - 1
    first = engine.step(state["prompts"]).clone()                    # the engine's logits are overwritten by its next step
    for k, entries in enumerate(state["decode"]):
        logits = engine.step(entries, end=[e.request for e in entries] if k == last else ())
    return {"first": first, "last": logits}


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    c = case
    matrices = sum(math.prod(s) for s, k in _shapes(c).values() if k == "m")
    size = 4 if c.get("dtype") == "float32" else 2
    if c["layer"] == "engine":
        tokens = [len(t) for t in _prompts(c, 0)]
        cache = 2 * c["kv_heads"] * HEAD * 2 * c["layers"]
        dense = matrices - c["vocab"] * c["hidden"]                  # the embedding is looked up
        keys = sum(n * (n + 1) / 2 for n in tokens)
        head = c["vocab"] * c["hidden"]
        flops = 2.0 * sum(tokens) * (dense - head) + 2.0 * c["requests"] * (1 + c["steps"]) * head + 4.0 * keys * c["heads"] * HEAD * c["layers"]
        return {"bytes": (1 + c["steps"]) * (2 * dense + 4 * c["requests"] * c["vocab"]) + c["steps"] * sum(tokens) * cache, "flops": flops}
    T, D = c["tokens"], c["hidden"]
    through = T * D * (size + 4)                                     # the input, and the 32-bit contribution
    if c["layer"] == "mlp":
        return {"bytes": matrices * size + through, "flops": 2.0 * T * matrices}
    if c["layer"] == "experts":
        one = 3 * D * c["inter"]
        used = c["experts"] * (1.0 - (1.0 - c["top"] / c["experts"]) ** T) + 1
        return {"bytes": 2 * (used * one + c["experts"] * D) + through, "flops": 2.0 * T * ((c["top"] + 1) * one + c["experts"] * D)}
    if c["layer"] == "delta":
        H = c["heads"]
        return {"bytes": 2 * matrices + through + c["requests"] * 8 * (H * HEAD * HEAD + (TAPS - 1) * 2 * H * HEAD),
                "flops": 2.0 * T * matrices + 6.0 * T * H * HEAD * HEAD}
    q, s = _lens(c)
    W = c.get("window", 0)
    keys = sum(min(p + 1, W) if W else p + 1 for a, b in zip(q, s) for p in range(b, b + a))
    rows = sum(min(a + b, a + W) if W else a + b for a, b in zip(q, s))
    per_key = c["heads"] * (2 * RANK + ROT if c["layer"] == "latent" else 2 * HEAD)
    return {"bytes": 2 * matrices + through + rows * _row_width(c) * 2, "flops": 2.0 * T * matrices + 2.0 * keys * per_key}


def tolerance(case):
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    if case["layer"] == "engine":
        return {"rel": 3e-2, "max": 3e-1}                            # roundings of every layer travel through those behind it
    if case["layer"] == "experts":
        return {"rel": 1e-2, "max": 3e-1}                            # two experts in a tie may change places
    return {"rel": 1e-2, "max": 1e-1}


# ----------------------------------------------------------------------------- the same in 64 bits, in plain torch
def _rms(x, gain=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if gain is None else y * gain


def _rotate(x, positions, dims):
    """Coordinate i of the first `dims` is turned with i + dims / 2; x [T, heads, size]."""
    half = dims // 2
    f = torch.tensor([THETA ** (-2.0 * i / dims) for i in range(half)], dtype=F64, device=x.device)
    a = positions.to(F64)[:, None] * f
    co, si = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * co - v * si, v * co + u * si, x[..., dims:]], -1)


def _swiglu(h, gate, up, down):
    g = h @ gate.t()
    return (g * torch.sigmoid(g) * (h @ up.t())) @ down.t()


def _attend(q, k, v, start, scale, window=0, keep_first=0, sink=None):
    """q [n, H, d] at positions start ..; k [m, G, d], v [m, G, dv]: causal softmax per head."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(start, start + n, device=q.device)[:, None]
    j = torch.arange(k.shape[0], device=q.device)[None, :]
    seen = (j <= i) & ((i - j < window) | (j < keep_first)) if window else j <= i
    out = []
    for a in range(H):
        s = (q[:, a] @ k[:, a // (H // G)].t() * scale).masked_fill(~seen, float("-inf"))
        m = s.max(-1, keepdim=True).values
        if sink is not None:
            m = torch.clamp(m, min=float(sink[a]))
        e = torch.exp(s - m)
        total = e.sum(-1, keepdim=True) + (torch.exp(sink[a] - m) if sink is not None else 0.0)
        out.append((e / total) @ v[:, a // (H // G)])
    return torch.stack(out, 1)


def _conv(u, before, taps):
    x = torch.cat([before, u], 0)
    return sum(x[j:j + u.shape[0]] * taps[:, j] for j in range(TAPS))


def _exact_delta(c, h, w, conv, state):
    H, n = c["heads"], "layer."
    qs = H // 2 * HEAD
    q_len, _ = _lens(c)
    conv, state, out, at = conv.clone(), state.clone(), [], 0
    u = torch.cat([h @ w[n + x].t() for x in ("q", "k", "v")], 1)
    taps = torch.cat([w[n + x + ".conv"] for x in ("q", "k", "v")], 0)
    beta, keep = torch.sigmoid(h @ w[n + "b"].t()), torch.exp(-torch.exp(w[n + "A_log"]) * torch.nn.functional.softplus(h @ w[n + "a"].t() + w[n + "dt_bias"]))
    gate = h @ w[n + "g"].t()
    for r, T in enumerate(q_len):
        y = _conv(u[at:at + T], conv[r], taps)
        y = y * torch.sigmoid(y)
        conv[r] = torch.cat([conv[r], u[at:at + T]], 0)[-(TAPS - 1):]
        unit = lambda x: x.view(T, H // 2, HEAD) / torch.sqrt((x.view(T, H // 2, HEAD) ** 2).sum(-1, keepdim=True) + 1e-6)
        q = (unit(y[:, :qs]) * HEAD ** -0.5).repeat_interleave(2, 1)
        k = unit(y[:, qs:2 * qs]).repeat_interleave(2, 1)
        v = y[:, 2 * qs:].view(T, H, HEAD)
        S, o = state[r], []                                          # [H, v, k]
        for t in range(T):
            S = keep[at + t][:, None, None] * S
            d = beta[at + t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0])
            S = S + d[:, :, None] * k[t][:, None, :]
            o.append((S @ q[t][:, :, None])[..., 0])
        state[r] = S
        y = (_rms(torch.stack(o)) * w[n + "norm"]).reshape(T, H * HEAD)
        g = gate[at:at + T]
        out.append((y * g * torch.sigmoid(g)) @ w[n + "o"].t())
        at += T
    return {"out": torch.cat(out), "conv": conv, "state": state}


def _exact_attention(c, seed, h, w):
    n, T, H = "layer.", c["tokens"], c["heads"]
    q_len, start = _lens(c)
    pages, count = _pages(c)
    cache = _cache_values(c, seed).double()
    positions = torch.tensor([s + i for a, s in zip(q_len, start) for i in range(a)], device=DEVICE)
    if c["layer"] == "latent":
        q = (h @ w[n + "q"].t()).view(T, H, NOPE + ROT)
        kv = h @ w[n + "dkv"].t()
        new = torch.cat([_rms(kv[:, :RANK], w[n + "dkv.norm"]), _rotate(kv[:, None, RANK:], positions, ROT)[:, 0]], 1)
        uk, uv = w[n + "uk"].view(H, NOPE, RANK), w[n + "uv"].view(H, VDIM, RANK)
        q = torch.cat([torch.einsum("thd,hdr->thr", q[..., :NOPE], uk), _rotate(q[..., NOPE:], positions, ROT)], -1)
        rows = cache.view(count * PAGE, RANK + ROT)
        out, at = [], 0
        for a, s, p in zip(q_len, start, pages):
            where = torch.tensor([p[i // PAGE] * PAGE + i % PAGE for i in range(a + s)], device=DEVICE)
            rows[where[s:]] = new[at:at + a]
            k = rows[where][:, None]
            out.append(_attend(q[at:at + a], k, k[..., :RANK], s, (NOPE + ROT) ** -0.5))
            at += a
        heads = torch.einsum("thr,hvr->thv", torch.cat(out), uv).reshape(T, H * VDIM) * torch.sigmoid(h @ w[n + "g"].t())
        return {"out": heads @ w[n + "o"].t(), "cache": rows.view(count, PAGE, RANK + ROT)}
    G = c["kv_heads"]
    if c["layer"] == "gqa":
        q, k, v = ((h @ w[n + x + "_proj.weight"].t()).view(T, -1, HEAD) for x in "qkv")
        q, k = (_rotate(_rms(x, w[n + y + "_norm.weight"]), positions, HEAD) for x, y in ((q, "q"), (k, "k")))
        more, w_o = {}, w[n + "o_proj.weight"]
    else:
        v = (h @ w[n + "v"].t()).view(T, G, HEAD)
        q, k = (_rotate(_rms(h @ w[n + y].t(), w[n + y + ".norm"]).view(T, -1, HEAD), positions, HEAD // 2) for y in "qk")
        more, w_o = {"window": c["window"], "keep_first": KEEP_FIRST, "sink": w[n + "sink"]}, w[n + "o"]
    paged = cache.view(count, 2, G, PAGE, HEAD)                      # a page: its keys head by head, then its values
    out, at = [], 0
    for a, s, p in zip(q_len, start, pages):
        page = torch.tensor([p[i // PAGE] for i in range(a + s)], device=DEVICE)
        slot = torch.arange(a + s, device=DEVICE) % PAGE
        paged[page[s:], 0, :, slot[s:]] = k[at:at + a]
        paged[page[s:], 1, :, slot[s:]] = v[at:at + a]
        out.append(_attend(q[at:at + a], paged[page, 0, :, slot], paged[page, 1, :, slot], s, HEAD ** -0.5, **more))
        at += a
    return {"out": torch.cat(out).reshape(T, H * HEAD) @ w_o.t(), "cache": paged if c["layer"] == "gqa" else paged.reshape(count, -1)}


def _exact_engine(c, seed, w):
    first, last = [], []
    for tokens in _prompts(c, seed):
        T, n = len(tokens), c["steps"]
        positions = torch.arange(T, device=DEVICE)
        x = w["model.embed_tokens.weight"][torch.tensor(tokens, device=DEVICE)]
        for i in range(c["layers"]):
            p = f"model.layers.{i}."
            h = _rms(x, w[p + "input_layernorm.weight"])
            q, k, v = ((h @ w[f"{p}self_attn.{y}_proj.weight"].t()).view(T, -1, HEAD) for y in "qkv")
            q, k = (_rotate(_rms(z, w[f"{p}self_attn.{y}_norm.weight"]), positions, HEAD) for z, y in ((q, "q"), (k, "k")))
            x = x + _attend(q, k, v, 0, HEAD ** -0.5).reshape(T, -1) @ w[p + "self_attn.o_proj.weight"].t()
            h = _rms(x, w[p + "post_attention_layernorm.weight"])
            x = x + _swiglu(h, *(w[f"{p}mlp.{y}_proj.weight"] for y in ("gate", "up", "down")))
        y = _rms(x[[T - n - 1, T - 1]], w["model.norm.weight"]) @ w["lm_head.weight"].t()
        first.append(y[0])
        last.append(y[1])
    return {"first": torch.stack(first), "last": torch.stack(last)}


def exact(case, seed):
    c, n = case, "layer."
    w = {k: t.double() for k, t in _weights(c, seed).items()}
    if c["layer"] == "engine":
        return _exact_engine(c, seed, w)
    h = _input(c, seed).double()
    if c["layer"] == "mlp":
        return {"out": _swiglu(h, *(w[f"{n}{y}_proj.weight"] for y in ("gate", "up", "down")))}
    if c["layer"] == "experts":
        s = torch.sigmoid(h @ w[n + "router"].t())
        top, which = torch.topk(s, c["top"], dim=-1)
        top = top / (top.sum(-1, keepdim=True) + 1e-20) * 2.5
        out = _swiglu(h, *(w[f"{n}shared.{y}"] for y in ("gate", "up", "down")))
        for e in range(c["experts"]):
            rows, place = torch.nonzero(which == e, as_tuple=True)
            out[rows] += top[rows, place][:, None] * _swiglu(h[rows], *(w[f"{n}e{e}.{y}"] for y in ("gate", "up", "down")))
        return {"out": out}
    if c["layer"] == "delta":
        return _exact_delta(c, h, w, *(t.double() for t in _states(c, seed)))
    return _exact_attention(c, seed, h, w)
