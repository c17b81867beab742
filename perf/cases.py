"""The work by which this framework's speed is followed: single layers and whole calls at the layer sizes of its
designs, each through an entry point that a program can call.

* ``experts``: a routed feed-forward at MiniMax M2's layer sizes (``SparseMoE.forward``).
* ``attention``: a grouped-query attention layer of the same sizes over its paged cache (``PagedAttention.forward``).
* ``state_space``, ``delta``: the recurrent mixers of the hybrid design, and the delta rule with one decay per head.
* ``latent``, ``retention``: latent attention and retention of the looped design.
* ``generate``: prompts and the decode steps that follow them through ``build_runner`` and ``ModelRunner.step``, with the
  next tokens given (the logits of every step are what is returned).

Steps of single tokens are replayed from a CUDA graph that ``prepare`` captures, as the engine does with its decode steps;
steps with prompt portions are launched as they come, as the engine does with those.  Whole calls go through the engine,
which makes its graphs itself.  All weights and inputs are made from the seed, matrices N(0, 0.02), activations of order one
(what a norm hands to a sublayer), decays and step sizes in the ranges that trained recurrent layers have.
"""
import math

import torch

from sparseengine_b200.config.specs import (AttentionSpec, GatedDeltaSpec, LatentAttentionSpec, MoESpec, RetentionSpec,
                                            RotarySpec, StateSpaceSpec)
from sparseengine_b200.engine.factory import build_runner
from sparseengine_b200.engine.runner import StepEntry
from sparseengine_b200.parts.base import LayerSlot, StepContext, make_feed_forward, make_mixer

PAGE = 16
F64 = torch.float64
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}

# MiniMax M2 layer sizes
M2 = {"hidden": 3072, "heads": 48, "kv_heads": 8, "dim": 128, "rot": 64, "theta": 5e6, "experts": 256, "top": 8, "inter": 1536,
      "vocab": 200064, "eps": 1e-6}
GRAPH_TOKENS = 64           # the largest decode batch: steps of single tokens up to this are replayed


# ---- the cases ----------------------------------------------------------------------------------

def listed():
    return [
        # one request decoding: the smallest step there is, eight experts' weights streamed for one token
        {"name": "experts_1", "kind": "experts", "dtype": "bf16", "tokens": 1},
        # an ordinary prompt step
        {"name": "experts_2048", "kind": "experts", "dtype": "bf16", "tokens": 2048},
        # a full decode batch in the middle of its contexts, every request of another length
        {"name": "attention_decode_64", "kind": "attention", "dtype": "bf16", "requests": 64, "tokens": 1, "held": 3000},
        # an 8,192-token portion of a long prompt, behind the portions before it
        {"name": "attention_portion_8192", "kind": "attention", "dtype": "bf16", "requests": 1, "tokens": 8192, "held": 16384},
        # the recurrent mixers over one prompt, and over a batch of ragged ones
        {"name": "state_space_2048", "kind": "state_space", "dtype": "bf16", "width": 2048, "requests": 1, "tokens": 2048},
        {"name": "delta_channel_4x1500", "kind": "delta", "dtype": "bf16", "width": 2048, "requests": 4, "tokens": 1500,
         "decay_per": "channel"},
        {"name": "delta_head_2048", "kind": "delta", "dtype": "bf16", "width": 2048, "requests": 1, "tokens": 2048,
         "decay_per": "head"},
        # long prompts through the looped design's mixers
        {"name": "latent_8192", "kind": "latent", "dtype": "bf16", "width": 2048, "requests": 1, "tokens": 8192, "held": 0,
         "window": 1024},
        {"name": "retention_8192", "kind": "retention", "dtype": "bf16", "width": 4096, "requests": 1, "tokens": 8192},
        # a small batch served from prompt to answer, the flagship's layers
        {"name": "generate_m2_bf16", "kind": "generate", "design": "m2", "dtype": "bf16", "requests": 8, "tokens": 256, "steps": 16},
        # the true 32-bit path: prompts of 1, 300, 1,024 and 2,047 tokens and a few decode steps
        {"name": "generate_m2_fp32", "kind": "generate", "design": "m2", "dtype": "fp32", "requests": 4, "tokens": 2047, "steps": 4},
        # a full batch decoding with the hybrid design (recurrent states of 64 requests read and written every step)
        {"name": "generate_hybrid_64", "kind": "generate", "design": "hybrid", "dtype": "bf16", "requests": 64, "tokens": 48, "steps": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["experts", "attention", "attention", "state_space", "delta", "delta", "latent", "retention", "generate"])
    dtype = "fp32" if rng.random() < 0.25 else "bf16"
    fp32 = dtype == "fp32"
    c = {"kind": kind, "dtype": dtype}
    if kind == "experts":
        c["tokens"] = _log(rng, 1, 512 if fp32 else 2048)
    elif kind == "attention":
        if rng.random() < 0.4:
            c.update(requests=_log(rng, 1, 64), tokens=1, held=_log(rng, 1, 3000))
        else:
            n = rng.choice([1, 1, 1, 2, 4])
            c.update(requests=n, tokens=_log(rng, 17, (2048 if fp32 else 8192) // n), held=rng.choice([0, 0, _log(rng, 1, (2048 if fp32 else 16384) // n)]))
    elif kind in ("state_space", "delta"):
        n = rng.choice([1, 1, 2, 4])
        c.update(width=2048, requests=n, tokens=_log(rng, 17, 6000 // n))
        if kind == "delta":
            c["decay_per"] = rng.choice(["channel", "head"])
    elif kind == "latent":
        n = rng.choice([1, 1, 2, 4])
        c.update(width=rng.choice([2048, 4096]), requests=n, tokens=_log(rng, 17, (1024 if fp32 else 4096) // n),
                 held=rng.choice([0, 0, _log(rng, 1, 1024 if fp32 else 4096)]), window=rng.choice([0, 1024]))
    elif kind == "retention":
        n = rng.choice([1, 1, 2, 4])
        c.update(width=rng.choice([2048, 4096]), requests=n, tokens=_log(rng, 17, 8192 // n))
    else:
        c["design"] = rng.choice(["m2", "hybrid"])
        n = _log(rng, 1, 4 if fp32 else 64)
        c.update(requests=n, tokens=_log(rng, 17, 2047 if c["design"] == "m2" and n <= 4 else 256), steps=rng.randint(1, 16))
    return c


# ---- sizes ---------------------------------------------------------------------------------------

def _lengths(case):
    """Tokens that each request brings: "tokens" at most, ragged where there are several."""
    n, t = case["requests"], case["tokens"]
    if n == 1 or t == 1:
        return [t] * n
    if case["kind"] == "generate" and n == 4 and t >= 1024:
        return [1, 300 * t // 2047, t // 2, t]
    return [max(1, t - int(t * 0.5 * ((i * 0.6180339887) % 1.0))) for i in range(n)]


def _held(case):
    """Keys that each request already holds, ragged where there are several."""
    n, h = case["requests"], case.get("held", 0)
    return [h] if n == 1 else [h - int(h * 0.5 * ((i * 0.6180339887) % 1.0)) for i in range(n)]


def _state_sizes(width):
    return {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 8, "taps": 4, "norm_groups": 8}


def _latent_sizes(width):
    return {"heads": width // 64, "dim": 64, "rot": 64, "vdim": 64, "q_rank": width // 2, "rank": 192, "base": 500000.0}


def _decays(heads):
    return [1.0 - 2.0 ** (-5 - 7 * i / max(1, heads - 1)) for i in range(heads)]


def _hybrid_config():
    width = 2048
    heads = width // 128
    a = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "q_temp": {"coef": 0.1, "every": 1024}}
    ff = {"kind": "dense", "ff": 4 * width}
    s = _state_sizes(width)
    return {"architecture": "Bavutar", "vocab": 32768, "width": width, "postln_alpha": 2.0, "embedding": {"scale": 1.0},
            "logit_softcap": 30.0, "norm": {"eps": 1e-6}, "max_position": 16384, "layers": [
                {"type": "attention", "mixer": dict(a), "mlp": ff},
                {"type": "mamba2", "mixer": {"heads": s["heads"], "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8},
                 "mlp": ff},
                {"type": "channel_delta", "mixer": {"heads": heads, "kv_heads": heads, "dim": 128, "vdim": 128, "conv": 4, "rank": 64},
                 "mlp": ff},
                {"type": "attention", "mixer": dict(a, kv_from=0), "mlp": ff}]}


def _m2_config(layers=2):
    m = M2
    return {"architectures": ["MiniMaxM2ForCausalLM"], "model_type": "minimax_m2", "hidden_size": m["hidden"],
            "num_attention_heads": m["heads"], "num_key_value_heads": m["kv_heads"], "head_dim": m["dim"], "rotary_dim": m["rot"],
            "rope_theta": m["theta"], "rms_norm_eps": m["eps"], "num_local_experts": m["experts"], "num_experts_per_tok": m["top"],
            "intermediate_size": m["inter"], "vocab_size": m["vocab"], "max_position_embeddings": 4096,
            "num_hidden_layers": layers, "torch_dtype": "bfloat16"}


def _shapes(case):
    """Name -> (shape, kept in 32-bit) of a layer's or model's parameters, under the framework's names."""
    kind = case["kind"]
    act, f32 = False, True
    if kind == "experts":
        m = M2
        return {"gate": ((m["experts"], m["hidden"]), f32), "w13": ((m["experts"], 2 * m["inter"], m["hidden"]), act),
                "w2": ((m["experts"], m["hidden"], m["inter"]), act), "selection_bias": ((m["experts"],), f32)}
    if kind == "attention":
        m = M2
        q, k = m["heads"] * m["dim"], m["kv_heads"] * m["dim"]
        return {"qkv": ((q + 2 * k, m["hidden"]), act), "o": ((m["hidden"], q), act), "q_norm": ((q,), act), "k_norm": ((k,), act)}
    if kind == "state_space":
        w, s = case["width"], _state_sizes(case["width"])
        inner, gn = s["heads"] * s["vdim"], s["groups"] * s["state"]
        return {"in_proj": ((2 * inner + 2 * gn + s["heads"], w), act), "conv_w": ((inner + 2 * gn, s["taps"]), f32),
                "conv_b": ((inner + 2 * gn,), f32), "dt_bias": ((s["heads"],), f32), "a_log": ((s["heads"],), f32),
                "d_skip": ((s["heads"],), f32), "norm_w": ((inner,), f32), "o": ((w, inner), act)}
    if kind == "delta":
        w = case["width"]
        h, d, r = w // 128, 128, 64
        vv, per_head = h * d, case["decay_per"] == "head"
        out = {"in_proj": ((3 * vv + h + (h + vv if per_head else 2 * r), w), act), "conv_w": ((3 * vv, 4), f32),
               "dt_bias": ((h if per_head else vv,), f32), "a_log": ((h,), f32), "norm_w": ((d,), f32), "o": ((w, vv), act)}
        if not per_head:
            out.update(a2=((vv, r), act), g2=((vv, r), act))
        return out
    if kind == "latent":
        w, s = case["width"], _latent_sizes(case["width"])
        H = s["heads"]
        return {"down": ((s["q_rank"] + s["rank"] + s["rot"], w), act), "q_norm": ((s["q_rank"],), act),
                "uq": ((H * (s["dim"] + s["rot"]), s["q_rank"]), act), "kv_norm": ((s["rank"],), act),
                "uk": ((H * s["dim"], s["rank"]), act), "uv": ((H * s["vdim"], s["rank"]), act),
                "o": ((w, H * s["vdim"]), act), "sink": ((H,), f32)}
    if kind == "retention":
        w = case["width"]
        return {"in_proj": ((4 * w, w), act), "o": ((w, w), act)}
    out = {}
    if case["design"] == "m2":
        m = M2
        layers = [{"mixer.": _shapes({"kind": "attention"}), "feed_forward.": _shapes({"kind": "experts"}),
                   "mixer_norm.": {"weight": ((m["hidden"],), act)}, "feed_forward_norm.": {"weight": ((m["hidden"],), act)}}] * 2
        out.update({"embed": ((m["vocab"], m["hidden"]), act), "head": ((m["vocab"], m["hidden"]), act),
                    "final_norm.weight": ((m["hidden"],), act)})
    else:
        cfg = _hybrid_config()
        w, n = cfg["width"], {"weight": ((cfg["width"],), act), "bias": ((cfg["width"],), act)}
        q, k = w, w // 4
        att = {"qkv": ((q + 2 * k, w), act), "o": ((w, q), act), "q_norm": ((q,), act), "k_norm": ((k,), act)}
        borrowed = {"qkv": ((q, w), act), "o": ((w, q), act), "q_norm": ((q,), act)}
        mixers = [att, _shapes({"kind": "state_space", "width": w}), _shapes({"kind": "delta", "width": w, "decay_per": "channel"}), borrowed]
        layers = [{"mixer.": x, "feed_forward.": {"up": ((4 * w, w), act), "down": ((w, 4 * w), act)}, "mixer_norm.": n,
                   "feed_forward_norm.": n} for x in mixers]
        out.update({"embed": ((cfg["vocab"], w), act), "head": ((cfg["vocab"], w), act), "final_norm.weight": ((w,), act),
                    "final_norm.bias": ((w,), act)})
    for i, layer in enumerate(layers):
        for part, tensors in layer.items():
            out.update({f"layers.{i}.{part}{name}": v for name, v in tensors.items()})
    return out


def _fill(name, t, seed):
    """Seeded values for the parameter ``name`` in place, in the tensor's own type."""
    g = torch.Generator(device=t.device)
    g.manual_seed(int(seed) * 1000003 + sum((i + 1) * b for i, b in enumerate(name.encode())))
    last = name.rsplit(".", 1)[-1]
    if last in ("weight", "q_norm", "k_norm", "kv_norm", "norm_w", "d_skip"):
        t.normal_(1.0, 0.05, generator=g)
    elif last == "bias" or last in ("conv_b", "selection_bias"):
        t.normal_(0.0, 0.1, generator=g)
    elif last == "sink":
        t.normal_(0.0, 0.7, generator=g)
    elif last == "conv_w":
        t.normal_(0.0, 0.4, generator=g)
    elif last == "a_log":           # rates of 1 to 16
        t.uniform_(1.0, 16.0, generator=g).log_()
    elif last == "dt_bias":         # softplus(bias): step sizes of 0.001 to 0.1
        t.uniform_(math.log(1e-3), math.log(1e-1), generator=g).exp_().expm1_().log_()
    elif last == "embed":           # a stream of order one, larger than what a single sublayer adds to it
        t.normal_(0.0, 1.0, generator=g)
    else:
        t.normal_(0.0, 0.02, generator=g)
    return t


def _weights(case, seed):
    return {n: _fill(n, torch.empty(shape, dtype=torch.float32 if f32 else DTYPES[case["dtype"]], device="cuda"), seed)
            for n, (shape, f32) in _shapes(case).items()}


def _normal(shape, dtype, seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + salt)
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(generator=g)


def _hidden(case):
    return case.get("width", M2["hidden"])


def _layer_input(case, seed):
    tokens = sum(_lengths(case)) if "requests" in case else case["tokens"]
    return _normal((tokens, _hidden(case)), DTYPES[case["dtype"]], seed, 1)


def _pages(case, seed):
    """A block table [requests, pages] of shuffled pages for requests that hold ``held`` keys and bring ``tokens`` more."""
    most = -(-max(h + t for h, t in zip(_held(case), _lengths(case))) // PAGE)
    n = case["requests"] * most
    g = torch.Generator()
    g.manual_seed(int(seed) * 31 + 5)
    return torch.randperm(n, generator=g, dtype=torch.int64).to(torch.int32).view(case["requests"], most).cuda(), n


def _cache(case, seed, pages):
    dtype = DTYPES[case["dtype"]]
    if case["kind"] == "latent":
        s = _latent_sizes(case["width"])
        return _normal((pages, PAGE, s["rank"] + s["rot"]), dtype, seed, 2)
    return _normal((pages, 2, M2["kv_heads"], PAGE, M2["dim"]), dtype, seed, 2)


def _token_ids(case, seed, vocab):
    """(prompts, tokens of the decode steps [steps][requests])."""
    g = torch.Generator()
    g.manual_seed(int(seed) * 131 + 7)
    prompts = [torch.randint(0, vocab, (n,), generator=g).tolist() for n in _lengths(case)]
    return prompts, torch.randint(0, vocab, (case["steps"], case["requests"]), generator=g).tolist()


# ---- what a program has in hand ------------------------------------------------------------------

def _step_context(case):
    lens, held = _lengths(case), _held(case)
    n, total = len(lens), sum(lens)

    def i32(v):
        return torch.tensor(v, dtype=torch.int32, device="cuda")

    cu = [0]
    for t in lens:
        cu.append(cu[-1] + t)
    kv = [h + t for h, t in zip(held, lens)]
    return StepContext(
        num_tokens=total, num_seqs=n, token_ids=i32([0] * total), positions=i32([h + i for h, t in zip(held, lens) for i in range(t)]),
        token_seq=i32([j for j, t in enumerate(lens) for _ in range(t)]), seq_rows=i32(list(range(n))), cu_q=i32(cu), kv_len=i32(kv),
        q_lens=lens, q_starts=held, kv_lens=kv, rows=list(range(n)), dtype=DTYPES[case["dtype"]])


def _spec(case):
    kind, m = case["kind"], M2
    if kind == "experts":
        return MoESpec(hidden_size=m["hidden"], num_experts=m["experts"], top_k=m["top"], intermediate_size=m["inter"])
    if kind == "attention":
        return AttentionSpec(hidden_size=m["hidden"], num_heads=m["heads"], num_kv_heads=m["kv_heads"], head_dim=m["dim"],
                             scale=m["dim"] ** -0.5, qk_norm="whole_projection", qk_norm_eps=m["eps"],
                             position=RotarySpec(rotary_dim=m["rot"], theta=m["theta"]))
    w = case["width"]
    if kind == "state_space":
        s = _state_sizes(w)
        return StateSpaceSpec(hidden_size=w, num_heads=s["heads"], head_dim=s["vdim"], state_size=s["state"], groups=s["groups"],
                              conv_taps=s["taps"], norm_groups=s["norm_groups"])
    if kind == "delta":
        h, ranks = w // 128, {} if case["decay_per"] == "head" else {"decay_rank": 64, "gate_rank": 64}
        return GatedDeltaSpec(hidden_size=w, num_heads=h, num_kv_heads=h, head_dim=128, v_head_dim=128, conv_taps=4,
                              decay_per=case["decay_per"], gate_activation="silu" if case["decay_per"] == "head" else "sigmoid", **ranks)
    if kind == "latent":
        s = _latent_sizes(w)
        return LatentAttentionSpec(hidden_size=w, num_heads=s["heads"], head_dim=s["dim"], rot_dim=s["rot"], v_head_dim=s["vdim"],
                                   q_rank=s["q_rank"], kv_rank=s["rank"], scale=128 ** -0.5, window=case["window"] or None, sink=True,
                                   position=RotarySpec(rotary_dim=s["rot"], theta=s["base"]))
    h = w // 128
    return RetentionSpec(hidden_size=w, num_heads=h, head_dim=128, v_head_dim=128, decays=tuple(_decays(h)),
                         position=RotarySpec(rotary_dim=128, theta=1e6))


class _Graphed:
    """A forward pass captured once, replayed per call."""

    def __init__(self, fn):
        self.fn = fn            # it holds the tensors that the graph reads
        fn()
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.out = fn()

    def __call__(self):
        self.graph.replay()
        return self.out


def _prepare_generate(case, seed):
    m2 = case["design"] == "m2"
    cfg = _m2_config() if m2 else _hybrid_config()
    prompts, answers = _token_ids(case, seed, M2["vocab"] if m2 else cfg["vocab"])
    most = max(len(p) for p in prompts) + case["steps"]
    pages = sum(-(-(len(p) + case["steps"]) // PAGE) for p in prompts) + case["requests"]
    runner = build_runner(cfg, dtype="bfloat16" if case["dtype"] == "bf16" else "float32", page_size=PAGE, num_pages=pages,
                          max_rows=case["requests"], max_seq_len=-(-most // PAGE) * PAGE, random_weights=True, seed=int(seed))
    shapes = _shapes(case)
    for p in runner.model.params():
        t = getattr(p.owner, p.name)
        shape = shapes[p.qualified][0]
        _fill(p.qualified, t[:shape[0]], seed)
    ids = list(range(case["requests"]))
    return {"runner": runner, "ids": ids, "prompts": prompts, "answers": answers}


def prepare(case, seed):
    if case["kind"] == "generate":
        return _prepare_generate(case, seed)
    dtype = DTYPES[case["dtype"]]
    spec = _spec(case)
    part = (make_feed_forward if case["kind"] == "experts" else make_mixer)(spec, dtype)
    part.bind(_weights(case, seed))
    x = _layer_input(case, seed)
    state = {"part": part, "x": x}
    if case["kind"] == "experts":
        fn = lambda: part.forward(x, None)      # noqa: E731
        state["run"] = _Graphed(fn) if case["tokens"] <= GRAPH_TOKENS else fn
        return state
    step = _step_context(case)
    if case["kind"] in ("attention", "latent"):
        table, pages = _pages(case, seed)
        slot = LayerSlot(kv=_cache(case, seed, pages), table=table, page_size=PAGE)
        state["kept"] = slot.kv
        fn = lambda: part.forward(x, step, slot)        # noqa: E731
    else:
        slot = LayerSlot(state=torch.zeros(case["requests"], *part.state_request().shape, device="cuda"))
        state["kept"] = slot.state

        def fn():
            slot.state.zero_()                  # what admitting the requests does
            return part.forward(x, step, slot)
    state["run"] = _Graphed(fn) if max(step.q_lens) == 1 and step.num_tokens <= GRAPH_TOKENS else fn
    return state


def run(state):
    if "runner" not in state:
        y = state["run"]()
        return {"y": y, "kept": state["kept"]} if "kept" in state else {"y": y}
    runner, ids, out = state["runner"], state["ids"], []
    for s in ids:
        runner.admit(s)
    out.append(runner.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(ids, state["prompts"])]))
    for tokens in state["answers"]:
        out.append(runner.step([StepEntry(s, [t], [0]) for s, t in zip(ids, tokens)]).clone())      # the next step writes it anew
    for s in ids:
        runner.release(s)
    return {"logits": torch.stack(out)}


# ---- what a pass cannot do without ---------------------------------------------------------------

def _seen(case):
    """(query, key) pairs that attention visits, and the key rows that are read."""
    w = case.get("window") or 0
    pairs = rows = 0
    for h, t in zip(_held(case), _lengths(case)):
        first = h + 1
        if w:
            pairs += sum(min(w, p) for p in range(first, first + t))
            rows += min(h + t, w + t - 1)
        else:
            pairs += t * h + t * (t + 1) // 2
            rows += h + t
    return pairs, rows


def _experts_work(tokens, size):
    m = M2
    used = m["experts"] * (1.0 - (1.0 - m["top"] / m["experts"]) ** tokens)
    return {"bytes": used * 3 * m["hidden"] * m["inter"] * size + m["experts"] * m["hidden"] * 4 + 2 * tokens * m["hidden"] * size,
            "flops": tokens * (m["top"] * 6.0 * m["hidden"] * m["inter"] + 2.0 * m["hidden"] * m["experts"])}


def _attention_work(tokens, pairs, rows, size):
    m = M2
    q, k = m["heads"] * m["dim"], m["kv_heads"] * m["dim"]
    mats = m["hidden"] * (q + 2 * k) + q * m["hidden"]
    return {"bytes": mats * size + 2 * tokens * m["hidden"] * size + 2 * rows * k * size,
            "flops": 2.0 * tokens * mats + 4.0 * pairs * q}


def _mixer_work(case, tokens, requests, size):
    """Products and recurrence of a recurrent mixer: per token and state element a decay, an update and a read-out."""
    mats = sum(math.prod(s) for n, (s, _) in _shapes(case).items() if n in ("in_proj", "o", "a2", "g2"))
    if case["kind"] == "state_space":
        s = _state_sizes(case["width"])
        state, per = s["heads"] * s["vdim"] * s["state"], 5.0
    else:
        state, per = case["width"] * 128, 7.0 if case["kind"] == "delta" else 5.0
    return {"bytes": mats * size + 2 * tokens * case["width"] * size + requests * state * 4, "flops": 2.0 * tokens * mats + per * tokens * state}


def work(case):
    size = 2 if case["dtype"] == "bf16" else 4
    kind = case["kind"]
    if kind == "experts":
        return _experts_work(case["tokens"], size)
    lens = _lengths(case)
    tokens = sum(lens)
    if kind == "attention":
        return _attention_work(tokens, *_seen(case), size)
    if kind == "latent":
        s, (pairs, rows) = _latent_sizes(case["width"]), _seen(case)
        mats = sum(math.prod(v) for n, (v, _) in _shapes(case).items() if len(v) == 2)
        # scores and sums over per-head keys of dim + rot and values of vdim
        return {"bytes": mats * size + 2 * tokens * case["width"] * size + rows * (s["rank"] + s["rot"]) * size,
                "flops": 2.0 * tokens * mats + 2.0 * pairs * s["heads"] * (s["dim"] + s["rot"] + s["vdim"])}
    if kind != "generate":
        return _mixer_work(case, tokens, case["requests"], size)
    # the prompt step, then the decode steps
    n, steps, total = case["requests"], case["steps"], {"bytes": 0.0, "flops": 0.0}
    passes = [(lens, [0] * n)] + [([1] * n, [t + i for t in lens]) for i in range(steps)]
    for brought, held in passes:
        t = sum(brought)
        pairs = sum(b * h + b * (b + 1) // 2 for b, h in zip(brought, held))
        rows = sum(b + h for b, h in zip(brought, held))
        if case["design"] == "m2":
            parts = [_attention_work(t, pairs, rows, size), _experts_work(t, size)] * 2
            parts.append({"bytes": M2["vocab"] * (M2["hidden"] + n) * size, "flops": 2.0 * n * M2["vocab"] * M2["hidden"]})
        else:
            w = _hybrid_config()["width"]
            mats = {"own": w * (w + w // 2) + w * w, "borrowed": 2 * w * w, "ff": 8 * w * w, "head": 32768 * w}
            parts = [{"bytes": (mats[k] + 2 * rows * w // 4) * size, "flops": 2.0 * t * mats[k] + 4.0 * pairs * w} for k in ("own", "borrowed")]
            parts += [{"bytes": mats["ff"] * size, "flops": 2.0 * t * mats["ff"]}] * 4
            parts.append({"bytes": (mats["head"] + n * 32768) * size, "flops": 2.0 * n * mats["head"]})
            for c in ({"kind": "state_space", "width": w}, {"kind": "delta", "width": w, "decay_per": "channel"}):
                one = _mixer_work(c, t, n, size)
                state = n * w * 128 * 4 * (2 if c["kind"] == "state_space" else 1)
                parts.append({"bytes": one["bytes"] + (0 if held == [0] * n else state), "flops": one["flops"]})
        for p in parts:
            total = {k: total[k] + p[k] for k in total}
    return total


def tolerance(case):
    """About four times what the path is off from 64 bits: 32-bit layers 1e-6 to 1e-5 (angles of late positions most),
    16-bit ones 4e-3; in a whole 16-bit model of routed experts a near-tie of two experts moves single tokens (2e-2 over all)."""
    if case["dtype"] == "fp32":
        return {"rel": 4e-5, "max": 5e-3}
    if case["kind"] == "generate":
        return {"rel": 3e-2, "max": 1.0 - 1e-9}
    return {"rel": 1.8e-2, "max": 0.6}


# ---- the same in 64 bits ---------------------------------------------------------------------------

def _rms64(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rope64(x, pos, dims, theta):
    """Split halves of the first ``dims`` of x [T, heads, D] rotated by position."""
    freq = (1.0 / (theta ** (torch.arange(0, dims, 2, dtype=torch.float32) / dims))).double().to(x.device)
    a = pos.double()[:, None] * freq
    c, s, h = a.cos()[:, None], a.sin()[:, None], dims // 2
    u, v = x[..., :h], x[..., h:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _attend64(q, k, v, pos, scale, window=0, sink=None):
    """q [T, H, d] at positions ``pos``; k, v [S, G, *] at positions 0..S-1."""
    (T, H, d), (S, G), dv = q.shape, k.shape[:2], v.shape[2]
    kt, vt, out = k.permute(1, 2, 0), v.transpose(0, 1), q.new_empty(T, H, dv)
    at = torch.arange(S, device=q.device)
    block = max(1, min(T, int(2e8) // (H * S)))
    for a in range(0, T, block):
        b = min(T, a + block)
        p = pos[a:b, None]
        hidden = at[None] > p if not window else (at[None] > p) | (at[None] <= p - window)
        s = torch.matmul(q[a:b].view(b - a, G, H // G, d).permute(1, 2, 0, 3).reshape(G, -1, d), kt).view(H, b - a, S).mul_(scale)
        s.masked_fill_(hidden[None], float("-inf"))
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink.view(H, 1, 1))
        s.sub_(top).exp_()
        den = s.sum(-1, keepdim=True)
        if sink is not None:
            den = den + (sink.view(H, 1, 1) - top).exp()
        o = torch.matmul(s.view(G, -1, S), vt).view(H, b - a, dv) / den
        out[a:b] = o.transpose(0, 1)
    return out


def _experts64(x, w, p=""):
    m = M2
    score = torch.sigmoid(x @ w[p + "gate"].double().t())
    idx = torch.topk(score + w[p + "selection_bias"].double(), m["top"], -1).indices
    share = score.gather(1, idx)
    share = share / share.sum(-1, keepdim=True)
    y = torch.zeros_like(x)
    for e in range(m["experts"]):
        t, slot = (idx == e).nonzero(as_tuple=True)
        if t.numel():
            g, u = (x[t] @ w[p + "w13"][e].double().t()).chunk(2, -1)
            y.index_add_(0, t, (torch.nn.functional.silu(g) * u) @ w[p + "w2"][e].double().t() * share[t, slot][:, None])
    return y


def _m2_qkv64(x, w, p, pos):
    m = M2
    T = x.shape[0]
    q, k, v = (x @ w[p + "qkv"].double().t()).split([m["heads"] * 128, m["kv_heads"] * 128, m["kv_heads"] * 128], -1)
    q = _rope64(_rms64(q, w[p + "q_norm"].double(), m["eps"]).view(T, -1, 128), pos, m["rot"], m["theta"])
    k = _rope64(_rms64(k, w[p + "k_norm"].double(), m["eps"]).view(T, -1, 128), pos, m["rot"], m["theta"])
    return q, k, v.view(T, -1, 128)


def _conv64(x, w, bias):
    taps = w.shape[1]
    pad = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x], 0)
    y = sum(pad[j:j + x.shape[0]] * w[:, j].double() for j in range(taps))
    return torch.nn.functional.silu(y if bias is None else y + bias.double()), pad[x.shape[0]:]


def _state_space64(x, w, p, width):
    """(output, final state row) of one request's tokens."""
    s, T = _state_sizes(width), x.shape[0]
    H, P, N, G = s["heads"], s["vdim"], s["state"], s["groups"]
    inner = H * P
    z, xbc, dt = (x @ w[p + "in_proj"].double().t()).split([inner, inner + 2 * G * N, H], -1)
    xbc, carried = _conv64(xbc, w[p + "conv_w"], w[p + "conv_b"])
    xs, B, C = xbc[:, :inner].view(T, H, P), xbc[:, inner:inner + G * N].view(T, G, N), xbc[:, inner + G * N:].view(T, G, N)
    B, C = B.repeat_interleave(H // G, 1), C.repeat_interleave(H // G, 1)
    dt = torch.nn.functional.softplus(dt + w[p + "dt_bias"].double())
    keep = torch.exp(-torch.exp(w[p + "a_log"].double()) * dt)[..., None, None]
    xd = xs * dt[..., None]
    S, y = x.new_zeros(H, N, P), x.new_empty(T, H, P)
    for t in range(T):
        S.mul_(keep[t]).baddbmm_(B[t][:, :, None], xd[t][:, None])
        torch.bmm(C[t][:, None], S, out=y[t][:, None])
    y = (y + w[p + "d_skip"].double()[:, None] * xs).reshape(T, inner) * torch.nn.functional.silu(z)
    n = s["norm_groups"]
    y = _rms64(y.view(T, n, -1), 1.0, 1e-6).reshape(T, inner) * w[p + "norm_w"].double()
    return y @ w[p + "o"].double().t(), torch.cat([S.transpose(1, 2).flatten(), carried.flatten()])


def _delta64(x, w, p, width, decay_per):
    T, H, d = x.shape[0], width // 128, 128
    vv, per_head = H * d, decay_per == "head"
    F = torch.nn.functional
    proj = x @ w[p + "in_proj"].double().t()
    qkv, carried = _conv64(proj[:, :3 * vv], w[p + "conv_w"], None)
    q, k, v = (t.view(T, H, d) for t in qkv.split(vv, -1))
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(proj[:, 3 * vv:3 * vv + H])
    rest = proj[:, 3 * vv + H:]
    if per_head:
        a, gate = rest[:, :H, None], F.silu(rest[:, H:])
        a = a + w[p + "dt_bias"].double().view(H, 1)
    else:
        a = (rest[:, :64] @ w[p + "a2"].double().t() + w[p + "dt_bias"].double()).view(T, H, d)
        gate = torch.sigmoid(rest[:, 64:] @ w[p + "g2"].double().t())
    keep = torch.exp(-torch.exp(w[p + "a_log"].double())[:, None] * F.softplus(a))[..., None]        # [T, H, 1 or d, 1]
    S, o = x.new_zeros(H, d, d), x.new_empty(T, H, d)
    for t in range(T):
        S.mul_(keep[t])
        u = beta[t][:, None, None] * (v[t][:, None] - torch.bmm(k[t][:, None], S))
        S.baddbmm_(k[t][:, :, None], u)
        torch.bmm(q[t][:, None], S, out=o[t][:, None])
    o = _rms64(o, w[p + "norm_w"].double(), 1e-6).reshape(T, vv) * gate
    return o @ w[p + "o"].double().t(), torch.cat([S.transpose(1, 2).flatten(), carried.flatten()])


def _retention64(x, w, width):
    T, H = x.shape[0], width // 128
    pos = torch.arange(T, device=x.device)
    q, k, v, g = (x @ w["in_proj"].double().t()).split(width, -1)
    q = _rope64(q.view(T, H, 128), pos, 128, 1e6)
    k, v = _rope64(k.view(T, H, 128), pos, 128, 1e6) * 128 ** -0.5, v.view(T, H, 128)
    keep = torch.tensor(_decays(H), dtype=torch.float32).double().to(x.device).view(H, 1, 1)
    S, o = x.new_zeros(H, 128, 128), x.new_empty(T, H, 128)
    for t in range(T):
        S.mul_(keep).baddbmm_(k[t][:, :, None], v[t][:, None])
        torch.bmm(q[t][:, None], S, out=o[t][:, None])
    o = _rms64(o, 1.0, 1e-6).reshape(T, width) * torch.nn.functional.silu(g)
    return o @ w["o"].double().t(), S.flatten()


def _latent64(case, x, w, table, cache):
    s, T0 = _latent_sizes(case["width"]), 0
    H, d, r, rank = s["heads"], s["dim"], s["rot"], s["rank"]
    outs = []
    for j, (h, t) in enumerate(zip(_held(case), _lengths(case))):
        pos = torch.arange(h, h + t, device=x.device)
        proj = x[T0:T0 + t] @ w["down"].double().t()
        q = (_rms64(proj[:, :s["q_rank"]], w["q_norm"].double(), 1e-6) @ w["uq"].double().t()).view(t, H, d + r)
        c = _rms64(proj[:, s["q_rank"]:s["q_rank"] + rank], w["kv_norm"].double(), 1e-6)
        kr = _rope64(proj[:, None, s["q_rank"] + rank:], pos, r, s["base"])[:, 0]
        where = (table[j].long()[:, None] * PAGE + torch.arange(PAGE, device=x.device)).flatten()
        flat = cache.view(-1, rank + r)
        flat[where[pos]] = torch.cat([c, kr], -1)
        first = max(0, h - case["window"] + 1) if case["window"] else 0
        rows = flat[where[first:h + t]]
        k = torch.cat([(rows[:, :rank] @ w["uk"].double().t()).view(-1, H, d), rows[:, None, rank:].expand(-1, H, r)], -1)
        v = (rows[:, :rank] @ w["uv"].double().t()).view(-1, H, s["vdim"])
        q = torch.cat([q[..., :d], _rope64(q[..., d:], pos, r, s["base"])], -1)
        o = torch.cat([_attend64(q[a:a + 1024], k[lo:a + 1024 + h - first], v[lo:a + 1024 + h - first],
                                 pos[a:a + 1024] - first - lo, 128 ** -0.5, case["window"], w["sink"].double())
                       for a in range(0, t, 1024)
                       for lo in [max(0, a + h - first - case["window"]) if case["window"] else 0]], 0)
        outs.append(o.reshape(t, -1) @ w["o"].double().t())
        T0 += t
    return {"y": torch.cat(outs, 0), "kept": cache}


def _attention64(case, x, w, table, cache):
    outs, T0 = [], 0
    for j, (h, t) in enumerate(zip(_held(case), _lengths(case))):
        pos = torch.arange(h, h + t, device=x.device)
        q, k, v = _m2_qkv64(x[T0:T0 + t], w, "", pos)
        page, slot = table[j].long()[pos // PAGE], pos % PAGE
        cache[page, 0, :, slot], cache[page, 1, :, slot] = k, v
        every = torch.arange(h + t, device=x.device)
        page, slot = table[j].long()[every // PAGE], every % PAGE
        o = _attend64(q, cache[page, 0, :, slot], cache[page, 1, :, slot], pos, M2["dim"] ** -0.5)
        outs.append(o.reshape(t, -1) @ w["o"].double().t())
        T0 += t
    return {"y": torch.cat(outs, 0), "kept": cache}


def _m2_logits64(w, seqs, wanted):
    """Logits [wanted places] of whole sequences."""
    m = M2
    xs = torch.cat([w["embed"][torch.tensor(s, device="cuda")].double() for s in seqs], 0)
    pos = torch.cat([torch.arange(len(s), device="cuda") for s in seqs])
    for i in range(2):
        p = f"layers.{i}."
        q, k, v = _m2_qkv64(_rms64(xs, w[p + "mixer_norm.weight"].double(), m["eps"]), w, p + "mixer.", pos)
        lens, o = [len(s) for s in seqs], []
        for a, b, c, d in zip(q.split(lens), k.split(lens), v.split(lens), pos.split(lens)):
            o.append(_attend64(a, b, c, d, m["dim"] ** -0.5))
        xs = xs + torch.cat(o, 0).reshape(len(xs), -1) @ w[p + "mixer.o"].double().t()
        xs = xs + _experts64(_rms64(xs, w[p + "feed_forward_norm.weight"].double(), m["eps"]), w, p + "feed_forward.")
    xs = _rms64(xs[wanted], w["final_norm.weight"].double(), m["eps"])
    return torch.cat([xs @ w["head"][a:a + 16384].double().t() for a in range(0, m["vocab"], 16384)], -1)


def _hybrid_logits64(w, seqs, wanted):
    cfg = _hybrid_config()
    width, eps = cfg["width"], 1e-6
    H, lens = width // 128, [len(s) for s in seqs]
    xs = torch.cat([w["embed"][torch.tensor(s, device="cuda")].double() for s in seqs], 0)
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    temp = 1.0 + 0.1 * torch.log(torch.div(pos + 1, 1024, rounding_mode="floor").double() + 1.0)

    def norm(x, p):
        mu = x.mean(-1, keepdim=True)
        x = x - mu
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w[p + "weight"].double() + w[p + "bias"].double()

    for i, layer in enumerate(cfg["layers"]):
        p = f"layers.{i}.mixer."
        if layer["type"] == "attention":
            proj = xs @ w[p + "qkv"].double().t()
            q = _rms64(proj[:, :width], w[p + "q_norm"].double(), eps) * temp[:, None]
            if layer["mixer"].get("kv_from") is None:
                kept = (_rms64(proj[:, width:width + width // 4], w[p + "k_norm"].double(), eps).view(-1, H // 4, 128),
                        proj[:, width + width // 4:].view(-1, H // 4, 128))
            y = [_attend64(a, b, c, d, 128 ** -0.5) for a, b, c, d in
                 zip(q.view(-1, H, 128).split(lens), kept[0].split(lens), kept[1].split(lens), pos.split(lens))]
            y = torch.cat(y, 0).reshape(len(xs), width) @ w[p + "o"].double().t()
        elif layer["type"] == "mamba2":
            y = torch.cat([_state_space64(x, w, p, width)[0] for x in xs.split(lens)], 0)
        else:
            y = torch.cat([_delta64(x, w, p, width, "channel")[0] for x in xs.split(lens)], 0)
        xs = norm(2.0 * xs + y, f"layers.{i}.mixer_norm.")
        y = torch.relu(xs @ w[f"layers.{i}.feed_forward.up"].double().t()) ** 2 @ w[f"layers.{i}.feed_forward.down"].double().t()
        xs = norm(2.0 * xs + y, f"layers.{i}.feed_forward_norm.")
    xs = norm(xs[wanted], "final_norm.")
    return 30.0 * torch.tanh(xs @ w["head"].double().t() / 30.0)


@torch.no_grad()
def exact(case, seed):
    w = _weights(case, seed)
    if case["kind"] == "generate":
        if case["design"] == "hybrid" and case["requests"] * (case["tokens"] + case["steps"]) > 20000:
            return None
        m2 = case["design"] == "m2"
        prompts, answers = _token_ids(case, seed, M2["vocab"] if m2 else 32768)
        seqs = [p + [a[j] for a in answers] for j, p in enumerate(prompts)]
        base, wanted = 0, []
        for p, s in zip(prompts, seqs):
            wanted.append(torch.arange(base + len(p) - 1, base + len(s)))
            base += len(s)
        wanted = torch.stack(wanted, 1).flatten().cuda()                # [steps + 1, requests]
        logits = (_m2_logits64 if m2 else _hybrid_logits64)(w, seqs, wanted)
        return {"logits": logits.view(case["steps"] + 1, case["requests"], -1)}
    x = _layer_input(case, seed).double()
    if case["kind"] == "experts":
        return {"y": _experts64(x, w)}
    if case["kind"] in ("attention", "latent"):
        table, pages = _pages(case, seed)
        return (_attention64 if case["kind"] == "attention" else _latent64)(case, x, w, table, _cache(case, seed, pages).double())
    ys = []
    for part in x.split(_lengths(case)):
        if case["kind"] == "state_space":
            ys.append(_state_space64(part, w, "", case["width"]))
        elif case["kind"] == "delta":
            ys.append(_delta64(part, w, "", case["width"], case["decay_per"]))
        else:
            ys.append(_retention64(part, w, case["width"]))
    return {"y": torch.cat([y for y, _ in ys], 0), "kept": torch.stack([s for _, s in ys])}
