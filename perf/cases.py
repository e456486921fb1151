"""What a program that serves models with this package has it do, as cases that can be timed and compared.

Two kinds of entry point are used.  ``step`` cases are whole calls of the step function on a model of the 1B
benchmark shape with half its layers (differences of rounding grow with the depth; ``ModelRunner``), which replays its steps of
single tokens from captured graphs.  All others are one
part of a layer, or one whole layer, run on one step's batch against a paged cache or state slots, as the model runs
them: a mixer, a feed-forward or a block with its tensors, built once, and the batch's descriptors, laid out once a step.

Sizes are those of the repository's benchmark: the 1B, 3B and 8B shapes, and the comparison's widths 1024 and 2048 for
the mixers of the other designs.  Weights are random as there; activations that a norm made are N(0, 1); decay and gate
parameters follow the customary initialisation of such mixers, so that states neither vanish nor blow up.

A case names the step's requests: ``single`` requests decode one token each, with contexts spread evenly from ``ctx_lo`` to
``ctx_hi``; ``runs`` lists prompt portions as "start:tokens", separated by commas.
"""

import math

import numpy as np
import torch

PAGE = 16
LAYER_1B = dict(hidden=2048, inter=8192, heads=32, kv_heads=8, dim=64, factor=32.0)
LAYER_3B = dict(hidden=3072, inter=8192, heads=24, kv_heads=8, dim=128, factor=32.0)
LAYER_8B = dict(hidden=4096, inter=14336, heads=32, kv_heads=8, dim=128, factor=8.0)
LAYERS = {"1b": LAYER_1B, "3b": LAYER_3B, "8b": LAYER_8B}
STEP_LAYERS, STEP_VOCAB = 8, 128256
ROPE = {"rope_type": "llama3", "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}
EPS = 1e-6
STD = 0.02


def listed():
    return [
        # the smallest call: one user's next token, a whole model, replayed from a graph; bound by latency and launches
        {"name": "step_decode_1", "kind": "step", "single": 1, "ctx_lo": 200, "ctx_hi": 200},
        # an ordinary serving step: a few dozen users' next tokens beside each other, contexts of a chat
        {"name": "step_decode_48", "kind": "step", "single": 48, "ctx_lo": 70, "ctx_hi": 900},
        # decoding over long contexts at the 8B shape: the attention part reads most of what a step reads
        {"name": "attention_decode_8b", "kind": "attention", "shape": "8b", "single": 24, "ctx_lo": 500, "ctx_hi": 7900},
        # reading a prompt: one layer of the 1B shape on a full portion of the token budget
        {"name": "block_prompt_1b", "kind": "block", "shape": "1b", "dtype": "bfloat16", "runs": "0:2048"},
        # continuous batching: one layer of the 3B shape on a prompt's later portion beside decoding requests
        {"name": "block_mixed_3b", "kind": "block", "shape": "3b", "dtype": "bfloat16", "single": 40, "ctx_lo": 100,
         "ctx_hi": 2500, "runs": "512:701"},
        # the true 32-bit mode: one layer of the 1B shape, a short prompt beside decoding requests
        {"name": "block_float32_1b", "kind": "block", "shape": "1b", "dtype": "float32", "single": 5, "ctx_lo": 40, "ctx_hi": 700,
         "runs": "0:333"},
        # attention over a cached latent, prompts of two requests (one continued)
        {"name": "latent_prompt", "kind": "latent", "width": 2048, "runs": "0:1400,600:648"},
        # the gated delta rule with its short convolution, a long prompt beside a shorter one
        {"name": "delta_prompt", "kind": "delta", "width": 2048, "runs": "0:1548,0:500"},
        # the matrix memory with exponential gates, one full portion
        {"name": "mlstm_prompt", "kind": "mlstm", "width": 2048, "runs": "0:2048"},
        # state-space duality, three ragged prompts
        {"name": "ssd_prompt", "kind": "ssd", "width": 2048, "runs": "0:1111,0:700,0:237"},
        # routed experts with a shared one, the tokens of a prompt portion
        {"name": "experts_prompt", "kind": "experts", "width": 2048, "tokens": 2048},
        # decoding with attention over blocks of positions, many users
        {"name": "chunk_attention_decode", "kind": "chunk_attention", "width": 2048, "single": 64, "ctx_lo": 30, "ctx_hi": 3000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_runs(rng, most, starts):
    """One to three portions of together at most ``most`` tokens, log-uniform, ragged."""
    total, n = _log(rng, 64, most), rng.choice((1, 1, 2, 3))
    cuts = sorted(rng.randrange(1, total) for _ in range(n - 1))
    counts = [b - a for a, b in zip([0] + cuts, cuts + [total]) if b > a]
    return ",".join("%d:%d" % (rng.choice((0, rng.randrange(1, 1500))) if starts else 0, c) for c in counts)


def draw(rng):
    kind = rng.choice(("step", "attention", "block", "block", "mixed", "float32", "latent", "delta", "mlstm", "ssd", "experts",
                       "chunk_attention"))
    if kind == "step":
        lo = rng.randrange(4, 500)
        return {"kind": "step", "single": _log(rng, 1, 64), "ctx_lo": lo, "ctx_hi": lo + rng.randrange(0, 700)}
    if kind == "attention":
        lo = rng.randrange(4, 2000)
        return {"kind": "attention", "shape": rng.choice(("1b", "3b", "8b")), "single": _log(rng, 8, 64), "ctx_lo": lo,
                "ctx_hi": lo + rng.randrange(500, 4000)}
    if kind == "block":
        return {"kind": "block", "shape": rng.choice(("1b", "3b")), "dtype": "bfloat16", "runs": _draw_runs(rng, 2048, True)}
    if kind == "mixed":
        lo = rng.randrange(4, 1000)
        return {"kind": "block", "shape": rng.choice(("1b", "3b")), "dtype": "bfloat16", "single": _log(rng, 2, 60), "ctx_lo": lo,
                "ctx_hi": lo + rng.randrange(0, 3000), "runs": _draw_runs(rng, 1500, True)}
    if kind == "float32":
        lo = rng.randrange(4, 500)
        return {"kind": "block", "shape": "1b", "dtype": "float32", "single": _log(rng, 1, 16), "ctx_lo": lo,
                "ctx_hi": lo + rng.randrange(0, 800), "runs": _draw_runs(rng, 512, True)}
    if kind == "experts":
        return {"kind": "experts", "width": rng.choice((1024, 2048)), "tokens": _log(rng, 16, 2048)}
    if kind == "chunk_attention":
        lo = rng.randrange(4, 1500)
        return {"kind": kind, "width": rng.choice((1024, 2048)), "single": _log(rng, 8, 128), "ctx_lo": lo,
                "ctx_hi": lo + rng.randrange(200, 2500)}
    return {"kind": kind, "width": rng.choice((1024, 2048)), "runs": _draw_runs(rng, 2048, kind == "latent")}


# ------------------------------------------------------------------ what a case is made of

def _requests(case):
    """[(start, tokens)] of the step's requests, those that decode first."""
    n = int(case.get("single", 0))
    lo, hi = int(case.get("ctx_lo", 1)), int(case.get("ctx_hi", 1))
    out = [(lo + (hi - lo) * i // max(1, n - 1) - 1 if n > 1 else lo - 1, 1) for i in range(n)]
    for part in str(case.get("runs", "")).split(","):
        if part:
            start, tokens = part.split(":")
            out.append((int(start), int(tokens)))
    return out


def _dtype(case):
    return getattr(torch, case.get("dtype", "bfloat16"))


class _Draws:
    """Tensors drawn on the device from one seed, in the order in which they are asked for."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(int(seed))

    def normal(self, shape, std=1.0, mean=0.0, dtype=torch.float32):
        return (torch.randn(tuple(shape), generator=self.gen, dtype=torch.float32, device="cuda") * std + mean).to(dtype)

    def uniform(self, shape, lo, hi):
        return torch.rand(tuple(shape), generator=self.gen, dtype=torch.float32, device="cuda") * (hi - lo) + lo


def _latent_sizes(width):
    if width == 2048:
        return dict(heads=16, dim=128, rot=64, vdim=128, q_rank=768, rank=512)
    return dict(heads=8, dim=64, rot=32, vdim=64, q_rank=384, rank=256)


def _inputs(case, seed):
    """The case's weights, activations and cached rows: the same for the package and for ``exact``."""
    d, dt, kind = _Draws(seed), _dtype(case), case["kind"]
    w, out = {}, {}
    reqs = _requests(case)
    T = sum(n for _, n in reqs) or int(case.get("tokens", 0))

    def mat(name, *shape):
        w[name] = d.normal(shape, STD, dtype=dt)

    if kind in ("attention", "block"):
        z = LAYERS[case["shape"]]
        H, nq, nkv, D, I = z["hidden"], z["heads"], z["kv_heads"], z["dim"], z["inter"]
        mat("q", nq * D, H), mat("k", nkv * D, H), mat("v", nkv * D, H), mat("o", H, nq * D)
        if kind == "block":
            mat("gate", I, H), mat("up", I, H), mat("down", H, I)
            for n in ("norm1", "norm2", "norm3"):
                w[n] = d.normal((H,), STD, 1.0)
        out["rows"] = [(d.normal((s, nkv, D), dtype=dt), d.normal((s, nkv, D), dtype=dt)) if s else None for s, _ in reqs]
        out["x"] = d.normal((T, H), dtype=dt if kind == "attention" else torch.float32)
        return w, out
    W = int(case["width"])
    heads = W // 64
    if kind == "latent":
        z = _latent_sizes(W)
        h, D, r, V, qr, kr = (z[k] for k in ("heads", "dim", "rot", "vdim", "q_rank", "rank"))
        mat("dq", qr, W), mat("uq", h * (D + r), qr), mat("dkv", kr + r, W), mat("uk", h * D, kr), mat("uv", h * V, kr), mat("o", W, h * V)
        w["dq_norm"], w["dkv_norm"], w["sink"] = d.normal((qr,), STD, 1.0), d.normal((kr,), STD, 1.0), d.normal((h,))
        out["rows"] = [d.normal((s, 1, kr + r), dtype=dt) if s else None for s, _ in reqs]
    elif kind == "delta":
        G = heads // 4
        mat("q", G * 64, W), mat("k", G * 64, W), mat("v", W, W), mat("b", heads, W), mat("a", heads, W), mat("g", W, W), mat("o", W, W)
        for n, c in (("q_conv", G * 64), ("k_conv", G * 64), ("v_conv", W)):
            w[n] = d.normal((c, 4), 0.5)
        w["A_log"] = d.uniform((heads,), 1.0, 16.0).log()
        w["dt_bias"] = torch.expm1(d.uniform((heads,), math.log(1e-3), math.log(0.1)).exp()).log()
        w["norm"] = d.normal((64,), STD, 1.0)
    elif kind == "mlstm":
        for n in ("q", "k", "v", "g", "o"):
            mat(n, W, W)
        mat("i", heads, W), mat("f", heads, W)
        w["i_bias"], w["f_bias"] = d.normal((heads,), 0.1), torch.linspace(3.0, 6.0, heads, device="cuda")
        w["norm"] = d.normal((W,), STD, 1.0)
    elif kind == "ssd":
        inner, N, G = 2 * W, 128, 8
        hs = inner // 64
        mat("in", 2 * inner + 2 * G * N + hs, W), mat("o", W, inner)
        w["conv"], w["conv_bias"] = d.normal((inner + 2 * G * N, 4), 0.5), d.normal((inner + 2 * G * N,), 0.1)
        w["dt_bias"] = torch.expm1(d.uniform((hs,), math.log(1e-3), math.log(0.1)).exp()).log()
        w["A_log"], w["D"], w["norm"] = d.uniform((hs,), 1.0, 16.0).log(), d.normal((hs,), 0.1, 1.0), d.normal((inner,), STD, 1.0)
    elif kind == "experts":
        E, F, S = 32, W // 8, W
        mat("router", E, W)
        for e in range(E):
            mat("gate%d" % e, F, W), mat("up%d" % e, F, W), mat("down%d" % e, W, F)
        mat("shared_gate", S, W), mat("shared_up", S, W), mat("shared_down", W, S), mat("shared_sg", 1, W)
    elif kind == "chunk_attention":
        G = heads // 4
        mat("q", W, W), mat("k", G * 64, W), mat("v", G * 64, W), mat("o", W, W)
        for n, c in (("q_bias", W), ("k_bias", G * 64), ("v_bias", G * 64), ("o_bias", W)):
            w[n] = d.normal((c,), STD)
        w["q_norm"], w["k_norm"], w["sink"] = d.normal((W,), STD, 1.0), d.normal((G * 64,), STD, 1.0), d.normal((heads,))
        out["rows"] = [d.normal((s, G, 128), dtype=dt) if s else None for s, _ in reqs]
    out["x"] = d.normal((T, W), dtype=dt)
    return w, out


def _params(case):
    """(registered kind of the mixer or feed-forward, its sizes and constants) of the cases that run one part."""
    from kv_cache_optimization_for_llm_b200.models.spec import PartSpec
    kind = case["kind"]
    if kind in ("attention", "block"):
        z = LAYERS[case["shape"]]
        rope = PartSpec("rope", {"head_dim": z["dim"], "rotary_dim": z["dim"], "theta": 500000.0,
                                 "scaling": dict(ROPE, factor=z["factor"])})
        return "attention", {"hidden_size": z["hidden"], "num_heads": z["heads"], "num_kv_heads": z["kv_heads"],
                             "head_dim": z["dim"], "window": None, "position": rope}
    W = int(case["width"])
    heads = W // 64
    if kind == "latent":
        z = _latent_sizes(W)
        rope = PartSpec("rope_interleaved", {"dims": z["rot"], "base": 10000.0})
        return "latent_attention", {"hidden_size": W, "heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot"], "vdim": z["vdim"],
                                    "q_rank": z["q_rank"], "kv_rank": z["rank"], "scale": (z["dim"] + z["rot"]) ** -0.5,
                                    "eps": EPS, "position": rope}
    if kind == "delta":
        return "gated_delta", {"hidden_size": W, "heads": heads, "kv_heads": heads // 4, "dim": 64, "vdim": 64, "conv": 4, "eps": EPS}
    if kind == "mlstm":
        return "mlstm", {"hidden_size": W, "heads": heads, "dim": 64, "vdim": 64, "gate_cap": 15.0, "eps": EPS}
    if kind == "ssd":
        return "state_space_duality", {"hidden_size": W, "heads": 2 * W // 64, "vdim": 64, "state": 128, "groups": 8,
                                       "norm_groups": 8, "conv": 4, "eps": EPS}
    if kind == "experts":
        return "limited_experts", {"hidden_size": W, "experts": 32, "top": 4, "expert_ff": W // 8, "limit": 7.0, "shared_ff": W,
                                   "shared_limit": 7.0, "alpha": 1.702}
    rope = PartSpec("rope", {"head_dim": 64, "rotary_dim": 64, "theta": 10000.0, "scaling": None})
    return "rotary_chunk_attention", {"hidden_size": W, "heads": heads, "kv_heads": heads // 4, "dim": 64, "vdim": 64,
                                      "scale": 0.125, "chunk": 1024, "softcap": None, "sink": True, "gate": False, "bias": True,
                                      "qk_norm": True, "eps": EPS, "position": rope}


# ------------------------------------------------------------------ the package's side

def _step_config():
    return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": STEP_VOCAB, "hidden_size": 2048,
            "intermediate_size": 8192, "num_hidden_layers": STEP_LAYERS, "num_attention_heads": 32, "num_key_value_heads": 8,
            "head_dim": 64, "rms_norm_eps": 1e-5, "rope_theta": 500000.0, "rope_scaling": dict(ROPE, factor=32.0),
            "max_position_embeddings": 131072, "tie_word_embeddings": True, "hidden_act": "silu"}


def _step_tokens(case, seed):
    rng = np.random.default_rng(int(seed))
    return [rng.integers(0, STEP_VOCAB, s + 1).tolist() for s, _ in _requests(case)]


def _prepare_step(case, seed):
    from kv_cache_optimization_for_llm_b200 import EngineConfig
    from kv_cache_optimization_for_llm_b200.engine.batch import StepEntry
    from kv_cache_optimization_for_llm_b200.engine.runner import ModelRunner
    tokens = _step_tokens(case, seed)
    pages = sum(-(-len(t) // PAGE) for t in tokens)
    runner = ModelRunner(None, EngineConfig(dtype="bfloat16", page_size=PAGE, num_pages=pages, max_num_seqs=64,
                                            max_num_batched_tokens=2048, max_model_len=4096),
                         random_init={"config": _step_config(), "seed": int(seed), "std": STD})
    group, held = [], 0
    for i, t in enumerate(tokens):      # the prompts are read as an engine reads them, up to 2048 tokens a step
        if held + len(t) - 1 > 2048:
            runner.step(group)
            group, held = [], 0
        if len(t) > 1:
            group.append(StepEntry(i, t[:-1], 0, ()))
            held += len(t) - 1
    if group:
        runner.step(group)
    entries = [StepEntry(i, [t[-1]], len(t) - 1, (0,)) for i, t in enumerate(tokens)]
    runner.step(entries)                # takes the pages of the decoded position and captures the step's graph
    return {"kind": "step", "runner": runner, "entries": entries}


def _fill(pool, table, rows):
    """Writes a request's earlier rows [n, heads, size] into its pages [pages, heads, PAGE, size]; pages that a window has given
    back are left out."""
    n = -(-rows.shape[0] // PAGE)
    padded = torch.zeros((n * PAGE,) + tuple(rows.shape[1:]), dtype=rows.dtype, device=rows.device)
    padded[:rows.shape[0]] = rows
    at = torch.as_tensor(np.asarray(table[:n]), dtype=torch.int64, device=rows.device)
    pool[at[at >= 0]] = padded.view(n, PAGE, *rows.shape[1:]).transpose(1, 2)[at >= 0]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _prepare_step(case, seed)
    from kv_cache_optimization_for_llm_b200 import ops
    from kv_cache_optimization_for_llm_b200.cache.paged_cache import PagedCache
    from kv_cache_optimization_for_llm_b200.cache.specs import paged_part
    from kv_cache_optimization_for_llm_b200.engine.arena import StepArena
    from kv_cache_optimization_for_llm_b200.engine.batch import BatchBuilder, StepEntry
    from kv_cache_optimization_for_llm_b200.parts import BuildContext, lookup
    torch.backends.cuda.matmul.allow_tf32 = False
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    dev, dt, reqs = torch.device("cuda:0"), _dtype(case), _requests(case)
    w, given = _inputs(case, seed)
    ctx = BuildContext(dtype=dt, device=dev, max_positions=8192, status=ops.kernel_status(dev))
    part_kind, params = _params(case)

    def make(family, name, prm, roles=None):
        cls = lookup(family, name)
        return cls(prm, {r: w[(roles or {}).get(r, r)] for r in cls.weight_specs(prm)}, ctx)

    state = {"kind": kind, "x": given["x"]}
    if kind == "experts":
        part = make("feed_forward", part_kind, params)
        parts, reqs, wish = [part], [(0, int(case["tokens"]))], None
    else:
        part = make("mixer", part_kind, params)
        parts, wish = [part], part.cache_spec()
    if kind == "block":
        z = LAYERS[case["shape"]]
        norms = [make("norm", "rmsnorm", {"size": z["hidden"], "eps": EPS}, {"weight": n}) for n in ("norm1", "norm2", "norm3")]
        ff = make("feed_forward", "swiglu", {"hidden_size": z["hidden"], "intermediate_size": z["inter"]})
        parts += norms[:2] + [ff]
        part = lookup("block", "prenorm")({"mixer": part, "mixer_norm": norms[0], "feed_forward": ff, "ff_norm": norms[1]})
        state["next_norm"], state["residual"] = norms[2], torch.empty_like(given["x"])
    T = sum(n for _, n in reqs)
    cache = PagedCache([wish], [None], PAGE, sum(-(-(s + n) // PAGE) for s, n in reqs), len(reqs), 8192, dt, dev)
    manager = cache.manager
    for i, (s, n) in enumerate(reqs):
        manager.admit(i)
        if s:
            manager.extend(i, s)
            manager.advance(i, s)
        manager.extend(i, s + n)
    binding = cache.binding(0)
    if paged_part(wish) is not None:
        for i, rows in enumerate(given["rows"]):
            if rows is not None:
                table = manager.block_table(i, 0)
                for pool, r in zip((binding.k, binding.v), rows if isinstance(rows, tuple) else (rows,)):
                    _fill(pool, table, r)
    heights = [h for p in parts if hasattr(p, "query_tile_heights") for h in p.query_tile_heights()]
    builder = BatchBuilder(T, len(reqs), cache.max_pages, dev, ctx.status, page_size=PAGE, tile_heights=heights)
    batch = builder.build([StepEntry(i, [0] * n, s, ()) for i, (s, n) in enumerate(reqs)], manager)
    widths = sum(sum(p.activation_widths()) for p in parts)
    arena = StepArena(dev, 8 * T * given["x"].shape[1] + (1 << 16), int(1.2 * dt.itemsize * T * widths) + (1 << 16))
    state.update(part=part, batch=batch, binding=binding, cache=cache, builder=builder, arena=arena)
    return state


def run(state):
    if state["kind"] == "step":
        return state["runner"].run(state["entries"])
    from kv_cache_optimization_for_llm_b200 import ops
    part, batch, binding, arena = state["part"], state["batch"], state["binding"], state["arena"]
    with ops.use_current_stream(), ops.use_arena(arena):
        arena.begin_step()
        arena.begin_layer()
        if state["kind"] == "block":
            # the stream as the layer before left it, this layer, and the norm in front of the next one, which adds what is pending
            residual, delta = part.forward(state["residual"].copy_(state["x"]), None, batch, binding)
            y = state["next_norm"].forward(residual, delta)
            return {"y": y, "residual": residual, "k": binding.k, "v": binding.v}
        if state["kind"] == "experts":
            return {"y": part.forward(state["x"], batch)}
        y = part.forward(state["x"], batch, binding)
    if state["kind"] == "attention":
        return {"y": y, "k": binding.k, "v": binding.v}
    if state["kind"] in ("latent", "chunk_attention"):
        return {"y": y, "rows": binding.k}
    return {"y": y, "state": binding.state}


# ------------------------------------------------------------------ the least a pass has to do

def work(case):
    kind, reqs = case["kind"], _requests(case)
    esize = _dtype(case).itemsize
    T = sum(n for _, n in reqs) or int(case.get("tokens", 0))
    pairs = sum(n * s + n * (n + 1) // 2 for s, n in reqs)      # (query, key) pairs of causal attention
    keys = sum(s + n for s, n in reqs)
    if kind == "step":
        layer = (32 + 16) * 64 * 2048 + 2048 * 2048 + 3 * 2048 * 8192
        weights = STEP_LAYERS * layer + STEP_VOCAB * 2048
        kv = STEP_LAYERS * 2 * 8 * 64
        return {"bytes": 2 * weights + 2 * kv * keys + 4 * T * STEP_VOCAB,
                "flops": 2 * T * weights + STEP_LAYERS * 4 * 32 * 64 * pairs}
    if kind in ("attention", "block"):
        z = LAYERS[case["shape"]]
        H, nq, nkv, D, I = z["hidden"], z["heads"], z["kv_heads"], z["dim"], z["inter"]
        mats = (2 * nq + 2 * nkv) * D * H + (3 * H * I if kind == "block" else 0)
        rows = (2 * esize if kind == "attention" else 4 + 4 + esize) * T * H      # in and out; a block reads and writes the stream
        return {"bytes": esize * (mats + 2 * nkv * D * (keys + T)) + rows, "flops": 2 * T * mats + 4 * nq * D * pairs}
    W = int(case["width"])
    heads = W // 64
    io = 2 * 2 * T * W
    if kind == "latent":
        z = _latent_sizes(W)
        h, D, r, V, qr, kr = (z[k] for k in ("heads", "dim", "rot", "vdim", "q_rank", "rank"))
        mats = qr * W + h * (D + r) * qr + (kr + r) * W + W * h * V
        up = h * (D + V) * kr
        return {"bytes": 2 * (mats + up + (kr + r) * (keys + T)) + io,
                "flops": 2 * T * mats + 2 * keys * up + 2 * h * (D + r + V) * pairs}
    if kind == "delta":
        mats = (heads // 2 * 64 + 3 * W + 2 * heads) * W
        return {"bytes": 2 * mats + io + len(reqs) * 4 * heads * 64 * 64, "flops": 2 * T * mats + T * heads * 64 * 64 * 7}
    if kind == "mlstm":
        mats = (5 * W + 2 * heads) * W
        return {"bytes": 2 * mats + io + len(reqs) * 4 * heads * 64 * 64, "flops": 2 * T * mats + T * heads * 64 * 64 * 5}
    if kind == "ssd":
        mats = (6 * W + 16 * 128 + 2 * heads) * W
        return {"bytes": 2 * mats + io + len(reqs) * 4 * 2 * W * 128, "flops": 2 * T * mats + T * 2 * W * 128 * 5}
    if kind == "experts":
        touched = min(32, 4 * T)
        return {"bytes": 2 * (32 * W + touched * 3 * W * (W // 8) + 3 * W * W) + io,
                "flops": 2 * T * (32 * W + 4 * 3 * W * (W // 8) + 3 * W * W)}
    seen = sum(s % 1024 + 1 for s, _ in reqs)       # keys of the query's own block
    mats = (2 * heads + heads // 2) * 64 * W
    return {"bytes": 2 * (mats + heads // 4 * 128 * (seen + T)) + io, "flops": 2 * T * mats + 4 * W * seen}


def tolerance(case):
    if case["kind"] == "step":
        return {"rel": 0.03, "max": 0.3}
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 2e-4}
    return {"rel": 0.016, "max": 0.15}


# ------------------------------------------------------------------ the same in 64 bits

def _rms(x, weight=None, eps=EPS):
    y = x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _frequencies(dim, theta, scaling=None):
    f = theta ** (-torch.arange(0, dim, 2, dtype=torch.float64, device="cuda") / dim)
    if scaling is None:
        return f
    orig, low, high = scaling["original_max_position_embeddings"], scaling["low_freq_factor"], scaling["high_freq_factor"]
    wave = 2.0 * math.pi / f
    smooth = ((orig / wave - low) / (high - low)).clamp(0.0, 1.0)
    return (1.0 - smooth) * f / scaling["factor"] + smooth * f


def _rotate(x, positions, f, pairs=False):
    """x [T, heads, dim] turned by positions * f; channel i with i + dim / 2, or 2 i with 2 i + 1."""
    a = positions.double()[:, None] * f[None, :]
    c, s = a.cos()[:, None], a.sin()[:, None]
    if pairs:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    u, v = x.chunk(2, -1)
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _attend(q, k, v, start, scale, sink=None, chunk=0):
    """q [n, heads, dim] of the positions from ``start`` on over k, v [end, kv heads, *] -> [n, heads, value size]."""
    n, H, _ = q.shape
    end, G = k.shape[0], k.shape[1]
    i = torch.arange(start, start + n, device=q.device)[:, None]
    j = torch.arange(end, device=q.device)[None, :]
    hidden = (j > i) | ((i // chunk != j // chunk) if chunk else (j < 0))
    out = torch.empty((n, H, v.shape[2]), dtype=q.dtype, device=q.device)
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[:, g].T * scale).masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        out[:, h] = torch.softmax(s, -1)[:, :end] @ v[:, g]
    return out


def _spans(reqs):
    t = 0
    for s, n in reqs:
        yield slice(t, t + n), s, n
        t += n


def _positions(s, n):
    return torch.arange(s, s + n, device="cuda")


def _conv(x, weight, bias=None):
    """Causal convolution per channel, zeros before the start; x [T, C], weight [C, taps]."""
    taps = weight.shape[1]
    p = torch.cat([x.new_zeros((taps - 1, x.shape[1])), x])
    y = sum(p[j:j + x.shape[0]] * weight[:, j] for j in range(taps))
    return y if bias is None else y + bias


def _exact_part(case, w, given):
    """The output rows [T, width] of a mixer or feed-forward in 64 bits."""
    kind, reqs, x = case["kind"], _requests(case), given["x"].double()
    F = torch.nn.functional
    if kind in ("attention", "block"):
        z = LAYERS[case["shape"]]
        nq, nkv, D = z["heads"], z["kv_heads"], z["dim"]
        f = _frequencies(D, 500000.0, dict(ROPE, factor=z["factor"]))
        out = []
        for (at, s, n), rows in zip(_spans(reqs), given["rows"]):
            h, pos = x[at], _positions(s, n)
            q = _rotate((h @ w["q"].T).view(n, nq, D), pos, f)
            k, v = _rotate((h @ w["k"].T).view(n, nkv, D), pos, f), (h @ w["v"].T).view(n, nkv, D)
            if rows is not None:
                k, v = torch.cat([rows[0].double(), k]), torch.cat([rows[1].double(), v])
            out.append(_attend(q, k, v, s, D ** -0.5).flatten(1))
        return torch.cat(out) @ w["o"].T
    W = int(case["width"])
    heads = W // 64
    out = []
    if kind == "latent":
        z = _latent_sizes(W)
        H, D, r, V, kr = (z[k] for k in ("heads", "dim", "rot", "vdim", "rank"))
        f = _frequencies(r, 10000.0)
        for (at, s, n), rows in zip(_spans(reqs), given["rows"]):
            h, pos = x[at], _positions(s, n)
            q = (_rms(h @ w["dq"].T, w["dq_norm"]) @ w["uq"].T).view(n, H, D + r)
            q = torch.cat([q[..., :D], _rotate(q[..., D:], pos, f, True)], -1)
            kv = h @ w["dkv"].T
            c, kr_ = _rms(kv[:, :kr], w["dkv_norm"]), _rotate(kv[:, None, kr:], pos, f, True)[:, 0]
            if rows is not None:
                c, kr_ = torch.cat([rows[:, 0, :kr].double(), c]), torch.cat([rows[:, 0, kr:].double(), kr_])
            k = torch.cat([(c @ w["uk"].T).view(-1, H, D), kr_[:, None].expand(-1, H, -1)], -1)
            out.append(_attend(q, k, (c @ w["uv"].T).view(-1, H, V), s, (D + r) ** -0.5, w["sink"]).flatten(1))
        return torch.cat(out) @ w["o"].T
    if kind == "chunk_attention":
        G, f = heads // 4, _frequencies(64, 10000.0)
        for (at, s, n), rows in zip(_spans(reqs), given["rows"]):
            h, pos = x[at], _positions(s, n)
            q = _rms(h @ w["q"].T + w["q_bias"], w["q_norm"]).view(n, heads, 64)
            k = _rms(h @ w["k"].T + w["k_bias"], w["k_norm"]).view(n, G, 64)
            q, k, v = _rotate(q, pos, f), _rotate(k, pos, f), (h @ w["v"].T + w["v_bias"]).view(n, G, 64)
            if rows is not None:
                k, v = torch.cat([rows[..., :64].double(), k]), torch.cat([rows[..., 64:].double(), v])
            out.append(_attend(q, k, v, s, 0.125, w["sink"], 1024).flatten(1))
        return torch.cat(out) @ w["o"].T + w["o_bias"]
    if kind == "experts":
        E, S = 32, W

        def expert(v, gate, up, down):
            g, u = (v @ w[gate].T).clamp(max=7.0), (v @ w[up].T).clamp(-7.0, 7.0)
            return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[down].T

        score, chosen = torch.sigmoid(x @ w["router"].T).topk(4, dim=-1)
        y = expert(x, "shared_gate", "shared_up", "shared_down") * torch.sigmoid(x @ w["shared_sg"].T)
        for e in range(E):
            t, k = (chosen == e).nonzero(as_tuple=True)
            if len(t):
                y[t] += expert(x[t] * score[t, k][:, None], "gate%d" % e, "up%d" % e, "down%d" % e)
        return y
    for at, s, n in _spans(reqs):
        h = x[at]
        if kind == "delta":
            G = heads // 4
            q, k, v = (F.silu(_conv(h @ w[m].T, w[m + "_conv"])) for m in ("q", "k", "v"))
            q, k = (m.view(n, G, 64).repeat_interleave(4, 1) for m in (q, k))
            q, k = (m / torch.sqrt(m.square().sum(-1, keepdim=True) + 1e-6) for m in (q, k))
            q, v, beta = q * 0.125, v.view(n, heads, 64), torch.sigmoid(h @ w["b"].T)
            g = torch.exp(-w["A_log"].exp() * F.softplus(h @ w["a"].T + w["dt_bias"]))
            S, o = x.new_zeros((heads, 64, 64)), x.new_empty((n, heads, 64))
            for t in range(n):
                S = S * g[t, :, None, None]
                u = beta[t, :, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
                S = S + k[t, :, :, None] * u[:, None, :]
                o[t] = torch.einsum("hkv,hk->hv", S, q[t])
            o = _rms(o, w["norm"]) * F.silu(h @ w["g"].T).view(n, heads, 64)
        elif kind == "mlstm":
            q, k, v = ((h @ w[m].T).view(n, heads, 64) for m in ("q", "k", "v"))
            gi = 15.0 * torch.tanh((h @ w["i"].T + w["i_bias"]) / 15.0)
            gf = F.logsigmoid(15.0 * torch.tanh((h @ w["f"].T + w["f_bias"]) / 15.0))
            C, N, m, o = x.new_zeros((heads, 64, 64)), x.new_zeros((heads, 64)), x.new_zeros(heads), x.new_empty((n, heads, 64))
            for t in range(n):
                top = torch.maximum(gf[t] + m, gi[t])
                keep, take = torch.exp(gf[t] + m - top)[:, None], torch.exp(gi[t] - top)[:, None]
                C = C * keep[..., None] + (take * k[t])[:, :, None] * v[t][:, None, :]
                N, m = N * keep + take * k[t], top
                below = torch.maximum((N * q[t]).sum(-1).abs() * 0.125, torch.exp(-m)) + 1e-6
                o[t] = torch.einsum("hkv,hk->hv", C, q[t]) * 0.125 / below[:, None]
            o = (_rms(o).flatten(1) * w["norm"] * torch.sigmoid(h @ w["g"].T))
        else:
            inner, N, G = 2 * W, 128, 8
            hs = inner // 64
            p = h @ w["in"].T
            zz, xbc, dt = p.split([inner, inner + 2 * G * N, hs], -1)
            xbc = F.silu(_conv(xbc, w["conv"], w["conv_bias"]))
            u, B, C = xbc.split([inner, G * N, G * N], -1)
            u, B, C = u.reshape(n, hs, 64), *(m.reshape(n, G, N).repeat_interleave(hs // G, 1) for m in (B, C))
            dt = F.softplus(dt + w["dt_bias"])
            keep = torch.exp(-w["A_log"].exp() * dt)
            S, o = x.new_zeros((hs, N, 64)), x.new_empty((n, hs, 64))
            for t in range(n):
                S = S * keep[t, :, None, None] + (dt[t, :, None] * B[t])[:, :, None] * u[t][:, None, :]
                o[t] = torch.einsum("hkv,hk->hv", S, C[t])
            o = (o + w["D"][:, None] * u).flatten(1) * F.silu(zz)
            o = _rms(o.view(n, 8, -1)).flatten(1) * w["norm"]
        out.append(o.flatten(1))
    return torch.cat(out) @ w["o"].T


def _exact_step(case, seed):
    """Logits of each request's last token, its whole sequence run in 64 bits through the same random model."""
    tokens = _step_tokens(case, seed)
    shapes = {"model.embed_tokens.weight": (STEP_VOCAB, 2048), "model.norm.weight": (2048,)}
    for i in range(STEP_LAYERS):
        p = "model.layers.%d." % i
        shapes.update({p + "self_attn.q_proj.weight": (2048, 2048), p + "self_attn.k_proj.weight": (512, 2048),
                       p + "self_attn.v_proj.weight": (512, 2048), p + "self_attn.o_proj.weight": (2048, 2048),
                       p + "mlp.gate_proj.weight": (8192, 2048), p + "mlp.up_proj.weight": (8192, 2048),
                       p + "mlp.down_proj.weight": (2048, 8192), p + "input_layernorm.weight": (2048,),
                       p + "post_attention_layernorm.weight": (2048,)})
    d, w = _Draws(seed), {}
    for name in sorted(shapes):     # random weights are drawn in the order of the tensors' names
        w[name] = d.normal(shapes[name], STD) + 1.0 if len(shapes[name]) == 1 else d.normal(shapes[name], STD, dtype=torch.bfloat16)
    lens = [len(t) for t in tokens]
    x = w["model.embed_tokens.weight"][torch.as_tensor(sum(tokens, []), device="cuda")].double()
    f = _frequencies(64, 500000.0, dict(ROPE, factor=32.0))
    spans = list(_spans([(0, n) for n in lens]))
    for i in range(STEP_LAYERS):
        p = "model.layers.%d." % i
        m = {k: w[p + k + ".weight"].double() for k in ("self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj",
                                                        "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj", "input_layernorm",
                                                        "post_attention_layernorm")}
        h = _rms(x, m["input_layernorm"], 1e-5)
        q, k, v = (h @ m["self_attn.%s_proj" % n].T for n in ("q", "k", "v"))
        a = torch.empty_like(q)
        for at, _, n in spans:
            pos = _positions(0, n)
            a[at] = _attend(_rotate(q[at].view(n, 32, 64), pos, f), _rotate(k[at].view(n, 8, 64), pos, f), v[at].view(n, 8, 64),
                            0, 0.125).flatten(1)
        x = x + a @ m["self_attn.o_proj"].T
        h = _rms(x, m["post_attention_layernorm"], 1e-5)
        x = x + (torch.nn.functional.silu(h @ m["mlp.gate_proj"].T) * (h @ m["mlp.up_proj"].T)) @ m["mlp.down_proj"].T
    last = torch.as_tensor(np.cumsum(lens) - 1, device="cuda")
    return _rms(x[last], w["model.norm.weight"].double(), 1e-5) @ w["model.embed_tokens.weight"].double().T


def exact(case, seed):
    if case["kind"] == "step":
        return _exact_step(case, seed)
    w, given = _inputs(case, seed)
    w = {k: v.double() for k, v in w.items()}
    if case["kind"] == "block":
        x = given["x"].double()
        x = x + _exact_part(case, w, dict(given, x=_rms(x, w["norm1"])))
        h = _rms(x, w["norm2"])
        x = x + (torch.nn.functional.silu(h @ w["gate"].T) * (h @ w["up"].T)) @ w["down"].T
        return {"y": _rms(x, w["norm3"]), "residual": x, "k": None, "v": None}
    y = _exact_part(case, w, given)
    if case["kind"] == "attention":
        return {"y": y, "k": None, "v": None}
    if case["kind"] in ("latent", "chunk_attention"):
        return {"y": y, "rows": None}
    return {"y": y} if case["kind"] == "experts" else {"y": y, "state": None}
