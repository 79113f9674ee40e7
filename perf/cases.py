"""The work that users of this engine have it do, as cases that can be timed and checked.

Whole steps go through ``ModelRunner.step`` (CUDA graphs on, as the engine runs them) on models with the layer sizes of
``servelab_b200.bench`` cut to a few layers and a vocabulary of 32,000: decode at batch 1, 8 and 64 and a mixed step of
a prompt portion and single tokens.  Single layers go through the parts' ``forward`` on a packed step: prompts, because
that is where a layer is more than a few launches.  Weights are random at the checkpoint's usual spread, earlier tokens'
keys, values and states are random at the spread that such weights produce.
"""

from __future__ import annotations

import math
import random

import torch

from servelab_b200.bench import arch_compare as shapes
from servelab_b200.bench import workloads
from servelab_b200.cache.manager import paged_part, state_part
from servelab_b200.config import CacheConfig, config_from_dict
from servelab_b200.engine.batch import BatchEntry, StepContext
from servelab_b200.engine.runner import ModelRunner
from servelab_b200.models.causal_lm import declare_tensors
from servelab_b200.ops import kernels as K
from servelab_b200.parts import FEED_FORWARDS, MIXERS, BuildEnv, LayerCache, build_part, part_class
from servelab_b200.weights import RandomSource, WeightStore

DEV = "cuda:0"
F64 = torch.float64
PAGE = 16
VOCAB = 32000
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


# ---------------------------------------------------------------------------- cases
def listed():
    return [
        # one user's chat: a single decoded token of the smallest shape; launches and latency count
        {"name": "decode_1_small", "kind": "qwen_step", "shape": "qwen2.5-0.5b", "layers": 8, "decodes": 1, "past": 300,
         "chunk": 0, "chunk_past": 0},
        # a server's decode step at the benchmark's batch and context
        {"name": "decode_8_7b", "kind": "qwen_step", "shape": "qwen2.5-7b", "layers": 4, "decodes": 8, "past": 2048,
         "chunk": 0, "chunk_past": 0},
        # continuous batching: a portion of a prompt beside the decoded tokens of the other requests
        {"name": "portion_and_decodes_small", "kind": "qwen_step", "shape": "qwen2.5-0.5b", "layers": 8, "decodes": 31,
         "past": 700, "chunk": 449, "chunk_past": 512},
        # many users of a model with a state beside its attention
        {"name": "sunutar_decode_64", "kind": "sunutar_step", "size": "1b-like", "layers": 2, "decodes": 64, "past": 1536},
        # an attention layer over a prompt of the benchmark's length
        {"name": "attention_prompt_7b", "kind": "attention", "shape": "qwen2.5-7b", "dtype": "bf16", "lens": "2048",
         "past": 0},
        # the exact path that logits are checked with
        {"name": "feed_forward_fp32", "kind": "feed_forward", "shape": "qwen2.5-0.5b", "dtype": "fp32", "tokens": 257},
        # routed experts, a prompt and a decode step of many users
        {"name": "experts_prompt", "kind": "experts", "size": "lite-2048", "tokens": 2048},
        {"name": "experts_decode_64", "kind": "experts", "size": "lite-2048", "tokens": 64},
        # prompts of several lengths through a latent attention
        {"name": "latent_prompts", "kind": "latent", "size": "lite-2048", "lens": "1531,40,511"},
        # a convolved, windowed attention beside a linear attention with learned decays
        {"name": "gated_linear_prompt", "kind": "sumolorn", "size": "1b-like", "lens": "2048"},
        # an attention beside a state space, prompts of several lengths
        {"name": "state_space_prompts", "kind": "sunutar", "size": "1b-like", "lens": "1021,514,77,1300"},
        # a delta rule over a prompt
        {"name": "delta_rule_prompt", "kind": "delta", "size": "1b-like", "lens": "2048"},
    ]


def _between(rng, lo, hi):
    """A whole number, spread evenly over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lens(rng, total, most=5):
    n = rng.randint(1, most)
    cuts = sorted(rng.random() for _ in range(n - 1))
    parts = [max(1, int(total * (b - a))) for a, b in zip([0.0] + cuts, cuts + [1.0])]
    return ",".join(str(p) for p in parts)


def draw(rng):
    kind = rng.choice(["qwen_step", "qwen_step", "sunutar_step", "attention", "feed_forward", "experts", "latent",
                       "sumolorn", "sunutar", "delta"])
    big = rng.random() < 0.5
    if kind == "qwen_step":
        shape = "qwen2.5-7b" if big else "qwen2.5-0.5b"
        portion = rng.random() < 0.4
        return {"kind": kind, "shape": shape, "layers": rng.randint(1, 2) if big else rng.randint(2, 8),
                "decodes": rng.randint(0, 40) if portion else _between(rng, 1, 64), "past": _between(rng, 16, 2300),
                "chunk": _between(rng, 16, 900) if portion else 0, "chunk_past": rng.choice([0, rng.randint(1, 1500)])
                if portion else 0}
    if kind == "sunutar_step":
        return {"kind": kind, "size": "1b-like" if big else "small-1024", "layers": rng.randint(1, 2),
                "decodes": _between(rng, 1, 64), "past": _between(rng, 16, 2300)}
    if kind == "attention":
        exact32 = rng.random() < 0.25
        return {"kind": kind, "shape": "qwen2.5-7b" if big and not exact32 else "qwen2.5-0.5b",
                "dtype": "fp32" if exact32 else "bf16",
                "lens": _lens(rng, _between(rng, 20, 200 if exact32 else 2500)), "past": rng.choice([0, rng.randint(1, 900)])}
    if kind == "feed_forward":
        exact32 = rng.random() < 0.6
        return {"kind": kind, "shape": "qwen2.5-0.5b" if exact32 or not big else "qwen2.5-7b",
                "dtype": "fp32" if exact32 else "bf16", "tokens": _between(rng, 1, 500 if exact32 else 2500)}
    if kind == "experts":
        return {"kind": kind, "size": "lite-2048" if big else "small-1024", "tokens": _between(rng, 1, 2500)}
    if kind == "latent":
        return {"kind": kind, "size": "lite-2048", "lens": _lens(rng, _between(rng, 20, 2500))}
    return {"kind": kind, "size": "1b-like" if big else "small-1024", "lens": _lens(rng, _between(rng, 20, 2900))}


# ------------------------------------------------------------- models, layers, weights
SUNUTAR = {  # (a head's values are half its keys: a pair of sizes that the package builds ahead)
    "1b-like": (2048, 16, 4, 128, 64, 5632, 32, 64, 128, 4),
    "small-1024": (1024, 8, 2, 96, 64, 2816, 16, 64, 64, 2),
}


def _sunutar(size, layers):
    width, heads, kv, dim, vdim, ff, rh, rp, rn, rg = SUNUTAR[size]
    cfg = shapes.sunutar_config(width, heads, kv, dim, ff, rh, rp, rn, rg, 0, 0, layers)
    for layer in cfg["layers"]:
        layer["mixer"]["left"]["vdim"] = vdim
    return cfg


def _config(case):
    kind = case["kind"]
    if kind in ("qwen_step", "attention", "feed_forward"):
        return dict(workloads.SHAPES[case["shape"]], num_hidden_layers=case.get("layers", 1), vocab_size=VOCAB)
    if kind in ("sunutar_step", "sunutar"):
        return _sunutar(case["size"], case.get("layers", 1))
    if kind in ("experts", "latent"):
        return shapes.daferax_config(*shapes.DAFERAX_SIZES[case["size"]], layers=1)
    if kind == "sumolorn":
        return shapes.sumolorn_config(*shapes.SUMOLORN_SIZES[case["size"]], layers=2)
    return shapes.vufadra_config(*shapes.VUFADRA_SIZES[case["size"]], layers=2)


class _Weights(RandomSource):
    """Random tensors with the spread that trained ones have where a plain normal would be another regime: a state
    space's step sizes and rates, a delta rule's decays, a convolution's taps."""

    def __init__(self, decls, seed, dtype):
        super().__init__(decls, seed, std=0.02, device=DEV, dtype=dtype, std_of={"conv": 0.3})

    def read(self, name):
        t = super().read(name)
        last = name.rsplit(".", 1)[-1]
        if last in ("dt_bias", "A_log", "w0"):
            u = torch.special.ndtr(t.float() / self.std)                        # uniform in (0, 1)
            if last == "dt_bias":                                               # softplus(.) from 1e-3 to 1e-1
                dt = torch.exp(math.log(1e-3) + u * math.log(100.0))
                t = (dt + torch.log(-torch.expm1(-dt))).to(t.dtype)
            elif last == "A_log":
                t = torch.log(1.0 + 15.0 * u).to(t.dtype)
            else:
                t = (7.0 * u - 6.0).to(t.dtype)
        return t


def _seed(case, seed):
    return (seed * 1000003 + 17) % (1 << 40)


def _randn(gen, shape, std, dtype):
    return (torch.randn(shape, generator=gen, device=DEV) * std).to(dtype)


def _whole(lens):
    return [int(n) for n in str(lens).split(",")]


def _tables(rng, needs):
    """Pages of the requests, scattered over the pool as a running server leaves them."""
    pages = list(range(sum(needs)))
    rng.shuffle(pages)
    out = []
    for n in needs:
        out.append(pages[:n])
        pages = pages[n:]
    return out


# ------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    return _prepare_step(case, seed) if case["kind"].endswith("_step") else _prepare_layer(case, seed)


def _prepare_step(case, seed):
    cfg = config_from_dict(_config(case))
    spec = cfg.to_model_spec()
    src = _Weights(declare_tensors(spec), _seed(case, seed), torch.bfloat16)
    rng = random.Random(seed)
    # every request of a step has its own length, around the case's
    work = [(max(0, case["past"] - rng.randint(0, case["past"] // 8)), 1) for _ in range(case["decodes"])]
    if case.get("chunk"):
        work.append((case["chunk_past"], case["chunk"]))
    longest = max(p + n for p, n in work)
    pages = sum(-(-(p + n) // PAGE) + 1 for p, n in work) + 4
    runner = ModelRunner(cfg, src, "bfloat16", CacheConfig(block_size=PAGE, num_blocks=pages), max_num_seqs=len(work),
                         device=DEV, cuda_graphs=True, max_model_len=-(-(longest + 1) // 256) * 256)
    ids = []
    for i, (past, n) in enumerate(work):
        rid = f"r{i}"
        if not runner.cache.open(rid) or not runner.cache.ensure(rid, past + n):
            raise RuntimeError("the pool does not hold the case's requests")
        ids.append([rng.randrange(VOCAB) for _ in range(n)])
    state = {"runner": runner, "source": src, "work": work, "ids": ids, "config": _config(case)}
    for _ in range(3):                                    # a server's graphs are there before the step comes
        run(state)
    gen = torch.Generator(device=DEV).manual_seed(_seed(case, seed))
    for cache in runner.storage.layer_caches.values():
        for t in (cache.k, cache.v):
            if t is not None:
                t.copy_(_randn(gen, t.shape, 1.0, t.dtype))
        if cache.state is not None:
            cache.state.copy_(_randn(gen, cache.state.shape, 0.5, cache.state.dtype))
    return state


def _layer_spec(case):
    """(registry, the layer's part as the model's configuration describes it)"""
    layers = config_from_dict(_config(case)).to_model_spec().layers
    if case["kind"] in ("feed_forward", "experts"):
        return FEED_FORWARDS, layers[0].feed_forward
    return MIXERS, layers[1 if case["kind"] in ("sumolorn", "delta") else 0].mixer


def _prepare_layer(case, seed):
    table, spec = _layer_spec(case)
    dtype = DTYPES[case.get("dtype", "bf16")]
    decls = part_class(table, spec).declare(spec, "m")
    src = _Weights(decls, _seed(case, seed), dtype)
    part = build_part(table, spec, "m", BuildEnv(device=DEV, dtype=dtype, page_size=PAGE))
    part.load(WeightStore(src, decls, dtype, DEV))
    gen = torch.Generator(device=DEV).manual_seed(_seed(case, seed))
    lens = _whole(case["lens"]) if "lens" in case else [case["tokens"]]
    past = case.get("past", 0)
    x = _randn(gen, (sum(lens), spec.hidden_size), 1.0, dtype)         # (what a norm hands over)
    state = {"part": part, "source": src, "x": x, "ctx": None, "cache": None, "lens": lens, "past": past, "spec": spec}
    if table is FEED_FORWARDS:
        return state
    tables = _tables(random.Random(seed), [-(-(past + n) // PAGE) for n in lens])
    state["tables"] = tables
    state["ctx"] = StepContext.pack([BatchEntry(tokens=[0] * n, start=past, want=(), block_tables=[t], state_slot=i)
                                     for i, (n, t) in enumerate(zip(lens, tables))], 1, DEV)
    request = part_class(MIXERS, spec).cache_request(spec)
    cache = state["cache"] = LayerCache(group=0, page_size=PAGE)
    paged, fixed = paged_part(request), state_part(request)
    if paged is not None:
        n = sum(len(t) for t in tables)
        cache.k = _randn(gen, (n, paged.num_kv_heads, PAGE, paged.head_dim), 1.0, dtype)
        cache.v = cache.k if paged.tied_values else _randn(
            gen, (n, paged.num_kv_heads, PAGE, paged.value_dim or paged.head_dim), 1.0, dtype)
    if fixed is not None:
        cache.state = torch.zeros((len(lens), *fixed.shape), device=DEV)
    return state


@torch.no_grad()
def run(state):
    if "runner" in state:
        runner = state["runner"]
        entries = [runner.entry(f"r{i}", ids, past, (n - 1,))
                   for i, ((past, n), ids) in enumerate(zip(state["work"], state["ids"]))]
        logits = runner.step(entries)
        records = [c.state for c in runner.storage.layer_caches.values() if c.state is not None]
        return {"logits": logits, "records": records} if records else logits
    part, cache = state["part"], state["cache"]
    if cache is None:
        return K.plain_unless(None, part.forward(state["ctx"], state["x"]))
    if cache.state is not None:
        cache.state.zero_()                               # new requests begin with empty records
    out = {"y": K.plain_unless(None, part.forward(state["ctx"], state["x"], cache, True))}
    if cache.state is not None:
        out["state"] = cache.state
    return out


# ------------------------------------------------------------------------------ work
def _attention_pairs(past, n, window):
    return sum(min(past + i + 1, window or (1 << 60)) for i in range(n))


def work(case):
    kind, cfg = case["kind"], _config(case)
    if kind == "qwen_step":
        h, H, G, D, ff, L = (cfg[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim",
                                              "intermediate_size", "num_hidden_layers"))
        per = (H + 2 * G) * D * h + H * D * h + 3 * h * ff
        reqs = [(case["past"], 1)] * case["decodes"] + ([(case["chunk_past"], case["chunk"])] if case["chunk"] else [])
        tokens, keys = sum(n for _, n in reqs), sum(p + n for p, n in reqs)
        pairs = sum(_attention_pairs(p, n, None) for p, n in reqs)
        return {"bytes": 2.0 * (L * per + VOCAB * h) + L * keys * 2 * G * D * 2.0 + len(reqs) * VOCAB * 4.0,
                "flops": 2.0 * tokens * L * per + 4.0 * L * pairs * H * D + 2.0 * len(reqs) * VOCAB * h}
    if kind == "sunutar_step":
        w, H, G, D, Dv, ff, rh, rp, rn, rg = SUNUTAR[case["size"]]
        L, B = case["layers"], case["decodes"]
        inner, ch = rh * rp, rh * rp + 2 * rg * rn
        per = w * (H * D + G * D + G * Dv + H * Dv + 2 * inner + ch + rh + 3 * ff)
        keys = min(case["past"] + 1, shapes.WINDOW)
        return {"bytes": 2.0 * (L * per + VOCAB * w) + L * B * (keys * G * (D + Dv) * 2.0 + 2 * 4.0 * (rh * rp * rn + 3 * ch))
                + B * VOCAB * 4.0,
                "flops": 2.0 * B * (L * per + VOCAB * w) + L * B * (2.0 * keys * H * (D + Dv) + 4.0 * rh * rp * rn)}
    lens = _whole(case["lens"]) if "lens" in case else [case["tokens"]]
    T = sum(lens)
    if kind == "feed_forward":
        el = 4.0 if case["dtype"] == "fp32" else 2.0
        h, ff = cfg["hidden_size"], cfg["intermediate_size"]
        # (32-bit products run on the CUDA cores)
        return {"bytes": el * (3 * h * ff + 2 * T * h), "flops": 6.0 * T * h * ff}
    if kind == "attention":
        el = 4.0 if case["dtype"] == "fp32" else 2.0
        h, H, G, D = (cfg[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim"))
        per = (H + 2 * G) * D * h + H * D * h
        pairs = sum(_attention_pairs(case["past"], n, None) for n in lens)
        keys = sum(n + case["past"] for n in lens)
        return {"bytes": el * (per + 2 * T * h + keys * 2 * G * D), "flops": 2.0 * T * per + 4.0 * pairs * H * D}
    if kind == "experts":
        w, _, _, _, _, _, experts, _, _, top, eff, sff = shapes.DAFERAX_SIZES[case["size"]]
        used = min(experts, T * top)
        return {"bytes": 2.0 * (3 * w * (used * eff + sff) + 2 * T * w) + 4.0 * experts * w,
                "flops": 6.0 * T * w * (top * eff + sff) + 2.0 * T * w * experts}
    if kind == "latent":
        w, H, _, D, R, Dr = shapes.DAFERAX_SIZES[case["size"]][:6]
        per = w * (H * (D + Dr) + R + Dr + H * D) + 2 * H * D * R + H * D * w
        pairs = sum(_attention_pairs(0, n, shapes.WINDOW) for n in lens)
        return {"bytes": 2.0 * (per + 2 * T * w + T * (R + Dr)),
                "flops": 2.0 * T * per + 2.0 * pairs * H * (D + Dr + D)}
    if kind == "sumolorn":
        w, H, G, D, _, _, _, _, lh, ld, lv = shapes.SUMOLORN_SIZES[case["size"]]
        per = w * (H * D + 2 * G * D + H * D) + w * (2 * lh * ld + 2 * lh * lv + 32 + lh * lv) + 32 * lh * ld
        pairs = sum(_attention_pairs(0, n, shapes.WINDOW) for n in lens)
        return {"bytes": 2.0 * (per + 2 * T * w + T * 2 * G * D) + 4.0 * len(lens) * lh * ld * lv,
                "flops": 2.0 * T * per + 4.0 * pairs * H * D + 4.0 * T * lh * ld * lv}
    if kind == "sunutar":
        w, H, G, D, Dv, ff, rh, rp, rn, rg = SUNUTAR[case["size"]]
        inner, ch = rh * rp, rh * rp + 2 * rg * rn
        per = w * (H * D + G * D + G * Dv + H * Dv + 2 * inner + ch + rh)
        pairs = sum(_attention_pairs(0, n, shapes.WINDOW) for n in lens)
        return {"bytes": 2.0 * (per + 2 * T * w + T * G * (D + Dv)) + 4.0 * len(lens) * (rh * rp * rn + 3 * ch),
                "flops": 2.0 * T * per + 2.0 * pairs * H * (D + Dv) + 4.0 * T * rh * rp * rn}
    w, _, _, D, _, rh, rank = shapes.VUFADRA_SIZES[case["size"]]
    per = w * (6 * rh * D + rank) + rank * rh * D
    return {"bytes": 2.0 * (per + 2 * T * w) + 4.0 * len(lens) * rh * D * D,
            "flops": 2.0 * T * per + 8.0 * T * rh * D * D}


def tolerance(case):
    # float32: sums of up to 4,864 products in another order.  bfloat16: rounding of every intermediate row; steps
    # carry it through all their layers
    if case.get("dtype") == "fp32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.03 if case["kind"].endswith("_step") else 0.02, "max": 0.5}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    state = prepare(case, seed)
    src = state["source"]

    def w(name):
        return src.read(name).to(F64)
    if case["kind"] == "qwen_step":
        return _exact_qwen_step(state, w)
    if case["kind"] == "sunutar_step":
        return _exact_sunutar_step(state, w)
    x, lens = state["x"].to(F64), state["lens"]
    if case["kind"] == "feed_forward":
        return _gated(x, w, "m.", "_proj.weight")
    cfg = _config(case)
    if case["kind"] == "experts":
        return _exact_experts(x, w, cfg["layers"][0]["mlp"])
    eps = cfg["rms_norm_eps"] if "rms_norm_eps" in cfg else cfg["norm"]["eps"]
    ys, records, at = [], [], 0
    for i, n in enumerate(lens):
        h = x[at:at + n]
        at += n
        record = None
        if case["kind"] == "attention":
            y = _exact_attention(h, w, cfg, "m.", state["past"], *_cached(state["cache"], state["tables"][i], state["past"]))
        elif case["kind"] == "latent":
            y = _exact_latent(h, w, cfg["layers"][0]["mixer"], eps)
        elif case["kind"] == "sumolorn":
            y, record = _exact_sumolorn(h, w, cfg["layers"][1]["mixer"], eps)
        elif case["kind"] == "sunutar":
            y, record = _exact_sunutar(h, w, "m", cfg["layers"][0]["mixer"], eps)
        else:
            y, record = _exact_delta(h, w, cfg["layers"][1]["mixer"], eps)
        ys.append(y)
        records.append(record)
    out = {"y": torch.cat(ys)}
    if records[0] is not None:
        out["state"] = torch.stack(records).reshape(state["cache"].state.shape)
    return out


def _cached(cache, table, past):
    """Keys and values [past, kv heads, size] of a request's earlier tokens."""
    out = []
    for t in (cache.k, cache.v):
        rows = t[torch.tensor(table, dtype=torch.long, device=DEV)].permute(0, 2, 1, 3)
        out.append(rows.reshape(-1, *rows.shape[2:])[:past].to(F64))
    return out


def _rms(x, w, eps):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _silu(z):
    return z * torch.sigmoid(z)


def _gated(x, w, pre, suffix=""):
    return (_silu(x @ w(pre + "gate" + suffix).T) * (x @ w(pre + "up" + suffix).T)) @ w(pre + "down" + suffix).T


def _clamped(x, w, pre, limit):
    g = (x @ w(pre + "gate").T).clamp(max=limit)
    u = (x @ w(pre + "up").T).clamp(-limit, limit)
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(pre + "down").T


def _turn(x, pos, freq, halves, mag=1.0):
    """The first 2 * len(freq) elements of every head of x [T, heads, D] turned by position times frequency: element i
    with element i + len(freq), or neighbours."""
    n = len(freq)
    a = pos.to(F64)[:, None, None] * freq
    c, s = torch.cos(a) * mag, torch.sin(a) * mag
    first, second = (slice(0, n), slice(n, 2 * n)) if halves else (slice(0, 2 * n, 2), slice(1, 2 * n, 2))
    u, v, out = x[..., first], x[..., second], x.clone()
    out[..., first], out[..., second] = u * c - v * s, v * c + u * s
    return out


def _freq(dims, base):
    return base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device=DEV) / dims)


def _softmax_attention(q, k, v, scale, past=0, window=None, cap=None, slopes=None, one=False):
    """q [n, H, D] of the tokens from ``past`` on, k, v [past + n, G, .]; ``one``: exp(0) in the denominator."""
    n, H, _ = q.shape
    rep = H // k.shape[1]
    d = torch.arange(past, past + n, device=DEV)[:, None] - torch.arange(past + n, device=DEV)[None, :]
    hidden = (d < 0) if not window else (d < 0) | (d >= window)
    out = []
    for h in range(H):
        s = q[:, h] @ k[:, h // rep].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[h] * d
        s = s.masked_fill(hidden, -math.inf)
        if one:
            s = torch.cat([s, torch.zeros_like(s[:, :1])], -1)
        out.append(torch.softmax(s, -1)[:, :past + n] @ v[:, h // rep])
    return torch.stack(out, 1)


def _exact_attention(x, w, cfg, pre, past, k_past, v_past):
    H, G, D = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    n = x.shape[0]
    q, k, v = (x @ w(f"{pre}{c}_proj.weight").T + w(f"{pre}{c}_proj.bias") for c in "qkv")
    pos, freq = torch.arange(past, past + n, device=DEV), _freq(D, cfg["rope_theta"])
    q, k = _turn(q.view(n, H, D), pos, freq, True), _turn(k.view(n, G, D), pos, freq, True)
    o = _softmax_attention(q, torch.cat([k_past, k]), torch.cat([v_past, v.view(n, G, D)]), D ** -0.5, past)
    return o.reshape(n, H * D) @ w(pre + "o_proj.weight").T


def _requests(state):
    at = 0
    for i, (past, n) in enumerate(state["work"]):
        yield i, past, slice(at, at + n)
        at += n


def _exact_qwen_step(state, w):
    cfg, runner = state["config"], state["runner"]
    eps = cfg["rms_norm_eps"]
    embed = w("model.embed_tokens.weight")
    x = embed[torch.tensor(sum(state["ids"], []), device=DEV)]
    for i in range(cfg["num_hidden_layers"]):
        pre = f"model.layers.{i}."
        h = _rms(x, w(pre + "input_layernorm.weight"), eps)
        ys = []
        for r, past, rows in _requests(state):
            old = _cached(runner.storage.layer_caches[i], runner.cache.block_table(f"r{r}", 0), past)
            ys.append(_exact_attention(h[rows], w, cfg, pre + "self_attn.", past, *old))
        x = x + torch.cat(ys)
        x = x + _gated(_rms(x, w(pre + "post_attention_layernorm.weight"), eps), w, pre + "mlp.", "_proj.weight")
    last = torch.tensor([rows.stop - 1 for _, _, rows in _requests(state)], device=DEV)
    x = _rms(x[last], w("model.norm.weight"), eps)
    return x @ (embed if cfg["tie_word_embeddings"] else w("lm_head.weight")).T


def _exact_experts(x, w, mlp):
    r = mlp["router"]
    s = torch.softmax(x @ w("m.router").T, -1)
    n, keep, E = r["groups"]["count"], r["groups"]["keep"], r["experts"]
    best = s.view(-1, n, E // n).amax(-1).topk(keep, -1).indices
    kept = torch.zeros(s.shape[0], n, dtype=torch.bool, device=DEV).scatter_(1, best, True)
    top = s.masked_fill(~kept.repeat_interleave(E // n, 1), -1.0).topk(r["top"], -1).indices
    gate = torch.zeros_like(s).scatter_(1, top, s.gather(1, top) * r["scale"])
    out = _gated(x, w, "m.shared.")
    for e in range(E):
        rows = gate[:, e].nonzero().flatten()
        if len(rows):
            out[rows] += gate[rows, e, None] * _gated(x[rows], w, f"m.e{e}.")
    return out


def _stretched(dims, base, scaling):
    """Frequencies and the factor on sine and cosine of a rotation stretched between two numbers of turns."""
    f = _freq(dims, base)

    def at(turns):
        return dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    lo, hi = max(math.floor(at(scaling["fast"])), 0), min(math.ceil(at(scaling["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64, device=DEV) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / scaling["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0


def _exact_latent(h, w, m, eps):
    T, H, D, Dr, Dv, R = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    pos = torch.arange(T, device=DEV)
    f, mag = _stretched(Dr, m["rot"]["base"], m["rot"]["scaling"])
    q, down = (h @ w("m.q").T).view(T, H, D + Dr), h @ w("m.dkv").T
    c = _rms(down[:, :R], w("m.dkv.norm"), eps)
    kr = _turn(down[:, None, R:], pos, f, False, mag).expand(T, H, Dr)
    q = torch.cat([q[..., :D], _turn(q[..., D:], pos, f, False, mag)], -1)
    k = torch.cat([(c @ w("m.uk").T).view(T, H, D), kr], -1)
    o = _softmax_attention(q, k, (c @ w("m.uv").T).view(T, H, Dv), m["scale"], 0, m["mask"]["size"])
    return (o.reshape(T, H * Dv) * torch.sigmoid(h @ w("m.g").T)) @ w("m.o").T


def _convolved(u, taps, before=None, bias=None):
    """y_t = sum_j taps[:, j] u_{t - n + 1 + j}: (y, the last n - 1 rows)"""
    n = taps.shape[1]
    rows = torch.cat([torch.zeros((n - 1, u.shape[1]), dtype=F64, device=DEV) if before is None else before, u])
    y = sum(rows[j:j + u.shape[0]] * taps[:, j] for j in range(n))
    return (y if bias is None else y + bias), rows[u.shape[0]:]


def _exact_sumolorn(h, w, m, eps):
    T, a, b = h.shape[0], m["left"], m["right"]
    H, G, D, Dv = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
    u, taps = (torch.cat([f(c) for c in "qkv"], -1) for f in (lambda c: h @ w(f"m.left.{c}").T,
                                                              lambda c: w(f"m.left.{c}.conv").T))
    u, last = _convolved(u, taps.T)
    q, k, v = u.split([H * D, G * D, G * Dv], -1)
    pos, f = torch.arange(T, device=DEV), _freq(a["rot"]["dims"], a["rot"]["base"])
    q, k = (_rms(_turn(t.view(T, -1, D), pos, f, True), None, eps) for t in (q, k))
    o = _softmax_attention(q, k, v.reshape(T, G, Dv), a["scale"], 0, a["mask"]["size"])
    left = o.reshape(T, H * Dv) @ w("m.left.o").T
    H, D, Dv = b["heads"], b["dim"], b["vdim"]
    q, k, v, g = (h @ w(f"m.right.{c}").T for c in "qkvg")
    z = (h @ w("m.right.a1").T) @ w("m.right.a2").T + w("m.right.a2.b")
    decay = torch.exp(torch.nn.functional.logsigmoid(z) / b["tau"]).view(T, H, D)
    q, k, v = q.view(T, H, D) * D ** -0.5, k.view(T, H, D), v.view(T, H, Dv)
    S, out = torch.zeros((H, D, Dv), dtype=F64, device=DEV), []
    for t in range(T):
        S = decay[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
        out.append((S * q[t][:, :, None]).sum(1))
    o = _rms(torch.stack(out), w("m.right.norm"), eps).reshape(T, H * Dv)
    right = (o * _silu(g)) @ w("m.right.o").T
    y = 0.5 * (_rms(left, w("m.left.out"), eps) + _rms(right, w("m.right.out"), eps))
    return y, torch.cat([last.flatten(), S.flatten()])


def _exact_sunutar(h, w, pre, m, eps, past=0, k_past=None, v_past=None, record=None):
    """(y, the record after the tokens)"""
    T, a, b = h.shape[0], m["left"], m["right"]
    H, G, D, Dv = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
    q, k, v = (h @ w(f"{pre}.left.{c}").T + w(f"{pre}.left.{c}.b") for c in "qkv")
    q, k = (_rms(t, w(f"{pre}.left.{c}.norm"), eps).view(T, -1, D) for t, c in ((q, "q"), (k, "k")))
    v = v.view(T, G, Dv)
    keys, values = (k, v) if k_past is None else (torch.cat([k_past, k]), torch.cat([v_past, v]))
    slopes = [2.0 ** (-8.0 * (i + 1) / H) for i in range(H)]
    o = _softmax_attention(q, keys, values, a["scale"], past, a["mask"]["size"], a["softcap"], slopes, True)
    left = o.reshape(T, H * Dv) @ w(pre + ".left.o").T + w(pre + ".left.o.b")
    H, P, N, R = b["heads"], b["vdim"], b["state"], b["groups"]
    inner, C = H * P, H * P + 2 * R * N
    z, u, dt = (h @ w(pre + ".right.in").T).split([inner, C, H], -1)
    S, rows = torch.zeros((H, N, P), dtype=F64, device=DEV), None
    if record is not None:
        S, rows = record[:H * N * P].view(H, N, P), record[H * N * P:].view(-1, C)
    u, rows = _convolved(u, w(pre + ".right.conv"), rows, w(pre + ".right.conv.b"))
    x, B, O = _silu(u).split([inner, R * N, R * N], -1)
    x, B, O = x.reshape(T, H, P), *(t.reshape(T, R, N).repeat_interleave(H // R, 1) for t in (B, O))
    dt = torch.nn.functional.softplus(dt + w(pre + ".right.dt_bias"), threshold=1e9)
    keep, out = torch.exp(-torch.exp(w(pre + ".right.A_log")) * dt), []
    for t in range(T):
        S = keep[t][:, None, None] * S + (dt[t][:, None] * B[t])[:, :, None] * x[t][:, None, :]
        out.append((S * O[t][:, :, None]).sum(1))
    y = (torch.stack(out) + w(pre + ".right.D")[:, None] * x).reshape(T, inner) * _silu(z)
    groups = b["norm_groups"]
    y = _rms(y.view(T, groups, inner // groups), None, eps).reshape(T, inner) * w(pre + ".right.norm")
    right = y @ w(pre + ".right.o").T
    return m["left_scale"] * left + m["right_scale"] * right, torch.cat([S.flatten(), rows.flatten()])


def _exact_sunutar_step(state, w):
    cfg, runner = state["config"], state["runner"]
    eps, mult = cfg["norm"]["eps"], cfg["residual_mult"]
    embed = w("embed")
    x = embed[torch.tensor(sum(state["ids"], []), device=DEV)]
    records = []
    for i, layer in enumerate(cfg["layers"]):
        cache = runner.storage.layer_caches[i]
        after = cache.state.to(F64).clone()
        h, ys = _rms(x, w(f"l{i}.norm1"), eps), []
        for r, past, rows in _requests(state):
            slot = runner.cache.state_slot(f"r{r}")
            old = _cached(cache, runner.cache.block_table(f"r{r}", 0), past)
            y, after[slot] = _exact_sunutar(h[rows], w, f"l{i}.mix", layer["mixer"], eps, past, *old,
                                            after[slot].clone())
            ys.append(y)
        x = x + mult * _rms(torch.cat(ys), w(f"l{i}.norm1b"), eps)
        y = _clamped(_rms(x, w(f"l{i}.norm2"), eps), w, f"l{i}.mlp.", layer["mlp"]["limit"])
        x = x + mult * _rms(y, w(f"l{i}.norm2b"), eps)
        records.append(after)
    return {"logits": _rms(x, w("final.norm"), eps) @ embed.T, "records": records}


def _exact_delta(h, w, m, eps):
    T, H, D = h.shape[0], m["heads"], m["dim"]
    r, k, v = ((h @ w(f"m.{c}").T).view(T, H, D) for c in "rkv")
    z = torch.tanh(h @ w("m.w1").T) @ w("m.w2").T + w("m.w0")
    keep = torch.exp(-math.exp(-0.5) * torch.sigmoid(z)).view(T, H, D)
    a = torch.sigmoid(h @ w("m.a").T + w("m.a.b")).view(T, H, D)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    S, out = torch.zeros((H, D, D), dtype=F64, device=DEV), []
    for t in range(T):
        seen = (S * u[t][:, :, None]).sum(1)
        S = keep[t][:, :, None] * S - (a[t] * u[t])[:, :, None] * seen[:, None, :] + k[t][:, :, None] * v[t][:, None, :]
        out.append((S * r[t][:, :, None]).sum(1))
    o = _rms(torch.stack(out), None, eps).reshape(T, H * D) * w("m.norm") * torch.sigmoid(h @ w("m.g").T)
    return o @ w("m.o").T, S.flatten()
