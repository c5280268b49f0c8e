"""Calls that programs make of this library, at sizes they make them at: whole requests through `Engine`, and single parts
(mixers, routed experts) built with `build_part` and run over a step's tokens against a paged cache, as a model of a
registered architecture or a plugin runs them.  Used to time the library and to compare its outputs with 64-bit results.

A case is a dict of plain values.  `kind` names what runs; a part's case has

  new      tokens the step brings, per sequence ("700,33": two sequences);  past  positions each sequence has before it
  width    the residual's width;  dtype  "bf16" or "f32"

and the part's own sizes.  A step with one token per sequence is a decode step: the engine replays those as CUDA graphs
captured once per batch size, so a decode case's state holds such a graph.  Prompts are launched directly.
"""
from __future__ import annotations

import math

import torch

from cpi_b200.cache import CacheManager
from cpi_b200.config.spec import PartSpec
from cpi_b200.engine import Engine, StepEntry
from cpi_b200.engine.batch import BatchStager
from cpi_b200.models import llama4 as _llama4, veredra as _veredra   # noqa: F401  (registers the architectures and parts)
from cpi_b200.parts import CacheView, Workspace, build_part
from cpi_b200.weights import DictSource, RandomSource
from cpi_b200.config.registry import architecture_of
from cpi_b200.engine.model import tensor_requirements

DEV = "cuda:0"
EPS = 1e-6
THETA = 5e5
STD = 0.02                         # what random weights are drawn with


# ---- the cases -----------------------------------------------------------------------------------------------------
def listed():
    return [
        # One short question to a small dense decoder: a prompt of a few words and eight tokens of the answer.  Latency:
        # nothing here is large, launches and the host's part of a step count.
        {"name": "request_short", "kind": "request", "arch": "llama", "width": 2048, "ff": 8192, "heads": 16, "kv_heads": 4,
         "dim": 128, "new": "24", "steps": 8, "vocab": 32000},
        # Four unequal prompts to a hybrid decoder (gated linear attention, windowed attention, state-space layer), then
        # four tokens each: prompts and decode steps of recurrent layers through the engine.
        {"name": "request_hybrid", "kind": "request", "arch": "veredra", "width": 2048, "ff": 8192, "heads": 16, "kv_heads": 4,
         "dim": 128, "new": "37,700,260,411", "steps": 4, "vocab": 32000},
        # A decode step's routed experts at the layer sizes of the headline benchmark, batch 8: bound by reading weights.
        {"name": "experts_decode", "kind": "experts", "new": "1,1,1,1,1,1,1,1", "past": 0, "width": 5120, "experts": 16, "top": 1,
         "ff": 8192, "shared": 8192, "gate": "sigmoid_input", "dtype": "bf16"},
        # A prompt's routed experts, four of sixteen per token: the grouped products at many rows, and the routing.
        {"name": "experts_prompt", "kind": "experts", "new": "2048", "past": 0, "width": 2048, "experts": 16, "top": 4, "ff": 2048,
         "shared": 0, "gate": "softmax_chosen", "dtype": "bf16"},
        # A decode step of attention, eight sequences at a context of 4,096: the headline benchmark's attention layer.
        {"name": "attention_decode", "kind": "attention", "new": "1,1,1,1,1,1,1,1", "past": 4095, "width": 5120, "heads": 40,
         "kv_heads": 8, "dim": 128, "dtype": "bf16"},
        # A prompt of an odd length through the same layer.
        {"name": "attention_prompt", "kind": "attention", "new": "3001", "past": 0, "width": 5120, "heads": 40, "kv_heads": 8,
         "dim": 128, "dtype": "bf16"},
        # The float32 path, which users take to check results: a prompt through an attention layer.
        {"name": "attention_prompt_f32", "kind": "attention", "new": "509", "past": 0, "width": 2048, "heads": 16, "kv_heads": 4,
         "dim": 128, "dtype": "f32"},
        # Attention over a cached latent: a long prompt, and a decode step at batch 8 over a context of 2,000.
        {"name": "latent_prompt", "kind": "latent", "new": "2048", "past": 0, "width": 2048, "heads": 16, "dim": 128, "rot": 64,
         "vdim": 128, "q_rank": 768, "kv_rank": 512, "dtype": "bf16"},
        {"name": "latent_decode", "kind": "latent", "new": "1,1,1,1,1,1,1,1", "past": 2000, "width": 2048, "heads": 16, "dim": 128,
         "rot": 64, "vdim": 128, "q_rank": 768, "kv_rank": 512, "dtype": "bf16"},
        # Recurrent layers over a prompt: gated linear attention, a state-space layer over three unequal prompts in one
        # step, and the gated delta rule over a later piece of a prompt.
        {"name": "gla_prompt", "kind": "gla", "new": "2048", "past": 0, "width": 2048, "heads": 8, "dim": 128, "vdim": 256,
         "dtype": "bf16"},
        {"name": "mamba2_prompt", "kind": "mamba2", "new": "1025,130,700", "past": 0, "width": 2048, "heads": 64, "vdim": 64,
         "state": 128, "groups": 8, "dtype": "bf16"},
        {"name": "delta_prompt", "kind": "delta", "new": "1500", "past": 1000, "width": 2048, "heads": 8, "kv_heads": 4, "dim": 128,
         "vdim": 256, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _prompts(rng, most):
    """Lengths of one to four prompts of a step, `most` tokens together at most."""
    n = rng.choice((1, 1, 2, 4))
    return ",".join(str(max(20, _log(rng, 40, most) // n)) for _ in range(n))


def _ones(n):
    return ",".join(["1"] * n)


def draw(rng):
    kind = rng.choice(("request", "request", "experts", "experts", "attention", "attention", "attention_f32", "latent", "latent",
                       "gla", "gla", "mamba2", "mamba2", "delta", "delta"))
    width = rng.choice((1024, 1536, 2048, 3072))
    decode = rng.random() < 0.35
    if kind == "request":
        n, width = rng.choice((1, 1, 2, 4, 8)), min(width, 2048)
        heads = rng.choice((8, 16))
        return {"kind": "request", "arch": rng.choice(("llama", "veredra")), "width": width, "ff": 4 * width, "heads": heads,
                "kv_heads": rng.choice((2, 4, heads)), "dim": 128, "new": ",".join(str(_log(rng, 5, 1400 // n)) for _ in range(n)),
                "steps": rng.randint(2, 6), "vocab": 32000}
    if kind == "experts":
        top = rng.choice((1, 1, 2, 4))
        return {"kind": "experts", "new": _ones(_log(rng, 1, 64)) if decode else _prompts(rng, 2048), "past": 0, "width": width,
                "experts": rng.choice((8, 16, 32)), "top": top, "ff": rng.choice((768, 1024, 2048)),
                "shared": rng.choice((0, 1024)), "gate": "sigmoid_input" if top == 1 else "softmax_chosen", "dtype": "bf16"}
    if kind in ("attention", "attention_f32"):
        kv = rng.choice((2, 4, 8))
        f32 = kind == "attention_f32"
        return {"kind": "attention", "new": _ones(_log(rng, 1, 32)) if decode else _prompts(rng, 500 if f32 else 3000),
                "past": _log(rng, 30, 4000) if decode else 0, "width": min(width, 2048) if f32 else width,
                "heads": kv * rng.choice((1, 2, 4)) if f32 else kv * rng.choice((1, 4, 5)), "kv_heads": kv,
                "dim": rng.choice((64, 128)), "dtype": "f32" if f32 else "bf16"}
    if kind == "latent":
        heads = rng.choice((8, 16, 24))
        return {"kind": "latent", "new": _ones(_log(rng, 1, 32)) if decode else _prompts(rng, 2048),
                "past": _log(rng, 30, 4000) if decode else rng.choice((0, 0, 333)), "width": width, "heads": heads, "dim": 128,
                "rot": 64, "vdim": 128, "q_rank": rng.choice((512, 768)), "kv_rank": rng.choice((256, 512)), "dtype": "bf16"}
    new = _ones(_log(rng, 1, 32)) if decode else _prompts(rng, 2048)
    past = rng.choice((0, 900))
    if kind == "mamba2":
        groups = rng.choice((1, 2, 8))
        return {"kind": "mamba2", "new": new, "past": past, "width": width, "heads": groups * (width // 32 // groups), "vdim": 64,
                "state": rng.choice((64, 128)), "groups": groups, "dtype": "bf16"}
    heads = rng.choice((4, 8, 12))
    sizes = {"new": new, "past": past, "width": width, "heads": heads, "dim": rng.choice((64, 128)),
             "vdim": rng.choice((64, 128, 256)), "dtype": "bf16"}
    if kind == "gla":
        return {"kind": "gla", **sizes}
    return {"kind": "delta", **sizes, "kv_heads": heads // rng.choice((1, 2))}


# ---- parts: their specs, and inputs drawn from a seed -----------------------------------------------------------------
def _news(c):
    return [int(n) for n in str(c["new"]).split(",")]


def _dtype(c):
    return torch.float32 if c.get("dtype") == "f32" else torch.bfloat16


def _spec(c):
    """(family of the part, its PartSpec)."""
    k, W = c["kind"], c["width"]
    if k == "experts":
        return "feed_forward", PartSpec("moe_swiglu", {"hidden_size": W, "num_experts": c["experts"], "top_k": c["top"],
                                                       "expert_size": c["ff"], "shared_size": c["shared"], "router_gate": c["gate"]})
    if k == "attention":
        rope = PartSpec("rope", {"head_dim": c["dim"], "theta": THETA, "pairing": "half_split", "scaling": None,
                                 "frequency_math": "float64"})
        return "mixer", PartSpec("attention", {"hidden_size": W, "num_heads": c["heads"], "num_kv_heads": c["kv_heads"],
                                               "head_dim": c["dim"], "softmax_scale": c["dim"] ** -0.5, "position": rope,
                                               "qk_norm": True, "qk_norm_eps": EPS, "window": None, "query_temperature": None})
    if k == "latent":
        rope = PartSpec("rope", {"head_dim": c["rot"], "theta": 1e4, "pairing": "half_split", "scaling": None,
                                 "frequency_math": "float64"})
        return "mixer", PartSpec("latent_attention", {"hidden_size": W, "heads": c["heads"], "head_dim": c["dim"], "rot_dim": c["rot"],
                                                      "value_dim": c["vdim"], "q_rank": c["q_rank"], "kv_rank": c["kv_rank"],
                                                      "softmax_scale": (c["dim"] + c["rot"]) ** -0.5, "norm_eps": EPS,
                                                      "position": rope, "sink": False})
    if k == "gla":
        return "mixer", PartSpec("gla", {"hidden_size": W, "heads": c["heads"], "key_dim": c["dim"], "value_dim": c["vdim"],
                                         "tau": 16.0, "decay_rank": 16, "norm_eps": EPS})
    if k == "mamba2":
        return "mixer", PartSpec("mamba2", {"hidden_size": W, "heads": c["heads"], "head_dim": c["vdim"], "state": c["state"],
                                            "groups": c["groups"], "conv": 4, "norm_groups": c["groups"], "norm_eps": EPS})
    if k == "delta":
        return "mixer", PartSpec("gated_delta", {"hidden_size": W, "heads": c["heads"], "kv_heads": c["kv_heads"], "key_dim": c["dim"],
                                                 "value_dim": c["vdim"], "conv": 4, "decay_rank": 32, "gate_rank": 32,
                                                 "norm_eps": EPS, "unit_eps": EPS})
    raise ValueError(f"no case of kind '{k}'")


def _weight(req, g, dtype):
    """A tensor as a checkpoint of such a layer holds it: norms around one, the state-space layers' rates and step sizes
    in the ranges they are initialised to, everything else small and normal."""
    name, shape = req.name, tuple(req.shape)
    if name.endswith("A_log"):                       # rates from 1 to 16
        return torch.log(1 + 15 * torch.rand(shape, generator=g, device=DEV))
    if name.endswith("dt_bias"):                     # softplus of it: step sizes from 0.001 to 0.1
        dt = torch.exp(torch.rand(shape, generator=g, device=DEV) * math.log(100.0) + math.log(1e-3))
        return dt + torch.log(-torch.expm1(-dt))
    t = torch.randn(shape, generator=g, device=DEV, dtype=torch.float32 if len(shape) < 3 else dtype) * STD
    if "ones" in req.init:
        t += 1
    if "const" in req.init or name.endswith("conv1d.weight"):
        t += 0.3
    return t.to(dtype)


def _draw_inputs(c, seed):
    """What the layer reads: its weights, the normed rows of the step, and what the sequences have left in the cache."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    family, spec = _spec(c)
    part = build_part(family, spec, "", workspace=Workspace(DEV))
    w = {r.name: _weight(r, g, _dtype(c)) for r in part.requirements()}
    new, dt = _news(c), _dtype(c)
    x = {"part": part, "w": w, "h": randn(sum(new), c["width"]).to(dt), "past": {}, "state": {}}
    if family == "feed_forward":
        x["residual"] = randn(sum(new), c["width"])
    elif part.kv_requirement() is not None:
        for name, heads, dim in part.kv_requirement().stream_shapes():
            x["past"][name] = randn(len(new), heads, c["past"], dim).to(dt)
    for r in getattr(part, "state_requirements", lambda: [])():
        x["state"][r.name] = randn(len(new), *r.shape) * (0.1 if c["past"] else 0.0)
    return x


# ---- whole models ------------------------------------------------------------------------------------------------------
def _config(c):
    W, ff, H, G, D, V = c["width"], c["ff"], c["heads"], c["kv_heads"], c["dim"], c["vocab"]
    if c["arch"] == "llama":
        return {"architectures": ["Llama4ForCausalLM"], "num_hidden_layers": 2, "hidden_size": W, "num_attention_heads": H,
                "num_key_value_heads": G, "head_dim": D, "intermediate_size": ff, "intermediate_size_mlp": ff,
                "num_local_experts": 1, "num_experts_per_tok": 1, "interleave_moe_layer_step": 1 << 20, "vocab_size": V,
                "rms_norm_eps": EPS, "rope_theta": THETA, "nope_layer_interval": 0, "attention_chunk_size": 8192,
                "use_qk_norm": True, "attn_temperature_tuning": False, "tie_word_embeddings": False,
                "max_position_embeddings": 8192, "initializer_range": STD}
    mlp = {"kind": "dense", "ff": ff}
    return {"architecture": "Veredra", "norm": {"eps": EPS}, "vocab": V, "width": W, "logit_scale": 1.0, "logit_softcap": 30.0,
            "layers": [{"type": "gla", "mixer": {"heads": W // 256, "dim": 128, "vdim": 256, "tau": 16.0}, "mlp": mlp},
                       {"type": "attention", "mixer": {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": D ** -0.5,
                                                       "rot": {"base": THETA, "dims": D // 2}, "mask": {"size": 512}}, "mlp": mlp},
                       {"type": "mamba2", "mixer": {"heads": W // 32, "vdim": 64, "state": 128, "groups": 8, "conv": 4,
                                                    "norm_groups": 8}, "mlp": mlp}]}


def _model_inputs(c, seed):
    cfg = _config(c)
    arch = architecture_of(cfg)
    parsed = arch.parse_config(cfg)
    spec = arch.build_spec(parsed)
    src = RandomSource(tensor_requirements(spec), seed, spec.initializer_range)
    g = torch.Generator().manual_seed(int(seed))
    toks = [torch.randint(0, c["vocab"], (n + c["steps"],), generator=g).tolist() for n in _news(c)]
    return cfg, parsed, spec, src, toks


# ---- the calls -----------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "request":
        cfg, parsed, spec, src, toks = _model_inputs(c, seed)
        new = _news(c)
        eng = Engine(spec, src, config=parsed, dtype="bfloat16", device=DEV, max_seqs=len(new),
                     max_tokens=sum(-(-(n + c["steps"]) // 64) * 64 for n in new))
        return {"kind": "request", "engine": eng, "toks": toks, "new": new, "steps": c["steps"]}
    x = _draw_inputs(c, seed)
    part, new, past, dt = x["part"], _news(c), int(c["past"]), _dtype(c)
    part.load(DictSource(x["w"]), DEV)
    s = {"kind": c["kind"], "part": part, "h": x["h"], "out": torch.zeros(x["h"].shape, device=DEV), "graph": None}
    s["batch"] = None
    if "residual" in x:
        s["residual"], slots, starts = x["residual"], list(range(len(new))), [0] * len(new)
    else:
        kv, st = part.kv_requirement(), part.state_requirements()
        room = sum(-(-(past + n) // 64) * 64 for n in new)
        cache = CacheManager({0: kv} if kv is not None else {}, {0: st} if st else {}, max_tokens=room, max_seqs=len(new),
                             dtype=dt, device=DEV)
        slots, starts = [cache.acquire() for _ in new], [past] * len(new)
        if past:
            cache.prepare_step(slots, [past] * len(new))
            cache.commit_step(slots, [past] * len(new))
        cache.prepare_step(slots, new)
        for name, rows in x["past"].items() if past else ():
            pages, table, ps = cache.stream_view(0, name)
            full = torch.zeros(*rows.shape[:2], -(-past // ps) * ps, rows.shape[3], dtype=dt, device=DEV)
            full[:, :, :past] = rows
            for i, slot in enumerate(slots):
                n = full.shape[2] // ps
                pages[table[slot, :n].long()] = full[i].view(rows.shape[1], n, ps, -1).transpose(0, 1)
        s["cache"], s["view"], s["slots"] = cache, CacheView(cache, 0), slots
        s["streams"] = {name: cache.stream_view(0, name)[0] for name in x["past"]}
        s["states"] = {name: cache.state_view(0, name) for name in x["state"]}

        def fill():
            for name, t in x["state"].items():
                s["states"][name][torch.tensor(slots, device=DEV)] = t
        fill()
    stager = BatchStager(DEV)                      # (kept: it owns the device buffer that the batch's arrays live in)
    s["stager"] = stager
    s["batch"] = stager.stage(slots, starts, [[0] * n for n in new], [[] for _ in new], dt)
    if max(new) == 1:
        _forward(s)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _forward(s)
        s["graph"] = graph
        if "states" in s:
            fill()
    return s


def _forward(s):
    if "residual" in s:                            # the layer's output is added to the residual
        s["out"].copy_(s["residual"])
        s["part"].forward(s["h"], s["out"], s["batch"])
    else:
        s["part"].forward(s["h"], s["out"], s["batch"], s["view"], add=False)


def run(s):
    if s["kind"] == "request":
        eng, new, toks = s["engine"], s["new"], s["toks"]
        slots = [eng.acquire_slot() for _ in new]
        out = [eng.step([StepEntry(sl, t[:n], [n - 1]) for sl, t, n in zip(slots, toks, new)]).clone()]
        for i in range(s["steps"]):
            out.append(eng.step([StepEntry(sl, [t[n + i]], [0]) for sl, t, n in zip(slots, toks, new)]).clone())
        for sl in slots:
            eng.release_slot(sl)
        return {"logits": torch.stack(out)}
    if s["graph"] is not None:
        s["graph"].replay()
    else:
        _forward(s)
    if "residual" in s:
        return {"out": s["out"]}
    return {"out": s["out"], **{"pages." + n: t for n, t in s["streams"].items()},
            **{"state." + n: t for n, t in s["states"].items()}}


# ---- work and tolerance ----------------------------------------------------------------------------------------------------
def _pairs(new, past, window=1 << 40):
    """Query-key pairs of causal attention."""
    return sum(min(past + i + 1, window) for n in new for i in range(n))


def _recurrent_work(c, T, n):
    """(weights, flops beside the products with weights, state elements) of a recurrent mixer."""
    W, H, dv = c["width"], c["heads"], c["vdim"]
    if c["kind"] == "mamba2":
        inner, gn, dk = H * dv, c["groups"] * c["state"], c["state"]
        weights = W * (2 * inner + 2 * gn + H) + W * inner
    else:
        dk = c["dim"]
        qk, v = c.get("kv_heads", H) * dk, H * dv
        weights = W * (2 * qk + 2 * v) + W * v
        if c["kind"] == "delta":
            weights = W * (2 * qk + v + H + 64) + 32 * (H * dk + v) + W * v
    per_token = (4 if c["kind"] != "delta" else 6) * H * dk * dv
    return weights, T * per_token, n * H * dk * dv


def work(c):
    new = _news(c)
    T, W, n = sum(new), c["width"], len(new)
    if c["kind"] == "request":
        H, G, D, ff, V = c["heads"], c["kv_heads"], c["dim"], c["ff"], c["vocab"]
        attn = W * D * (2 * H + 2 * G)
        layers = 2 * (attn + 3 * W * ff)
        if c["arch"] == "veredra":
            inner = 2 * W
            layers = 3 * 3 * W * ff + attn + 3 * W * W + 2 * W * W // 2 + W * (2 * inner + 2048 + W // 32) + W * inner
        steps = c["steps"]
        return {"bytes": 2.0 * (layers + V * W) * (1 + steps) + 4.0 * V * n * (1 + steps),
                "flops": 2.0 * layers * (T + n * steps) + 2.0 * V * W * n * (1 + steps)}
    size = 4 if c["dtype"] == "f32" else 2
    rows = T * W * (size + 4)
    past = int(c["past"])
    if c["kind"] == "experts":
        touched = c["experts"] * (1 - (1 - c["top"] / c["experts"]) ** T)
        per = 3 * W * c["ff"]
        return {"bytes": 2.0 * (touched * per + 3 * W * c["shared"] + c["experts"] * W) + rows + 4.0 * T * W,
                "flops": 2.0 * T * (c["top"] * per + 3 * W * c["shared"] + c["experts"] * W)}
    if c["kind"] == "attention":
        H, G, D = c["heads"], c["kv_heads"], c["dim"]
        weights = W * D * (2 * H + 2 * G)
        return {"bytes": float(size * (weights + 2 * G * D * (n * past + T)) + rows),
                "flops": 2.0 * T * weights + 4.0 * H * D * _pairs(new, past)}
    if c["kind"] == "latent":
        H, d, r, dv, row = c["heads"], c["dim"], c["rot"], c["vdim"], c["kv_rank"] + c["rot"]
        weights = W * (c["q_rank"] + row) + c["q_rank"] * H * (d + r) + c["kv_rank"] * H * (d + dv) + W * H * dv
        pairs = _pairs(new, past)
        absorbed = 2.0 * H * (row + c["kv_rank"]) * pairs + 2.0 * T * c["kv_rank"] * H * (d + dv)
        plain = 2.0 * H * (d + r + dv) * pairs + 2.0 * (T + n * past) * c["kv_rank"] * H * (d + dv)
        return {"bytes": float(size * (weights + row * (n * past + T)) + rows),
                "flops": 2.0 * T * (weights - c["kv_rank"] * H * (d + dv)) + min(absorbed, plain)}
    weights, flops, state = _recurrent_work(c, T, n)
    return {"bytes": float(size * weights + 8 * state + rows), "flops": 2.0 * T * weights + flops}


def tolerance(c):
    if c.get("dtype") == "f32":
        return {"rel": 1e-5}
    if c["kind"] == "request":                     # two or three layers: a rounding travels through what follows (seen: 1e-2)
        return {"rel": 3e-2}
    return {"rel": 1e-2}                           # seen: 2e-3 to 3e-3


# ---- the same results in 64 bits ----------------------------------------------------------------------------------------------
def _rms(x, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _rotate(x, pos, theta, dims):
    """Pairs (i, i + dims / 2) of the first `dims` elements turn by pos * theta^(-2i / dims).  x [T, heads, D]."""
    half = dims // 2
    f = (theta ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / dims)).float().double()
    a = pos.double()[:, None] * f
    co, si = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * co - v * si, v * co + u * si, x[..., dims:]], -1)


def _softmax_attention(q, k, v, scale, start, window=1 << 40, sink=None):
    """q [T, H, D] at positions start ..; k [S, G, D], v [S, G, Dv] at positions 0 ..."""
    T, H, _ = q.shape
    S, G, _ = k.shape
    dist = (start + torch.arange(T, device=q.device))[:, None] - torch.arange(S, device=q.device)[None, :]
    hide = (dist < 0) | (dist >= window)
    out = torch.empty(T, H, v.shape[2], dtype=torch.float64, device=q.device)
    for h in range(H):
        s = (q[:, h] @ k[:, h // (H // G)].T * scale).masked_fill(hide, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out[:, h] = torch.softmax(s, -1)[:, :S] @ v[:, h // (H // G)]
    return out


def _conv(x, w, bias, carry):
    """Causal convolution per channel, x [T, C], w [C, taps], the inputs before it in carry [taps - 1, C]."""
    taps, T = w.shape[1], x.shape[0]
    full = torch.cat([carry, x])
    y = sum(full[j:j + T] * w[:, j] for j in range(taps))
    return torch.nn.functional.silu(y if bias is None else y + bias), full[T:]


def _scan(a, k, v, q, S, beta=None):
    """S <- diag(a) S + k u^T with u = v, or beta (v - S^T k) after the decay;  o = S^T q.  a, k, q [T, H, dk], v [T, H, dv]."""
    o = torch.empty(v.shape, dtype=torch.float64, device=v.device)
    S = S.clone()
    for t in range(v.shape[0]):
        S *= a[t][:, :, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S += k[t][:, :, None] * u[:, None, :]
        o[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return o, S


def _gla(h, w, H, dk, dv, S):
    q, k, v = ((h @ w("mixer.%s_proj.weight" % n).T).view(h.shape[0], H, -1) for n in "qkv")
    z = h @ w("mixer.gk_proj.0.weight").T @ w("mixer.gk_proj.1.weight").T + w("mixer.gk_proj.1.bias")
    a = torch.exp(torch.nn.functional.logsigmoid(z) / 16.0).view(-1, H, dk)
    o, S = _scan(a, k, v, q * dk ** -0.5, S)
    o = (_rms(o, w("mixer.g_norm.weight"))).reshape(h.shape[0], H * dv) * torch.nn.functional.silu(h @ w("mixer.g_proj.weight").T)
    return o @ w("mixer.o_proj.weight").T, S


def _mamba2(h, w, H, dv, N, G, S, carry):
    inner, T = H * dv, h.shape[0]
    p = h @ w("mixer.in_proj.weight").T
    z, x, dt = p[:, :inner], p[:, inner:2 * inner + 2 * G * N], p[:, 2 * inner + 2 * G * N:]
    x, carry = _conv(x, w("mixer.conv1d.weight"), w("mixer.conv1d.bias"), carry)
    B, C = (x[:, inner + i * G * N:inner + (i + 1) * G * N].view(T, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    x = x[:, :inner].view(T, H, dv)
    dt = torch.nn.functional.softplus(dt + w("mixer.dt_bias"))
    a = torch.exp(-torch.exp(w("mixer.A_log")) * dt)
    y, S = _scan(a[:, :, None].expand(T, H, N), B, dt[:, :, None] * x, C, S)
    y = (y + w("mixer.D")[:, None] * x).reshape(T, inner) * torch.nn.functional.silu(z)
    y = _rms(y.view(T, G, inner // G)).reshape(T, inner) * w("mixer.norm.weight")
    return y @ w("mixer.out_proj.weight").T, S, carry


def _delta(h, w, H, G, dk, dv, S, carry):
    T = h.shape[0]
    p = lambda n: h @ w("mixer.%s.weight" % n).T
    qkv = torch.cat([p("q_proj"), p("k_proj"), p("v_proj")], 1)
    taps = torch.cat([w("mixer.%s_conv.weight" % n) for n in "qkv"])
    x, carry = _conv(qkv, taps, None, carry)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + EPS)
    q, k = (unit(x[:, i * G * dk:(i + 1) * G * dk].view(T, G, dk)).repeat_interleave(H // G, 1) for i in (0, 1))
    rate = torch.exp(w("mixer.A_log"))[:, None]
    a = torch.exp(-rate * torch.nn.functional.softplus(p("a_proj.0") @ w("mixer.a_proj.1.weight").T + w("mixer.dt_bias")).view(T, H, dk))
    o, S = _scan(a, k, x[:, 2 * G * dk:].view(T, H, dv), q * dk ** -0.5, S, beta=torch.sigmoid(p("b_proj")))
    o = _rms(o, w("mixer.o_norm.weight")).reshape(T, H * dv) * torch.sigmoid(p("g_proj.0") @ w("mixer.g_proj.1.weight").T)
    return o @ w("mixer.o_proj.weight").T, S, carry


def _experts(c, h, w, residual):
    logits = h @ w("feed_forward.router.weight").T
    top, idx = logits.topk(c["top"], -1)
    out = residual.double().clone()
    swiglu = lambda x, gu, down: (torch.nn.functional.silu(x @ gu[:, :gu.shape[1] // 2]) * (x @ gu[:, gu.shape[1] // 2:])) @ down
    gate = torch.sigmoid(top) if c["gate"] == "sigmoid_input" else torch.softmax(top, -1)
    for e in range(c["experts"]):
        t, j = (idx == e).nonzero(as_tuple=True)
        if not t.numel():
            continue
        s, x = gate[t, j][:, None], h[t]
        gu, down = w("feed_forward.experts.gate_up_proj", e), w("feed_forward.experts.down_proj", e)
        out[t] += swiglu(x * s, gu, down) if c["gate"] == "sigmoid_input" else s * swiglu(x, gu, down)
    if c["shared"]:
        gu = torch.cat([w("feed_forward.shared_expert.%s_proj.weight" % n) for n in ("gate", "up")]).T
        out += swiglu(h, gu, w("feed_forward.shared_expert.down_proj.weight").T)
    return out


def _exact_request(c, seed):
    cfg, parsed, spec, src, toks = _model_inputs(c, seed)
    get = lambda n: src.get(n, DEV).double()
    V, W, H, G, D, steps = c["vocab"], c["width"], c["heads"], c["kv_heads"], c["dim"], c["steps"]
    llama = c["arch"] == "llama"
    pre, one = ("model.", 0.0) if llama else ("", 1.0)
    emb, head = get(pre + "embed_tokens.weight" if llama else "embed"), get("lm_head.weight" if llama else "head")
    fin = get(pre + "norm.weight" if llama else "final.norm")
    rename = {"mixer.gk_proj.0.weight": "a1", "mixer.gk_proj.1.weight": "a2", "mixer.gk_proj.1.bias": "a2.b",
              "mixer.g_norm.weight": "norm", "mixer.in_proj.weight": "in", "mixer.conv1d.weight": "conv",
              "mixer.conv1d.bias": "conv.b", "mixer.out_proj.weight": "o", "mixer.norm.weight": "norm"}
    rows = []
    for seq in toks:
        T = len(seq)
        x = emb[torch.tensor(seq, device=DEV)]
        pos = torch.arange(T, device=DEV)
        zeros = lambda *s: torch.zeros(*s, dtype=torch.float64, device=DEV)
        for i in range(len(spec.layers)):
            kind = "attention" if llama else cfg["layers"][i]["type"]
            l = f"model.layers.{i}." if llama else f"l{i}."
            w = lambda n: get(l + (n if llama else "mix." + rename.get(n, n.replace("mixer.", "").replace("_proj.weight", ""))))
            h = _rms(x, one + get(l + ("input_layernorm.weight" if llama else "norm1")))
            if kind == "gla":
                y = _gla(h, w, W // 256, 128, 256, zeros(W // 256, 128, 256))[0]
            elif kind == "mamba2":
                y = _mamba2(h, w, W // 32, 64, 128, 8, zeros(W // 32, 128, 64), zeros(3, 2 * W + 2048))[0]
            elif llama:
                q, k, v = ((h @ w("self_attn.%s_proj.weight" % n).T).view(T, -1, D) for n in "qkv")
                q, k = (_rms(_rotate(t, pos, THETA, D)) for t in (q, k))
                y = _softmax_attention(q, k, v, D ** -0.5, 0).reshape(T, H * D) @ w("self_attn.o_proj.weight").T
            else:
                q, k, v = (h @ get(l + "mix." + n).T + get(l + "mix." + n + ".b") for n in "qkv")
                q, k = ((_rms(t) * get(l + "mix." + n + ".norm")).view(T, -1, D) for t, n in ((q, "q"), (k, "k")))
                q, k = (_rotate(t, pos, THETA, D // 2) for t in (q, k))
                y = _softmax_attention(q, k, v.view(T, G, D), D ** -0.5, 0, 512, get(l + "mix.sink")).reshape(T, H * D) @ get(l + "mix.o").T
            x = x + y
            h = _rms(x, one + get(l + ("post_attention_layernorm.weight" if llama else "norm2")))
            gate, up, down = (get(l + (f"feed_forward.{n}_proj.weight" if llama else "mlp." + n)) for n in ("gate", "up", "down"))
            act = torch.nn.functional.silu(h @ gate.T) if llama else torch.nn.functional.gelu(h @ gate.T, approximate="tanh")
            x = x + (act * (h @ up.T)) @ down.T
        x = _rms(x[T - steps - 1:], one + fin)
        logits = x @ head.T
        rows.append(logits if llama else 30.0 * torch.tanh(logits / 30.0))
    return {"logits": torch.stack(rows, 1)}


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "request":
        return _exact_request(c, seed)
    x = _draw_inputs(c, seed)

    def w(name, e=None):
        t = x["w"][name]
        return (t if e is None else t[e]).double()
    h = x["h"].double()
    if c["kind"] == "experts":
        return {"out": _experts(c, h, w, x["residual"])}
    past, out, at, states = int(c["past"]), [], 0, {n: [] for n in x["state"]}
    for i, n in enumerate(_news(c)):
        hi = h[at:at + n]
        at += n
        pos = past + torch.arange(n, device=DEV)
        if c["kind"] == "attention":
            H, D = c["heads"], c["dim"]
            q, k, v = ((hi @ w("self_attn.%s_proj.weight" % m).T).view(n, -1, D) for m in "qkv")
            q, k = (_rms(_rotate(t, pos, THETA, D)) for t in (q, k))
            k, v = (torch.cat([x["past"][m][i].double().transpose(0, 1), t]) for m, t in (("k", k), ("v", v)))
            y = _softmax_attention(q, k, v, D ** -0.5, past).reshape(n, H * D) @ w("self_attn.o_proj.weight").T
        elif c["kind"] == "latent":
            H, d, r, dv, rank = c["heads"], c["dim"], c["rot"], c["vdim"], c["kv_rank"]
            q = _rms(hi @ w("mixer.q_a_proj.weight").T, w("mixer.q_a_norm.weight")) @ w("mixer.q_b_proj.weight").T
            q = q.view(n, H, d + r)
            q = torch.cat([q[..., :d], _rotate(q[..., d:], pos, 1e4, r)], -1)
            low = hi @ w("mixer.kv_a_proj.weight").T
            low = torch.cat([_rms(low[:, :rank], w("mixer.kv_a_norm.weight")), _rotate(low[:, None, rank:], pos, 1e4, r)[:, 0]], 1)
            low = torch.cat([x["past"]["latent"][i, 0].double(), low])
            k = torch.cat([(low[:, :rank] @ w("mixer.k_b_proj.weight").T).view(-1, H, d),
                           low[:, None, rank:].expand(-1, H, r)], -1)
            v = (low[:, :rank] @ w("mixer.v_b_proj.weight").T).view(-1, H, dv)
            y = _softmax_attention(q, k, v, (d + r) ** -0.5, past).reshape(n, H * dv) @ w("mixer.o_proj.weight").T
        else:
            st = {m: t[i].double() for m, t in x["state"].items()}
            if c["kind"] == "gla":
                y, st["s"] = _gla(hi, w, c["heads"], c["dim"], c["vdim"], st["s"])
            elif c["kind"] == "mamba2":
                y, st["ssm"], st["conv"] = _mamba2(hi, w, c["heads"], c["vdim"], c["state"], c["groups"], st["ssm"], st["conv"])
            else:
                y, st["s"], st["conv"] = _delta(hi, w, c["heads"], c["kv_heads"], c["dim"], c["vdim"], st["s"], st["conv"])
            for m, t in st.items():
                states[m].append(t)
        out.append(y)
    got = {"out": torch.cat(out)}
    got.update({"pages." + m: None for m in x["past"]})
    got.update({"state." + m: torch.stack(t) for m, t in states.items()})
    return got
