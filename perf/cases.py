"""What a user has this library do, as cases that can be timed and checked.

A case is one batch of requests through an engine that is already loaded, the way a serving or a
scoring program runs it: slots are taken, the prompts go through one step of ``Engine.step`` and
give the logits of their last tokens, ``steps`` further steps bring one known token a sequence
(teacher forced, as the trace replay does, so that a pass computes the same whatever an
implementation's rounding makes of a near tie), and the slots are given back.  A case with
``use = "generate"`` calls ``Engine.generate`` instead and then scores what was generated in one
step.  The engine outlives the pass, as it does in a program; prompts and fed tokens come from the
seed.

Models are the ones the library's presets, configurations and benchmark name: SmolLM2 sizes
(Llama) and the mixed models of the six other architectures at the benchmark's sizes ``s`` and
``m``, eight layers (or layer runs), with random weights.

A case: ``model``; ``dtype``; ``batch`` sequences whose prompts are ``shortest`` to ``longest``
tokens long (spread evenly over the logarithm, all of one length where the two are equal);
``steps`` decode steps after the prompt step; ``use`` "replay" or "generate".
"""
from __future__ import annotations

import math
import os
import shutil
import tempfile
import zlib
from typing import Dict, List

import numpy as np
import torch

VOCAB = 49152
MAX_POSITIONS = 4096

# ------------------------------------------------------------------------------------------
# models
# ------------------------------------------------------------------------------------------
SIZES = {
    "s": dict(width=576, ff=1536, heads=9, kv=3, dim=64, rank=128, d_heads=9, d_dim=64,
              window=1024, experts=8, top=2, expert_ff=384, decay_rank=32, ssm_groups=3),
    "m": dict(width=2048, ff=8192, heads=32, kv=8, dim=64, rank=128, d_heads=16, d_dim=128,
              window=1024, experts=32, top=4, expert_ff=1024, decay_rank=64, ssm_groups=4),
}
LAYERS = 8


def _moe(z, **router):
    return {"kind": "moe", "expert": {"ff": z["expert_ff"]},
            "router": {"experts": z["experts"], "top": z["top"], **router}}


def _rigozen(z):
    grouped = {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["dim"],
               "scale": z["dim"] ** -0.5, "mask": {"size": z["window"]}}
    latent = {"heads": z["heads"], "dim": z["dim"], "vdim": z["dim"], "kv_rank": z["rank"],
              "scale": z["dim"] ** -0.5, "mask": {"size": z["window"]}}
    delta = {"heads": z["d_heads"], "kv_heads": z["d_heads"], "dim": z["d_dim"],
             "vdim": z["d_dim"], "conv": 4}
    kinds = {"attention": grouped, "delta": delta, "latent_attention": latent}
    order = ["attention", "delta", "delta", "latent_attention"] * (LAYERS // 4)
    return {"architecture": "Rigozen", "norm": {"eps": 1e-6},
            "layers": [{"type": k, "mixer": kinds[k], "mlp": {"kind": "dense", "ff": z["ff"]}}
                       for k in order]}


def _losorax(z):
    att = {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["dim"],
           "scale": z["dim"] ** -0.5, "conv": 4, "bias_max": 1024, "bias_rows": 48,
           "q_temp": {"coef": 0.25, "every": 256}}
    delta = {"heads": z["d_heads"], "dim": z["d_dim"], "decay_rank": z["decay_rank"]}
    layers = []
    for i in range(LAYERS):
        kind = ["attention", "reader", "general_delta", "attention"][i % 4]
        mixer = delta if kind == "general_delta" else dict(att, kv_from=i - 1) \
            if kind == "reader" else att
        layers.append({"type": "attention" if kind == "reader" else kind, "mixer": mixer,
                       "mlp": _moe(z)})
    return {"architecture": "Losorax", "norm": {"eps": 1e-6}, "layers": layers}


def _virorax(z):
    att = {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["dim"],
           "scale": z["dim"] ** -0.5, "mask": {"size": z["window"]},
           "rot": {"base": 10000.0, "dims": z["dim"] // 2}}
    n = z["d_heads"]
    ret = {"heads": n, "dim": z["d_dim"], "vdim": z["d_dim"],
           "decay": [1.0 - 2.0 ** (-5.0 - 6.0 * h / max(1, n - 1)) for h in range(n)],
           "rot": {"base": 500000.0, "dims": z["d_dim"]}}
    kinds = {"attention": att, "retention": ret}
    order = (["retention", "attention", "attention", "retention"] * 2)[:LAYERS - 2]
    return {"architecture": "Virorax", "norm": {"eps": 1e-6}, "residual_mult": 0.6,
            "logit_softcap": 30.0, "loop": {"start": 2, "stop": 4, "times": 2},
            "layers": [{"type": k, "mixer": kinds[k], "mlp": {"kind": "dense", "ff": z["ff"]}}
                       for k in order]}


def _mipurax(z):
    rot = 32
    latent = {"heads": z["heads"], "dim": z["dim"], "rot_dim": rot, "vdim": z["dim"],
              "kv_rank": z["rank"] - rot, "q_rank": 3 * z["width"] // 8,
              "scale": (z["dim"] + rot) ** -0.5, "rot": {"base": 500000.0, "dims": rot}}
    att = {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["dim"],
           "scale": z["dim"] ** -0.5, "mask": {"size": z["window"]}}
    mlp = _moe(z, groups={"count": z["experts"] // 4, "keep": z["experts"] // 8})
    mlp["shared"] = {"ff": z["expert_ff"]}
    layers = []
    for i in range(LAYERS):
        kind = ["latent_attention", "attention", "latent_attention_2", "reader"][i % 4]
        mixer = dict(att, kv_from=i - 2) if kind == "reader" else att if kind == "attention" \
            else latent
        layers.append({"type": "attention" if kind == "reader" else kind, "mixer": mixer,
                       "mlp": mlp})
    return {"architecture": "Mipurax", "norm": {"eps": 1e-6}, "layers": layers}


def _gibipel(z):
    left = {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["dim"],
            "scale": z["dim"] ** -0.5, "mask": {"size": z["window"], "pool": 16},
            "rot": {"base": 500000.0, "dims": z["dim"],
                    "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 1024}}}
    right = {"heads": z["d_heads"], "dim": z["d_dim"], "vdim": z["d_dim"], "gate_cap": 15.0}
    same = z["experts"] // 8
    mlp = _moe(z, identity=same, groups={"count": z["experts"] // 4, "keep": z["experts"] // 8})
    mlp["router"]["experts"] = z["experts"] - same
    mlp["shared"] = {"ff": z["expert_ff"]}
    mixer = {"left": left, "right": right, "left_scale": 0.8, "right_scale": 1.1}
    return {"architecture": "Gibipel", "norm": {"eps": 1e-6}, "logit_scale": 0.5,
            "embedding": {"scale": z["width"] ** 0.5},
            "layers": [{"type": "parallel", "mixer": mixer, "mlp": mlp}] * LAYERS}


def _pudorax(z):
    inner = z["d_heads"] * z["d_dim"]
    att = {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["dim"],
           "scale": z["dim"] ** -0.5, "conv": 4, "rot": {"base": 250000.0, "dims": z["dim"] // 2}}
    ssm = {"heads": inner // 64, "vdim": 64, "state": z["d_dim"], "groups": z["ssm_groups"],
           "norm_groups": z["ssm_groups"], "conv": 4}
    mlp = _moe(z)
    mlp["expert"]["limit"] = 7.0
    mlp["shared"] = {"ff": z["expert_ff"], "limit": 7.0}
    kinds = {"attention": att, "mamba2": ssm}
    order = ["mamba2", "mamba2", "mamba2", "attention"] * (LAYERS // 4)
    return {"architecture": "Pudorax", "norm": {"eps": 1e-5}, "embedding": {"scale": 3.0},
            "logit_softcap": 30.0, "token_side": {"dim": 128},
            "loop": {"start": LAYERS // 2, "stop": LAYERS, "times": 2},
            "layers": [{"type": k, "mixer": kinds[k], "mlp": mlp} for k in order]}


DESIGNS = {"rigozen": _rigozen, "losorax": _losorax, "virorax": _virorax, "mipurax": _mipurax,
           "gibipel": _gibipel, "pudorax": _pudorax}
LLAMAS = ("smollm2-135m", "smollm2-360m", "smollm2-1.7b")


def config_of(model: str) -> dict:
    """config.json of a model name: a preset's, or "<design>-<size>"."""
    if model in LLAMAS:
        from cretif_b200.config.presets import preset
        return preset(model)
    design, size = model.rsplit("-", 1)
    z = SIZES[size]
    return {**DESIGNS[design](z), "vocab": VOCAB, "width": z["width"],
            "max_positions": MAX_POSITIONS}


def _manifest(cfg):
    from cretif_b200.config.registry import architecture_name, resolve_architecture
    from cretif_b200.engine.model import manifest
    arch = resolve_architecture(architecture_name(cfg))
    return manifest(arch.build_spec(arch.config_from_dict(cfg)))[0]


# How strongly a token's own experts stand in its embedding, and the router's gain, by design.
ROUTING = {"losorax": (5.0, 0.4), "mipurax": (0.25, 0.6), "gibipel": (1.0, None),
           "pudorax": (8.0, 0.3)}


def _route_by_token(model, cfg, out, gen):
    """Routers that a token's identity decides, as trained ones do: every router output has a
    direction, a token's embedding holds those of its experts (spread over groups, where experts
    are grouped), the routers' rows are the directions.  With routers of independent random rows
    every eighth choice or so is a near tie, and two correct implementations in 16 bits differ by
    whole experts."""
    design, (strength, gain) = model.rsplit("-", 1)[0], ROUTING[model.rsplit("-", 1)[0]]
    r, D = cfg["layers"][0]["mlp"]["router"], cfg["width"]
    n, top = r["experts"] + r.get("identity", 0), r["top"]
    count, keep = (r["groups"]["count"], r["groups"]["keep"]) if "groups" in r else (1, 1)
    gain = gain or D ** -0.5
    rows = torch.randn(n, D, device="cuda", generator=gen) * D ** -0.5
    kept = torch.rand(VOCAB, count, device="cuda", generator=gen).argsort(1)[:, :keep]
    inside = torch.rand(VOCAB, count, n // count, device="cuda", generator=gen).argsort(2)
    embed, every = out["embed"].float(), torch.arange(VOCAB, device="cuda")
    for j in range(top):
        g = kept[:, j % keep]
        e = g * (n // count) + inside[every, g, j // keep]
        embed += strength * (1.0 + 0.5 * (top - 1 - j)) * rows[e]
    out["embed"] = embed.to(out["embed"].dtype)
    for i in range(len(cfg["layers"])):
        at = rows
        if design == "pudorax" and i >= cfg["loop"]["start"]:
            # the input reaches these layers through the merging matrix
            at = rows @ out["loop.in"][:, D:].float().T
            at = at / at.norm(dim=1, keepdim=True)
        p = "l%d.mlp." % i
        out[p + "router"] = (gain * at).to(out[p + "router"].dtype)
        for name, scale in ((p + "router.b", 0.2), (p + "correction", 0.1)):
            if name in out:                     # a trained router's balancing terms are small
                out[name] = (scale * out[name].float()).to(out[name].dtype)


def weights_of(model: str, dtype: str) -> Dict[str, torch.Tensor]:
    """Random weights in the distributions the model's parts declare, the same ones every time."""
    stored = torch.bfloat16 if dtype == "bfloat16" else torch.float32
    out = {}
    for name, spec in _manifest(config_of(model)).items():
        gen = torch.Generator(device="cuda")
        gen.manual_seed(zlib.crc32(name.encode()))
        mean, std = spec.init
        t = torch.empty(spec.shape, dtype=torch.float32, device="cuda")
        out[name] = t.normal_(mean, std, generator=gen).to(stored)
    if model.rsplit("-", 1)[0] in ROUTING:
        _route_by_token(model, config_of(model), out, torch.Generator("cuda").manual_seed(5))
    return out


_LOADED: dict = {}


def _engine(case):
    """The engine a program has loaded; the last model asked for is kept."""
    import cretif_b200
    from cretif_b200.weights.loader import write_model_folder
    room = -(-(case["longest"] + case["steps"] + 64) // 64) * 64 * case["batch"]
    key = (case["model"], case["dtype"])
    if key in _LOADED and _LOADED[key].cache.max_tokens >= room \
            and _LOADED[key].cache.max_slots >= case["batch"]:
        return _LOADED[key]
    _LOADED.clear()
    torch.cuda.empty_cache()
    folder = tempfile.mkdtemp(prefix="cases_")
    try:
        write_model_folder(folder, config_of(case["model"]), {
            k: v.cpu() for k, v in weights_of(case["model"], case["dtype"]).items()})
        _LOADED[key] = cretif_b200.load(folder, dtype=case["dtype"], max_tokens=room,
                                        max_len=MAX_POSITIONS, max_slots=max(16, case["batch"]))
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    return _LOADED[key]


# ------------------------------------------------------------------------------------------
# cases
# ------------------------------------------------------------------------------------------
def _case(model, batch, shortest, longest, steps, dtype="bfloat16", use="replay", name=None):
    c = {"model": model, "dtype": dtype, "batch": batch, "shortest": shortest,
         "longest": longest, "steps": steps, "use": use}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one chat turn on the smallest model: a short prompt, then token after token
        _case("smollm2-135m", 1, 61, 61, 40, name="135m chat b1"),
        # eight long conversations decoding side by side, the benchmark's batch and context
        _case("smollm2-135m", 8, 2048, 2048, 32, name="135m long b8"),
        # one document scored: a lone prompt step of an odd length, no decoding
        _case("smollm2-135m", 1, 2047, 2047, 0, name="135m score b1"),
        # a server's batch of unequal requests
        _case("smollm2-360m", 64, 256, 2048, 12, name="360m serve b64"),
        # the largest model, half prompt and half decoding
        _case("smollm2-1.7b", 8, 1024, 1024, 24, name="1.7b b8"),
        # the true 32-bit path: greedy generation, then its tokens scored
        _case("smollm2-135m", 3, 90, 300, 8, dtype="float32", use="generate",
              name="135m fp32 generate b3"),
        # the other architectures' mixed models
        _case("rigozen-m", 1, 2048, 2048, 8, name="rigozen m b1"),
        _case("losorax-m", 4, 300, 1500, 8, name="losorax m b4"),
        _case("virorax-s", 8, 777, 777, 16, name="virorax s b8"),
        _case("mipurax-m", 2, 1300, 1300, 16, name="mipurax m b2"),
        _case("gibipel-s", 1, 1601, 1601, 16, name="gibipel s b1"),
        _case("pudorax-m", 8, 200, 700, 8, name="pudorax m b8"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Any model at any batch its listed cases stand for; lengths and steps over their range."""
    steps = rng.choice([0, _log_int(rng, 1, 40), _log_int(rng, 1, 40)])
    longest = _log_int(rng, 16, 2048)
    shortest = longest if rng.random() < 0.5 else max(8, longest // rng.randint(2, 8))
    kind = rng.random()
    if kind < 0.4:
        model = rng.choice(LLAMAS)
        most = {"smollm2-135m": 64, "smollm2-360m": 48, "smollm2-1.7b": 8}[model]
        batch = min(_log_int(rng, 1, most), max(1, 65536 // longest))
        return _case(model, batch, shortest, longest, steps)
    if kind < 0.5:
        longest = min(longest, 400)
        return _case("smollm2-135m", rng.randint(1, 4), min(shortest, longest), longest,
                     max(1, steps // 4), dtype="float32", use="generate")
    model = "%s-%s" % (rng.choice(sorted(DESIGNS)), rng.choice(sorted(SIZES)))
    batch = min(_log_int(rng, 1, 16), max(1, 8192 // longest))
    return _case(model, batch, shortest, longest, min(steps, 20))


def lengths_of(case) -> List[int]:
    a, b, n = case["shortest"], case["longest"], case["batch"]
    if n == 1:
        return [b]
    return [int(round(a * (b / a) ** (i / (n - 1)))) for i in range(n)]


def _tokens(case, seed):
    """(prompts, tokens fed in the decode steps [batch][steps]), uniform ids."""
    rng = np.random.default_rng(seed)
    prompts = [rng.integers(0, VOCAB, size=n).tolist() for n in lengths_of(case)]
    return prompts, rng.integers(0, VOCAB, size=(case["batch"], case["steps"])).tolist()


def prepare(case, seed):
    prompts, fed = _tokens(case, seed)
    return {"engine": _engine(case), "prompts": prompts, "fed": fed, "steps": case["steps"],
            "use": case["use"]}


def run(state):
    engine, prompts = state["engine"], state["prompts"]
    if state["use"] == "generate":
        made = [r.tokens for r in engine.generate(prompts, max_tokens=state["steps"],
                                                  stop_ids=[])]
        texts = [p + t for p, t in zip(prompts, made)]
        want = [range(len(p) - 1, len(x) - 1) for p, x in zip(prompts, texts)]
    else:
        made, texts, want = None, prompts, "last"
    slots = [engine.alloc_slot() for _ in texts]
    try:
        logits = [engine.step(list(zip(slots, texts)), want, check=False)]
        if made is not None:
            return {"tokens": np.asarray(made), "logits": logits}
        for t in range(state["steps"]):
            logits.append(engine.step([(s, row[t:t + 1]) for s, row in zip(slots, state["fed"])],
                                      check=False))
    finally:
        for s in slots:
            engine.free_slot(s)
    return {"logits": logits}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def _runs(cfg) -> List[int]:
    """The layers in the order they run (a repeated span several times)."""
    n = len(cfg["layers"])
    loop = cfg.get("loop") or {"start": 0, "stop": n, "times": 1}
    span = list(range(loop["start"], loop["stop"]))
    return list(range(loop["start"])) + span * loop["times"] + list(range(loop["stop"], n))


def _mixers(layer):
    m = layer["mixer"]
    return [("attention", m["left"]), ("memory", m["right"])] if layer["type"] == "parallel" \
        else [(layer["type"], m)]


def work(case):
    """Every matrix a step multiplies by read once a step (of the experts those its tokens can
    use), keys, values and states of the live sequences read in every decode step, logits written;
    two operations a weight and token, and the attention's and the recurrences' products."""
    cfg, size = config_of(case["model"]), 2 if case["dtype"] == "bfloat16" else 4
    n_params = {k: math.prod(s.shape) for k, s in _manifest(cfg).items()}
    if case["model"] in LLAMAS:
        L, H, d = cfg["num_hidden_layers"], cfg["num_attention_heads"], cfg["head_dim"]
        layers = [("attention", {"heads": H, "kv_heads": cfg["num_key_value_heads"], "dim": d,
                                 "vdim": d})] * L
        runs, width = [n_params_of(n_params, "model.layers.%d." % i) for i in range(L)], \
            cfg["hidden_size"]
        moes = []
    else:
        order = _runs(cfg)
        layers = [m for i in order for m in _mixers(cfg["layers"][i])]
        runs, width = [n_params_of(n_params, "l%d." % i) for i in order], cfg["width"]
        moes = [cfg["layers"][i]["mlp"] for i in order if cfg["layers"][i]["mlp"]["kind"] == "moe"]
    mats = 2 if cfg.get("architecture") == "Mipurax" else 3
    expert = [mats * width * m["expert"]["ff"] for m in moes]
    every = sum(e * m["router"]["experts"] for e, m in zip(expert, moes))
    base, head = sum(runs) - every, VOCAB * width
    lens, K, B = lengths_of(case), case["steps"], case["batch"]
    if case["use"] == "generate":
        made, lens, K = lens, lens + [n + K for n in lens], K - 1
    T = sum(lens)

    def experts(tokens):
        return sum(e * min(m["router"]["experts"], tokens * m["router"]["top"])
                   for e, m in zip(expert, moes))

    def seen(n, m):                       # keys that query n of a sequence reads
        return min(n, (m.get("mask") or {}).get("size", n))
    flops = nbytes = 0.0
    active = base + sum(e * m["router"]["top"] for e, m in zip(expert, moes))
    flops += 2.0 * active * (T + B * K) + 2.0 * head * B * (1 + K)
    nbytes += size * (base + experts(T) + head + K * (base + experts(B) + head))
    nbytes += 4.0 * VOCAB * B * (1 + K)
    for kind, m in layers:
        for n in lens:
            if "attention" in kind:
                w = (m.get("mask") or {}).get("size", n)
                pairs = n * (n + 1) / 2 - max(0, n - w) * (n - w + 1) / 2
                flops += 2.0 * pairs * m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"])
            else:
                flops += 4.0 * n * m["heads"] * m.get("state", m.get("dim")) \
                    * m.get("vdim", m.get("dim"))
        for t in range(K):
            for n in lens[:B]:
                if "attention" in kind:
                    kept = m.get("kv_rank", 0) + m.get("rot_dim", 0) if "kv_rank" in m \
                        else m["kv_heads"] * (m["dim"] + m["vdim"])
                    nbytes += size * kept * seen(n + t + 1, m)
                else:
                    nbytes += 8.0 * m["heads"] * m.get("state", m.get("dim")) \
                        * m.get("vdim", m.get("dim"))
    return {"bytes": nbytes, "flops": flops}


def n_params_of(n_params, prefix):
    return sum(n for k, n in n_params.items() if k.startswith(prefix))


def tolerance(case):
    """About four times what the outputs are off the 64-bit ones (bfloat16: 0.007 to 0.025, by
    depth; 0.0025 and less where bounded norms or the embedding's share in the logits hide the
    layers' roundings; float32: 4e-7, and a greedy token may change at a near tie)."""
    if case["dtype"] == "float32":
        return {"rel": 2e-6, "max": 5e-5, "differ": 0.01}
    rel = {"losorax": 0.012, "mipurax": 0.006}.get(case["model"].rsplit("-", 1)[0], 0.03)
    return {"rel": rel, "max": 10 * rel}


# ------------------------------------------------------------------------------------------
# the same in 64 bits, elementary torch
# ------------------------------------------------------------------------------------------
def _unit(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _rotate(z, freq, pairs="half"):
    """z [S, heads, d]; the first 2 * len(freq) channels of a head turn, pair i by p * freq[i]."""
    half = len(freq)
    ang = torch.arange(z.shape[0], dtype=z.dtype, device=z.device)[:, None] * freq
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    out = z.clone()
    a, b = (slice(0, half), slice(half, 2 * half)) if pairs == "half" \
        else (slice(0, 2 * half, 2), slice(1, 2 * half, 2))
    u, v = z[..., a], z[..., b]
    out[..., a], out[..., b] = u * c - v * s, v * c + u * s
    return out


def _freq(base, dims, scaling=None):
    f = float(base) ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)
    if scaling:                     # long wavelengths stretched, a blend between
        r = scaling["original"] * f / (2.0 * math.pi)
        t = ((r - scaling["low"]) / (scaling["high"] - scaling["low"])).clamp(0.0, 1.0)
        f = (1.0 - t) * f / scaling["factor"] + t * f
    return f


def _conv(z, taps):
    K = taps.shape[1]
    padded = torch.cat([z.new_zeros(K - 1, z.shape[1]), z])
    return sum(padded[j:j + z.shape[0]] * taps[:, j] for j in range(K))


def _distance(S):
    i = torch.arange(S, device="cuda")
    return i[:, None] - i[None, :]


def _attend(q, k, v, scale, visible, bias=None, sink=None):
    """q [S, H, d], k [N, G, d], v [N, G, e] -> [S, H, e]; ``sink`` [H]: a term exp(sink) of the
    denominator; ``bias`` a function of the head."""
    H, G = q.shape[1], k.shape[1]
    out = q.new_empty(q.shape[0], H, v.shape[2])
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[:, g].T) * scale
        if bias is not None:
            s += bias(h)
        s.masked_fill_(~visible, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
        p = torch.softmax(s, -1)
        out[:, h] = (p if sink is None else p[:, :-1]) @ v[:, g]
    return out


def _experts(x, chosen, weights, ff):
    """Sum over a token's chosen experts; chosen, weights [S, top]; ff(e, rows, weights)."""
    out = torch.zeros_like(x)
    for e in torch.unique(chosen).tolist():
        at, slot = torch.nonzero(chosen == e, as_tuple=True)
        out.index_add_(0, at, ff(e, x[at], weights[at, slot][:, None]))
    return out


def _best_groups(score, groups, of_group):
    """score with the outputs outside the best groups at -inf."""
    if not groups or groups["count"] <= 1:
        return score
    s = score.view(score.shape[0], groups["count"], -1)
    kept = of_group(s).topk(groups["keep"], -1).indices
    ok = torch.zeros(s.shape[:2], dtype=torch.bool, device=s.device).scatter_(1, kept, True)
    return s.masked_fill(~ok[:, :, None], -math.inf).reshape(score.shape)


class _Plain:
    """A model in float64: whole sequences, no cache."""

    def __init__(self, case):
        self.cfg = config_of(case["model"])
        # matrices are widened where they are used
        self.raw = weights_of(case["model"], case["dtype"])
        self.eps = self.cfg["rms_norm_eps"] if case["model"] in LLAMAS else self.cfg["norm"]["eps"]
        self.forward = getattr(self, "llama" if case["model"] in LLAMAS
                               else case["model"].rsplit("-", 1)[0])

    def w(self, name):
        return self.raw[name].double()

    def lin(self, x, name):
        return x @ self.w(name).T

    def heads(self, x, name, n):
        return self.lin(x, name).view(x.shape[0], n, -1)

    def swiglu(self, x, p):
        return self.lin(_silu(self.lin(x, p + "gate")) * self.lin(x, p + "up"), p + "down")

    # -- Llama: every sequence's rows through the matrices at once --
    def llama(self, seqs, rows):
        c, eps = self.cfg, self.eps
        H, G, d = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        freq = _freq(c["rope_theta"], d)
        cu = np.cumsum([0] + [len(s) for s in seqs])
        E = self.raw["model.embed_tokens.weight"]
        x = E[torch.tensor([t for s in seqs for t in s], device="cuda")].double()
        for i in range(c["num_hidden_layers"]):
            p = "model.layers.%d." % i
            n = _unit(x, eps) * self.w(p + "input_layernorm.weight")
            q, k, v = (self.heads(n, p + "self_attn.%s_proj.weight" % a, m)
                       for a, m in zip("qkv", (H, G, G)))
            o = torch.empty_like(q)
            for a, b in zip(cu, cu[1:]):
                o[a:b] = self.causal(_rotate(q[a:b], freq), _rotate(k[a:b], freq), v[a:b])
            x = x + self.lin(o.reshape(len(x), -1), p + "self_attn.o_proj.weight")
            n = _unit(x, eps) * self.w(p + "post_attention_layernorm.weight")
            y = _silu(self.lin(n, p + "mlp.gate_proj.weight")) \
                * self.lin(n, p + "mlp.up_proj.weight")
            x = x + self.lin(y, p + "mlp.down_proj.weight")
        at = torch.tensor([a + r for a, rr in zip(cu, rows) for r in rr], device="cuda")
        out = (_unit(x[at], eps) * self.w("model.norm.weight")) @ E.double().T
        return list(out.split([len(r) for r in rows]))

    @staticmethod
    def causal(q, k, v):
        S, H, d = q.shape
        G = k.shape[1]
        q = q.view(S, G, H // G, d).permute(1, 2, 0, 3).reshape(G, -1, d)
        s = (q @ k.permute(1, 2, 0)).view(H, S, S) * d ** -0.5
        s.masked_fill_(_distance(S) < 0, -math.inf)
        o = torch.softmax(s, -1).view(G, -1, S) @ v.transpose(0, 1)
        return o.view(H, S, -1).transpose(0, 1)

    def each(self, seqs, rows, stream, last):
        """Sequences one by one: the stream after the layers, then the wanted rows' logits."""
        return [last(stream(torch.tensor(s, device="cuda"))[torch.tensor(r, device="cuda")])
                for s, r in zip(seqs, rows)]

    # -- Rigozen --
    def rigozen(self, seqs, rows):
        eps = self.eps

        def around(x, name):
            return _unit(x, eps) * (1.0 + self.w(name))

        def attention(x, p, m):
            S, G, d = len(x), m["kv_heads"], m["dim"]
            q = _unit(self.lin(x, p + "q"), eps) * self.w(p + "q.norm")
            k = self.lin(x, p + "k")
            kn = _unit(k, eps) * self.w(p + "k.norm")
            n = _distance(S)
            return _attend(q.view(S, -1, d), kn.view(S, G, d), k.view(S, G, d), m["scale"],
                           (n >= 0) & (n < m["mask"]["size"]))

        def latent_attention(x, p, m):
            S, H = len(x), m["heads"]
            c = _unit(self.lin(x, p + "dkv"), eps) * self.w(p + "dkv.norm")
            n = _distance(S)
            return _attend(self.heads(x, p + "q", H), self.heads(c, p + "uk", H),
                           self.heads(c, p + "uv", H), m["scale"],
                           (n >= 0) & (n < m["mask"]["size"]), sink=self.w(p + "sink"))

        def delta(x, p, m):
            S, G, d = len(x), m["kv_heads"], m["dim"]
            q, k, v = (_silu(_conv(self.lin(x, p + n), self.w(p + n + ".conv"))) for n in "qkv")
            q, k = q.view(S, G, d), k.view(S, G, d)
            q = q * torch.rsqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
            k = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            rep = m["heads"] // G
            q, k = q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1)
            v = v.view(S, m["heads"], -1)
            beta = torch.sigmoid(self.lin(x, p + "b"))
            decay = torch.exp(-torch.exp(self.w(p + "A_log")) * torch.nn.functional.softplus(
                self.lin(x, p + "a") + self.w(p + "dt_bias")))
            M = x.new_zeros(m["heads"], d, v.shape[2])
            o = torch.empty_like(v)
            for t in range(S):
                M = M * decay[t, :, None, None]
                u = beta[t, :, None] * (v[t] - torch.einsum("hde,hd->he", M, k[t]))
                M = M + k[t, :, :, None] * u[:, None, :]
                o[t] = torch.einsum("hde,hd->he", M, q[t])
            return _unit(o, eps) * self.w(p + "norm") * _silu(self.lin(x, p + "g")).view(o.shape)

        mixers = {"attention": attention, "latent_attention": latent_attention, "delta": delta}

        def stream(ids):
            x = self.raw["embed"][ids].double()
            for i, layer in enumerate(self.cfg["layers"]):
                p = "l%d." % i
                o = mixers[layer["type"]](x, p + "mix.", layer["mixer"])
                x = x + around(self.lin(o.reshape(len(x), -1), p + "mix.o"), p + "norm1")
                x = x + around(self.swiglu(x, p + "mlp."), p + "norm2")
            return x
        return self.each(seqs, rows, stream, lambda x: self.lin(around(x, "final.norm"), "embed"))

    # -- Losorax --
    def losorax(self, seqs, rows):
        eps = self.eps

        def dyt(x, name):
            return torch.tanh(self.w(name + ".alpha") * x) * self.w(name) + self.w(name + ".b")

        def attention(x, p, m, kv):
            S, G, d = len(x), m["kv_heads"], m["dim"]
            q = _unit(_conv(self.lin(x, p + "q"), self.w(p + "q.conv")).view(S, -1, d), eps)
            if kv is None:
                k, v = (_conv(self.lin(x, p + n), self.w(p + n + ".conv")).view(S, G, -1)
                        for n in "kv")
                kv = _unit(k, eps), v
            t = torch.arange(S, device="cuda")
            gain = 1.0 + m["q_temp"]["coef"] * torch.log((t + 1) // m["q_temp"]["every"] + 1.0)
            rel, n = self.w(p + "rel"), _distance(S)
            R, half = rel.shape[0], rel.shape[0] // 2
            far = half + torch.floor(torch.log(t.clamp(min=1).double() / half)
                                     / math.log(m["bias_max"] / half) * (R - half)).long()
            bucket = torch.where(t < half, t, far.clamp(max=R - 1))
            o = _attend(q * gain.double()[:, None, None], kv[0], kv[1], m["scale"], n >= 0,
                        bias=lambda h: rel[:, h][bucket][n.clamp(min=0)],
                        sink=x.new_zeros(q.shape[1]))
            return o, kv

        def general_delta(x, p, m):
            S, H = len(x), m["heads"]
            r, k, v = (self.heads(x, p + n, H) for n in "rkv")
            w = torch.exp(-math.exp(-0.5) * torch.sigmoid(self.lin(torch.tanh(
                self.lin(x, p + "w1")), p + "w2") + self.w(p + "w0"))).view(r.shape)
            a = torch.sigmoid(self.lin(x, p + "a") + self.w(p + "a.b")).view(r.shape)
            u = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            M, o = x.new_zeros(H, r.shape[2], v.shape[2]), torch.empty_like(v)
            for t in range(S):
                uM = torch.einsum("hd,hde->he", u[t], M)
                M = w[t, :, :, None] * M - (a[t] * u[t])[:, :, None] * uM[:, None] \
                    + k[t, :, :, None] * v[t, :, None]
                o[t] = torch.einsum("hde,hd->he", M, r[t])
            return _unit(o, eps).view(S, -1) * self.w(p + "norm") * torch.sigmoid(
                self.lin(x, p + "g"))

        def routed(x, p, mlp):
            s = torch.sigmoid(self.lin(x, p + "router"))
            best = s.topk(mlp["router"]["top"], -1)
            return _experts(x, best.indices, best.values,
                            lambda e, rows, w: self.swiglu(w * rows, "%se%d." % (p, e)))

        def stream(ids):
            x, kept = self.raw["embed"][ids].double(), {}
            for i, layer in enumerate(self.cfg["layers"]):
                p, m = "l%d." % i, layer["mixer"]
                h = dyt(x, p + "norm1")
                h = h + (torch.cat([torch.zeros_like(h[:1]), h[:-1]]) - h) * self.w(p + "shift")
                if layer["type"] == "attention":
                    o, kept[i] = attention(h, p + "mix.", m, kept.get(m.get("kv_from")))
                else:
                    o = general_delta(h, p + "mix.", m)
                y = self.lin(o.reshape(len(x), -1), p + "mix.o")
                x = x + self.w(p + "ls1") * dyt(y, p + "norm1b")
                y = routed(dyt(x, p + "norm2"), p + "mlp.", layer["mlp"])
                x = x + self.w(p + "ls2") * dyt(y, p + "norm2b")
            return x
        return self.each(seqs, rows, stream, lambda x: self.lin(dyt(x, "final.norm"), "head"))

    # -- Virorax --
    def virorax(self, seqs, rows):
        eps, mult, cap = self.eps, self.cfg["residual_mult"], self.cfg["logit_softcap"]

        def attention(x, p, m):
            S, n = len(x), _distance(len(x))
            q, k, v = ((self.lin(x, p + a) + self.w(p + a + ".b")).view(S, c, -1) for a, c in
                       zip("qkv", (m["heads"], m["kv_heads"], m["kv_heads"])))
            f = _freq(m["rot"]["base"], m["rot"]["dims"])
            q, k = (_rotate(_unit(z, eps) * self.w(p + a + ".norm"), f)
                    for a, z in (("q", q), ("k", k)))
            o = _attend(q, k, v, m["scale"], (n >= 0) & (n < m["mask"]["size"]),
                        sink=self.w(p + "sink"))
            return (o * torch.sigmoid(self.lin(x, p + "g"))[:, :, None]).reshape(S, -1)

        def retention(x, p, m):
            S, H, d = len(x), m["heads"], m["dim"]
            f = _freq(m["rot"]["base"], m["rot"]["dims"])
            q, k = (_rotate(self.heads(x, p + a, H), f) for a in "qk")
            v, n = self.heads(x, p + "v", H), _distance(S)
            o = torch.empty_like(v)
            for h in range(H):
                far = torch.pow(x.new_tensor(m["decay"][h]), n.clamp(min=0)) * (n >= 0)
                o[:, h] = ((q[:, h] @ k[:, h].T) * d ** -0.5 * far) @ v[:, h]
            return _unit(o, eps).reshape(S, -1) * _silu(self.lin(x, p + "g"))

        mixers = {"attention": attention, "retention": retention}

        def stream(ids):
            x = self.raw["embed"][ids].double() + self.raw["pos"][:len(ids)].double()
            x0, before = x, set()
            for i in _runs(self.cfg):
                p, layer = "l%d." % i, self.cfg["layers"][i]
                if i == self.cfg["loop"]["start"] and i in before:
                    x = x + x0
                before.add(i)
                o = mixers[layer["type"]](_unit(x, eps) * self.w(p + "norm1"), p + "mix.",
                                          layer["mixer"])
                x = x + mult * self.lin(o, p + "mix.o")
                y = self.lin(_unit(x, eps) * self.w(p + "norm2"), p + "mlp.up")
                x = x + mult * self.lin(y.clamp(min=0.0) ** 2, p + "mlp.down")
            return x
        return self.each(seqs, rows, stream, lambda x: cap * torch.tanh(self.lin(
            _unit(x, eps) * self.w("final.norm"), "embed") / cap))

    # -- Mipurax --
    def mipurax(self, seqs, rows):
        eps = self.eps

        def around(x, name):
            return _unit(x, eps) * (1.0 + self.w(name))

        def ff(x, p):
            return self.lin(torch.nn.functional.gelu(self.lin(x, p + "up")), p + "down")

        def latent(x, p, m, first):
            S, H, d, rank = len(x), m["heads"], m["dim"], m["kv_rank"]
            f, pairs = _freq(m["rot"]["base"], m["rot"]["dims"]), "pairs" if first else "half"
            cq = _unit(self.lin(x, p + "dq"), eps) * self.w(p + "dq.norm")
            q = self.heads(cq, p + "uq", H)
            q = torch.cat([q[..., :d], _rotate(q[..., d:], f, pairs)], -1)
            ckr = self.lin(x, p + "dkv")
            c = _unit(ckr[:, :rank], eps) * self.w(p + "dkv.norm")
            kr = _rotate(ckr[:, None, rank:], f, pairs)
            k = torch.cat([self.heads(c, p + "uk", H), kr.expand(S, H, -1)], -1)
            o = _attend(q, k, self.heads(c, p + "uv", H), m["scale"], _distance(S) >= 0,
                        sink=None if first else self.w(p + "sink"))
            g = torch.sigmoid(self.lin(x, p + "g"))
            return (o * (g.view(o.shape) if first else g[:, :, None])).reshape(S, -1)

        def chunked(x, p, m, kv):
            S, H = len(x), m["heads"]
            if kv is None:
                kv = tuple(self.heads(x, p + a, m["kv_heads"]) for a in "kv")
            n, run = _distance(S), torch.arange(S, device="cuda") // m["mask"]["size"]
            o = _attend(self.heads(x, p + "q", H), kv[0], kv[1], m["scale"],
                        (n >= 0) & (run[:, None] == run[None, :]),
                        bias=lambda h: -(2.0 ** (-8.0 * (h + 1) / H)) * n)
            return o.reshape(S, -1), kv

        def routed(x, p, mlp):
            s = torch.sigmoid(self.lin(x, p + "router"))
            per = s.shape[1] // mlp["router"]["groups"]["count"]
            at = _best_groups(s, mlp["router"]["groups"],
                              lambda g: g.topk(min(2, per), -1).values.sum(-1)
                              ).topk(mlp["router"]["top"], -1).indices
            w = s.gather(1, at)
            w = w / (w.sum(-1, keepdim=True) + 1e-20)
            return ff(x, p + "shared.") + _experts(
                x, at, w, lambda e, rows, a: a * ff(rows, "%se%d." % (p, e)))

        def stream(ids):
            x, kept = around(self.raw["embed"][ids].double(), "embed.norm"), {}
            for i, layer in enumerate(self.cfg["layers"]):
                p, m, kind = "l%d." % i, layer["mixer"], layer["type"]
                h = around(x, p + "norm1")
                if kind == "attention":
                    o, kept[i] = chunked(h, p + "mix.", m, kept.get(m.get("kv_from")))
                else:
                    o = latent(h, p + "mix.", m, kind == "latent_attention")
                x = x + self.lin(o, p + "mix.o")
                x = x + routed(around(x, p + "norm2"), p + "mlp.", layer["mlp"])
            return x
        return self.each(seqs, rows, stream, lambda x: self.lin(around(x, "final.norm"), "embed"))

    # -- Gibipel --
    def gibipel(self, seqs, rows):
        eps = self.eps

        def attention(x, p, m):
            S, P, size = len(x), m["mask"]["pool"], m["mask"]["size"]
            q, k, v = (self.lin(x, p + a) + self.w(p + a + ".b") for a in "qkv")
            f = _freq(m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"])
            q = _rotate((_unit(q, eps) * self.w(p + "q.norm")).view(S, m["heads"], -1), f)
            k = _rotate((_unit(k, eps) * self.w(p + "k.norm")).view(S, m["kv_heads"], -1), f)
            v = v.view(S, m["kv_heads"], -1)
            k, v = (torch.cat([z, z[:S // P * P].view(-1, P, *z.shape[1:]).mean(1)])
                    for z in (k, v))
            n = _distance(S)
            last = torch.arange(S // P, device="cuda") * P + P - 1
            seen = torch.cat([(n >= 0) & (n < size), last[None] <= torch.arange(
                S, device="cuda")[:, None] - size], 1)
            return self.lin(_attend(q, k, v, m["scale"], seen, sink=self.w(p + "sink")
                                    ).reshape(S, -1), p + "o")

        def memory(x, p, m):
            S, H, cap = len(x), m["heads"], m["gate_cap"]
            q, k, v = (self.heads(x, p + a, H) for a in "qkv")
            q = q * m["dim"] ** -0.5
            i, f = (cap * torch.tanh((self.lin(x, p + a) + self.w(p + a + ".b")) / cap)
                    for a in "if")
            f = torch.nn.functional.logsigmoid(f)
            # the weight of token s in token t, all logarithms: the running maximum cancels
            F = f.cumsum(0)
            D = (F[:, None] - F[None] + i[None]).masked_fill((_distance(S) < 0)[:, :, None],
                                                             -math.inf)
            top = torch.maximum(D.max(1).values, F)                       # [S, H]
            o = torch.empty_like(v)
            for h in range(H):
                a = (q[:, h] @ k[:, h].T) * torch.exp(D[:, :, h] - top[:, h, None])
                den = torch.maximum(a.sum(1).abs(), torch.exp(-top[:, h])) + 1e-6
                o[:, h] = a @ v[:, h] / den[:, None]
            o = _unit(o, eps).reshape(S, -1) * self.w(p + "norm")
            return self.lin(o * torch.sigmoid(self.lin(x, p + "g")), p + "o")

        def routed(x, p, mlp):
            r = mlp["router"]
            s = torch.softmax(self.lin(x, p + "router"), -1)
            at = _best_groups(s + self.w(p + "correction"), r["groups"],
                              lambda g: g.max(-1).values).topk(r["top"], -1).indices
            w = s.gather(1, at)
            w = w / (w.sum(-1, keepdim=True) + 1e-20)
            return self.swiglu(x, p + "shared.") + _experts(
                x, at, w, lambda e, rows, a: a * (
                    self.swiglu(rows, "%se%d." % (p, e)) if e < r["experts"] else rows))

        def stream(ids):
            x = self.raw["embed"][ids].double() * self.cfg["embedding"]["scale"]
            for i, layer in enumerate(self.cfg["layers"]):
                p, m = "l%d." % i, layer["mixer"]
                y = m["left_scale"] * attention(x, p + "mix.left.", m["left"]) \
                    + m["right_scale"] * memory(x, p + "mix.right.", m["right"])
                x = x + _unit(y, eps) * self.w(p + "norm1")
                x = x + _unit(routed(x, p + "mlp.", layer["mlp"]), eps) * self.w(p + "norm2")
            return x
        return self.each(seqs, rows, stream, lambda x: self.cfg["logit_scale"] * self.lin(
            _unit(x, eps) * self.w("final.norm"), "head"))

    # -- Pudorax --
    def pudorax(self, seqs, rows):
        eps, cap = self.eps, self.cfg["logit_softcap"]

        def norm(x, name):
            return _unit(x - x.mean(-1, keepdim=True), eps) * self.w(name) + self.w(name + ".b")

        def attention(x, p, m):
            S = len(x)
            q, k, v = (_conv(self.lin(x, p + a), self.w(p + a + ".conv")) for a in "qkv")
            f = _freq(m["rot"]["base"], m["rot"]["dims"])
            q, k = (_rotate((_unit(z, eps) * self.w(p + a + ".norm")).view(S, c, -1), f, "pairs")
                    for a, z, c in (("q", q, m["heads"]), ("k", k, m["kv_heads"])))
            o = _attend(q, k, v.view(S, m["kv_heads"], -1), m["scale"], _distance(S) >= 0)
            return o.reshape(S, -1) * torch.sigmoid(self.lin(x, p + "g"))

        def mamba2(x, p, m):
            S, H, e, N, G = len(x), m["heads"], m["vdim"], m["state"], m["groups"]
            inner = H * e
            z, u, dt = self.lin(x, p + "in").split([inner, inner + 2 * G * N, H], 1)
            u = _silu(_conv(u, self.w(p + "conv")) + self.w(p + "conv.b"))
            xs, Bm, Cm = u.split([inner, G * N, G * N], 1)
            xs, Bm, Cm = xs.reshape(S, H, e), Bm.reshape(S, G, N), Cm.reshape(S, G, N)
            dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias"))
            F = (-torch.exp(self.w(p + "A_log")) * dt).cumsum(0)
            y, n = torch.empty_like(xs), _distance(S)
            for h in range(H):
                g = h // (H // G)
                far = torch.exp((F[:, None, h] - F[None, :, h]).masked_fill(n < 0, -math.inf))
                y[:, h] = ((Cm[:, g] @ Bm[:, g].T) * far * dt[None, :, h]) @ xs[:, h]
            y = (y + self.w(p + "D")[:, None] * xs).reshape(S, inner) * _silu(z)
            return _unit(y.view(S, m["norm_groups"], -1), eps).view(S, inner) * self.w(p + "norm")

        mixers = {"attention": attention, "mamba2": mamba2}

        def clamped(x, p, limit):
            g = self.lin(x, p + "gate").clamp(max=limit)
            u = self.lin(x, p + "up").clamp(-limit, limit)
            return self.lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), p + "down")

        def routed(x, p, mlp):
            best = (self.lin(x, p + "router") + self.w(p + "router.b")).topk(
                mlp["router"]["top"], -1)
            return clamped(x, p + "shared.", mlp["shared"]["limit"]) + _experts(
                x, best.indices, torch.softmax(best.values, -1),
                lambda e, rows, a: a * clamped(rows, "%se%d." % (p, e), mlp["expert"]["limit"]))

        def stream(ids):
            x = x0 = self.raw["embed"][ids].double() * self.cfg["embedding"]["scale"]
            dim = self.cfg["token_side"]["dim"]
            for i in _runs(self.cfg):
                p, layer = "l%d." % i, self.cfg["layers"][i]
                if i == self.cfg["loop"]["start"]:
                    x = self.lin(torch.cat([x, x0], 1), "loop.in")
                x = x + self.lin(mixers[layer["type"]](norm(x, p + "norm1"), p + "mix.",
                                                       layer["mixer"]), p + "mix.o")
                x = x + routed(norm(x, p + "norm2"), p + "mlp.", layer["mlp"])
                side = self.raw["side.embed"][ids, i * dim:(i + 1) * dim].double()
                y = torch.nn.functional.gelu(self.lin(x, p + "side.gate"),
                                             approximate="tanh") * side
                x = x + _unit(self.lin(y, p + "side.proj"), eps) * self.w(p + "side.norm")
            return x
        return self.each(seqs, rows, stream, lambda x: cap * torch.tanh(self.lin(
            norm(x, "final.norm"), "head") / cap))


@torch.no_grad()
def exact(case, seed):
    prompts, fed = _tokens(case, seed)
    _LOADED.clear()
    torch.cuda.empty_cache()
    plain, K = _Plain(case), case["steps"]
    if case["use"] == "generate":
        seqs, steps = [list(p) for p in prompts], []
        for _ in range(K):
            steps.append(torch.cat(plain.forward(seqs, [[len(s) - 1] for s in seqs])))
            for s, t in zip(seqs, steps[-1].argmax(-1).tolist()):
                s.append(t)
        made = [s[len(p):] for s, p in zip(seqs, prompts)]
        return {"tokens": np.asarray(made),
                "logits": [torch.stack(steps, 1).reshape(-1, VOCAB)]}
    rows = [list(range(len(p) - 1, len(p) + K)) for p in prompts]
    got = torch.stack(plain.forward([p + f for p, f in zip(prompts, fed)], rows), 1)
    return {"logits": list(got)}
