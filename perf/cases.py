"""The work the engine is measured on: steps of prompts, of decoded tokens and of both, and whole generations, through the
package's public entry points, over the model designs it serves.

A case names a model (``MODELS``: the shapes this repository's benchmark uses), a kind of pass and its sizes:

``prompt``    whole prompts in one step, logits at their last places, the requests finished: what a new request pays
``decode``    one token for each of ``requests`` live requests at about ``context`` positions: what every further token pays
``mixed``     a prompt and ``requests`` decoded tokens in one step: continuous batching
``generate``  ``Engine.generate`` on short prompts with sampling: scheduler, steps and sampler together

Weights and token ids are functions of the seed.  Matrices are N(0, 0.02) as an untrained model's (in the deep Qwen2 shapes the two
that write to the stream are smaller by the root of twice the layers, the usual start); decays, steps, gates and norms lie where
trained models have them.  Where a model routes tokens to experts, embeddings carry one of a few directions the routers
look for, so that experts are chosen by the token (as trained routers largely do) and not by rounding.
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

VOCAB = 32000
MODELS = {
    "qwen2-0.5b": dict(hidden=896, layers=24, heads=14, kv_heads=2, dim=64, ff=4864, vocab=151936, tied=True),
    "qwen2-0.5b-untied": dict(hidden=896, layers=24, heads=14, kv_heads=2, dim=64, ff=4864, vocab=151936, tied=False),
    "qwen2-7b": dict(hidden=3584, layers=28, heads=28, kv_heads=4, dim=128, ff=18944, vocab=152064, tied=False),
    "nunivik-2k": dict(width=2048, heads=16, kv_heads=4, window=1024, ff=8192, delta=16, states=64, groups=1),
    "nunivik-4k": dict(width=4096, heads=32, kv_heads=8, window=1024, ff=14336, delta=32, states=128, groups=8),
    "mirovik-2k": dict(width=2048, heads=16, kv_heads=4, retention=16, ff=8192, expert=2048, channels=4096, rank=128),
    "mirovik-4k": dict(width=4096, heads=32, kv_heads=8, retention=32, ff=14336, expert=3584, channels=8192, rank=256),
    "kudazen-2k": dict(width=2048, heads=16, kv_heads=4, chunk=1024, latent=16, wkv=32, ff=8192),
    "kudazen-4k": dict(width=4096, heads=32, kv_heads=8, chunk=2048, latent=32, wkv=64, ff=14336),
    "tobadra-2k": dict(width=2048, heads=16, kv_heads=4, window=1024, recurrent=16, ff=8192, expert=2048),
    "tobadra-4k": dict(width=4096, heads=32, kv_heads=8, window=2048, recurrent=32, ff=14336, expert=3584),
    "zurevik-2k": dict(width=2048, heads=16, kv_heads=4, window=1024, expert=2048),
    "zurevik-4k": dict(width=4096, heads=32, kv_heads=8, window=2048, expert=3584),
    "biropel-2k": dict(width=2048, heads=16, kv_heads=4, window=1024, recurrent=16, ff=8192),
    "biropel-4k": dict(width=4096, heads=32, kv_heads=8, window=2048, recurrent=32, ff=14336),
}
EXPERTS, CHOSEN = 16, 2
MORE_TOKENS = {"decode": 4096, "mixed": 4096}  # positions a live request may grow by before its conversation starts again


# ------------------------------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    return [
        # one user's next token on the smallest shape: launches and latency
        _case("one token 0.5B", "qwen2-0.5b", "decode", requests=1, context=512),
        # a short exact-mode run: the float32 path answers ragged prompts (it is what replays and comparisons use)
        _case("float32 prompts 0.5B", "qwen2-0.5b", "prompt", dtype="float32", requests=3, tokens=210),
        # a small batch job from prompts to sampled ids: the whole loop with its host side
        _case("generate 0.5B", "qwen2-0.5b-untied", "generate", requests=8, tokens=48, new=16),
        # a server's steady state: eight conversations of the headline shape
        _case("decode 8 7B", "qwen2-7b", "decode", requests=8, context=2048),
        # the same server under load
        _case("decode 64 7B", "qwen2-7b", "decode", requests=64, context=512, page_size=64),
        # time to first token of a long prompt on the headline shape: the largest case
        _case("prompt 2048 7B", "qwen2-7b", "prompt", requests=1, tokens=2048),
        # prompts of each hybrid design: delta rule and state space; retention, selective scan and experts with two prompts in the
        # step; attention over latents and time mixing at an odd length; lightning, channel decay, gates and experts
        _case("prompt Nunivik", "nunivik-2k", "prompt", requests=1, tokens=2048),
        _case("two prompts Mirovik", "mirovik-2k", "prompt", requests=2, tokens=1400),
        _case("odd prompt Kudazen", "kudazen-2k", "prompt", requests=1, tokens=1531, page_size=32),
        _case("prompt Tobadra", "tobadra-2k", "prompt", requests=1, tokens=2048),
        # routed experts fetch most of their matrices for a handful of tokens
        _case("decode 16 Zurevik", "zurevik-2k", "decode", requests=16, context=1500),
        # a new prompt joins conversations that go on
        _case("mixed step Biropel", "biropel-2k", "mixed", requests=7, context=900, tokens=1000),
    ]


def draw(rng) -> dict:
    kind = rng.choice(["prompt", "prompt", "prompt", "decode", "decode", "decode", "mixed", "mixed", "generate"])
    if kind == "generate":
        return _case(None, "qwen2-0.5b-untied", kind, requests=_spread(rng, 1, 16), tokens=_spread(rng, 8, 200), new=rng.randint(4, 24),
                     page_size=rng.choice([16, 32, 64]))
    model = rng.choice([m for m in MODELS if m != "qwen2-0.5b-untied"])
    sizes = {"page_size": rng.choice([16, 32, 64])}
    if kind in ("decode", "mixed"):
        sizes["requests"] = _spread(rng, 1, 64)
        sizes["context"] = min(_spread(rng, 64, 2048), 32768 // sizes["requests"])
    if kind == "prompt":
        sizes["requests"] = rng.choice([1, 1, 1, 2, 3, 5])
    if kind in ("prompt", "mixed"):
        sizes["tokens"] = _spread(rng, 24, 2048) // (1 if sizes["requests"] < 3 or kind == "mixed" else 2) + 1
        sizes["tokens"] = min(sizes["tokens"], 1024 if sizes["requests"] == 2 and kind == "prompt" else 2048)
        if kind == "mixed":
            sizes["tokens"] = min(sizes["tokens"], 1500)
    if model == "qwen2-0.5b" and kind == "prompt" and sizes["tokens"] <= 400 and rng.random() < 0.5:
        sizes["dtype"] = "float32"
    return _case(None, model, kind, **sizes)


def _case(name, model, kind, dtype="bfloat16", page_size=16, **sizes) -> dict:
    return {**({"name": name} if name else {}), "model": model, "kind": kind, "dtype": dtype, "page_size": page_size, **sizes}


def _spread(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _prompt_lengths(case: dict) -> list[int]:
    """Prompts of unequal lengths, the first the longest."""
    if case["kind"] == "generate":
        return [max(1, case["tokens"] - 5 * i % case["tokens"]) for i in range(case["requests"])]
    if case["kind"] == "mixed":
        return [case["tokens"]]
    return [max(1, case["tokens"] // (i + 1) + 3 * i) for i in range(case["requests"])]


def _contexts(case: dict) -> list[int]:
    """How many tokens the live requests hold: between half of ``context`` and all of it."""
    n = case["requests"]
    return [max(1, case["context"] - i * case["context"] // (2 * n)) for i in range(n)]


# ------------------------------------------------------------------------------------------ models as documents
def _document(model: str) -> dict:
    """config.json of the model."""
    s, family = MODELS[model], model.split("-")[0]
    if family == "qwen2":
        return {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "hidden_size": s["hidden"], "num_hidden_layers": s["layers"],
                "intermediate_size": s["ff"], "num_attention_heads": s["heads"], "num_key_value_heads": s["kv_heads"], "head_dim": s["dim"],
                "vocab_size": s["vocab"], "max_position_embeddings": 32768, "rope_theta": 1e6, "rms_norm_eps": 1e-6, "hidden_act": "silu",
                "tie_word_embeddings": s["tied"]}
    heads = {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
    top = {"vocab": VOCAB, "width": s["width"], "norm": {"eps": 1e-6}}
    dense = {"kind": "dense", "ff": s.get("ff")}
    if family == "nunivik":
        a = {"type": "attention", "mlp": dense, "mixer": {**heads, "softcap": 50.0, "mask": {"size": s["window"]}, "v_mix": True,
                                                          "rot": {"dims": 128, "base": 1e6, "scaling": {"factor": 1.0}}}}
        d = {"type": "delta", "mlp": None, "mixer": {"heads": s["delta"], "kv_heads": s["delta"] // 2, "dim": 128, "vdim": 128, "conv": 4}}
        m = {"type": "mamba2", "mlp": None, "mixer": {"heads": s["states"], "vdim": 64, "state": 128, "groups": s["groups"], "norm_groups": s["groups"], "conv": 4}}
        return {"architecture": "Nunivik", **top, "embedding": {"scale": 1.0}, "layers": [a, a, d, m, a, a, d, m]}
    if family == "mirovik":
        n = s["retention"]
        right = {"heads": n, "dim": 128, "vdim": 128, "rot": {"dims": 64, "base": 1e6}, "decay": [1.0 - 2.0 ** (-5 - 5 * h / (n - 1)) for h in range(n)]}
        mixer = {"left": {**heads, "bias_max": 256, "buckets": 32}, "right": right, "left_scale": 1.0, "right_scale": 1.0}
        routed = {"kind": "moe", "router": {"experts": EXPERTS, "top": CHOSEN}, "expert": {"ff": s["expert"]}, "shared": {"ff": s["expert"]}}
        selective = {"type": "mamba1", "mlp": dense, "mixer": {"inner": s["channels"], "state": 16, "dt_rank": s["rank"], "conv": 4}}
        p, q = ({"type": "parallel", "mixer": mixer, "mlp": mlp} for mlp in (dense, routed))
        return {"architecture": "Mirovik", **top, "embedding": {"scale": 1.0}, "layers": [p, q, selective, q], "loop": {"start": 0, "stop": 4, "times": 2}}
    if family == "kudazen":
        mlp = {**dense, "limit": 7.0}
        a = {"type": "attention", "mlp": mlp, "mixer": {**heads, "mask": {"size": s["chunk"]}}}
        l = {"type": "latent_attention", "mlp": mlp, "mixer": {"heads": s["latent"], "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 1536,
                                                               "scale": 192 ** -0.5, "rot": {"dims": 64, "base": 1e6}}}
        w = {"type": "wkv", "mlp": mlp, "mixer": {"heads": s["wkv"], "dim": 64, "decay_rank": 64}}
        return {"architecture": "Kudazen", **top, "norm": {"eps": 1e-6, "groups": 4}, "layers": [a, l, l, w, a, l, l, w]}
    if family == "tobadra":
        n = s["recurrent"]
        routed = {"kind": "moe", "expert": {"ff": s["expert"]}, "shared": {"ff": s["expert"]},
                  "router": {"experts": EXPERTS, "top": CHOSEN, "scale": 2.5, "identity": 2, "groups": {"count": 6, "keep": 4}}}
        attention = {**heads, "mask": {"size": s["window"]}, "rot": {"dims": 64, "base": 1e6}}
        lightning = {"heads": n, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-5 - 3 * i / n) for i in range(n)]}
        delta = {"heads": n, "kv_heads": n, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}
        first, a, l, d = ({"type": t, "mixer": m, "mlp": f} for t, m, f in (("attention", attention, dense), ("attention", attention, routed),
                                                                          ("lightning", lightning, routed), ("channel_delta", delta, routed)))
        return {"architecture": "Tobadra", **top, "canon": {"taps": 4}, "logit_scale": 1.0, "layers": [first, a, l, d, a, a, l, {**d, "weights_of": 3}]}
    if family == "zurevik":
        mlp = {"kind": "moe", "expert": {"ff": s["expert"]}, "router": {"experts": EXPERTS, "top": CHOSEN}}
        sinks = {**heads, "mask": {"size": s["window"]}}
        a, b, c = ({"type": "attention_2", "mlp": mlp, "mixer": m} for m in (sinks, {**sinks, "kv_from": 0}, {**sinks, "kv_from": 5}))
        d = {"type": "attention", "mlp": mlp, "mixer": {**heads, "dim": 64, "scale": 0.125, "diff": 0.5, "mask": {"size": s["window"], "keep_first": 4}}}
        return {"architecture": "Zurevik", **top, "embedding": {"scale": 1.0}, "logit_softcap": 30.0, "layers": [a, d, d, b, d, a, d, c]}
    windowed = {**heads, "mask": {"size": s["window"]}}
    a = {"type": "attention", "mlp": dense, "mixer": {**windowed, "rot": {"dims": 64, "base": 1e6}}}
    p = {"type": "parallel", "mlp": dense, "mixer": {
        "left": {**windowed, "softcap": 30.0, "rot": {"dims": 128, "base": 1e6, "scaling": {"factor": 4.0, "original": 1024, "fast": 32.0, "slow": 1.0}}},
        "right": {"heads": s["recurrent"], "vdim": 128, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}}}
    m = {"type": "parallel_2", "mlp": dense, "mixer": {"left": {**heads, "softcap": 50.0, "q_temp": {"coef": 0.1, "every": 1024}},
                                                      "right": {"heads": s["recurrent"], "dim": 128, "vdim": 128, "gate_cap": 15.0}}}
    shared = {**a, "mixer": {**a["mixer"], "kv_from": 0}}
    return {"architecture": "Biropel", **top, "streams": 4, "layers": [a, p, m, p, shared, m, p, m]}


# ------------------------------------------------------------------------------------------ weights
def _generator(text: str, device) -> torch.Generator:
    return torch.Generator(device).manual_seed(zlib.crc32(text.encode()))


def _tensor(case: dict, seed: int, name: str, shape) -> torch.Tensor:
    """One stored tensor (bfloat16) of the case's model."""
    shape, device, model = tuple(shape), torch.device("cuda"), case["model"]
    g = _generator(f"{seed}:{model}:{name}", device)
    family, last = model.split("-")[0], name.rsplit(".", 1)[-1]

    def normal(mean, std):
        return torch.empty(shape, dtype=torch.bfloat16 if mean == 0 else torch.float32, device=device).normal_(mean, std, generator=g)

    def uniform(low, high):
        return torch.empty(shape, device=device).uniform_(low, high, generator=g)

    routed = family in ("mirovik", "tobadra", "zurevik")
    if routed and (last in ("embed", "router")):
        outputs = EXPERTS + (2 if family == "tobadra" else 0)
        directions = torch.empty(outputs, shape[1], device=device).normal_(0, 1, generator=_generator(f"{seed}:{model}:directions", device))
        if last == "embed":
            out = normal(0, 1).float() + 2.0 * directions[torch.arange(shape[0], device=device) % outputs]
        else:
            out = (directions + 0.6 * directions.roll(1, 0)) * (8.0 / shape[1]) + normal(0, 0.002)
    elif model == "qwen2-0.5b-untied" and name in ("model.embed_tokens.weight", "lm_head.weight"):
        # every token has a likely successor, as text has: sampling sees a peaked distribution
        table = torch.empty(shape, dtype=torch.bfloat16, device=device).normal_(0, 1, generator=_generator(f"{seed}:{model}:successors", device))
        out = table if last == "weight" and name.startswith("model") else table.roll(1, 0) * 0.05 + normal(0, 0.02)
    elif family == "qwen2" and name == "model.embed_tokens.weight":
        out = normal(0, 1)
    elif family == "qwen2" and ("o_proj" in name or "down_proj" in name):
        out = normal(0, 0.02 / math.sqrt(2 * MODELS[model]["layers"]))
    elif last in ("dt_bias",) or name.endswith("dt.b"):
        out = uniform(math.log(1e-3), math.log(1e-1)).exp().expm1().log()  # softplus gives the step
    elif last == "A_log":
        out = torch.arange(1, shape[1] + 1, device=device).float().log().expand(shape) if len(shape) == 2 else uniform(1.0, 16.0).log()
    elif last == "w0":
        out = uniform(-6.0, -1.0)
    elif ".mu." in name:
        out = uniform(0.0, 1.0)
    elif last == "vmix":
        out = uniform(0.2, 0.8)
    elif last in ("in", "out", "mix") and ".hc" in name:
        out = normal(0.25, 0.05) if last == "in" else normal(1.0, 0.05) if last == "out" else normal(0.1, 0.02) + 0.6 * torch.eye(shape[0], device=device)
    elif name.endswith("f.b"):
        out = uniform(3.0, 6.0)
    elif last in ("conv", "canon1"):
        out = uniform(-0.5, 0.5) if last == "conv" else normal(0, 0.2)
    elif last in ("u", "sink", "rel") or name.endswith("i.b"):
        out = normal(0, 0.5)
    elif last in ("lq1", "lk1", "lq2", "lk2", "step"):
        out = normal(0, 0.1)
    elif last == "correction":
        out = normal(0, 0.005)
    elif family == "mirovik" and (last.startswith("norm") or name == "final.norm"):
        out = normal(0, 0.05)
    elif last in ("norm", "norm1", "norm2", "norm1b", "norm2b", "D", "temp") or "norm.weight" in name or name.endswith(("left.out", "right.out")):
        out = normal(1.0, 0.05)
    elif len(shape) == 2 and shape[1] <= 256:
        out = normal(0, shape[1] ** -0.5)
    else:
        out = normal(0, 0.02)
    return out.to(torch.bfloat16)


class _Weights:
    """The model's tensors by name and shape in 64 bits, made when asked for (a 7B model whole would be 60 GB)."""

    def __init__(self, case: dict, seed: int):
        self.case, self.seed = case, seed

    def __call__(self, name: str, *shape: int) -> torch.Tensor:
        return _tensor(self.case, self.seed, name, shape).double()


def _ids(case: dict, seed: int, what: str, count: int) -> list[int]:
    vocab = MODELS[case["model"]].get("vocab", VOCAB)
    return torch.randint(0, vocab, (count,), generator=_generator(f"{seed}:{what}", "cpu")).tolist()


# ------------------------------------------------------------------------------------------ what a user holds, and one pass
def prepare(case: dict, seed: int) -> dict:
    from hyperion_b200.api import Engine, resolve_dtype
    from hyperion_b200.models import DecoderModel, architecture_of

    document = _document(case["model"])
    architecture = architecture_of(document)
    config = architecture.read_config(document)
    dtype = resolve_dtype(case["dtype"])
    model = DecoderModel(architecture.build_spec(config), dtype, Engine._device("cuda:0"))
    model.load({name: _tensor(case, seed, name, wanted.shape).to(dtype) for name, wanted in model.expected_tensors().items()})
    kind, page = case["kind"], case["page_size"]
    prompts = [_ids(case, seed, f"prompt {i}", n) for i, n in enumerate(_prompt_lengths(case))] if "tokens" in case else []
    state = {"case": case, "prompts": prompts, "pass": 0}
    room = sum(len(p) + case.get("new", 0) + page for p in prompts)
    if kind in ("decode", "mixed"):
        more = MORE_TOKENS[kind] if case["requests"] <= 16 else 1024
        state["begun"] = [_ids(case, seed, f"context {i}", n) for i, n in enumerate(_contexts(case))]
        state["said"] = np.asarray(_ids(case, seed, "said", more * case["requests"])).reshape(more, -1).tolist()
        room += sum(len(c) + more + page for c in state["begun"])
    state["engine"] = Engine(model, config, page_size=page, max_tokens=room, max_requests=case["requests"] + 1)
    if kind in ("decode", "mixed"):
        _begin(state)
    return state


def _begin(state: dict) -> None:
    """Fill the live requests' caches with what was said before."""
    from hyperion_b200.engine.batch import StepEntry

    for i, ids in enumerate(state["begun"]):
        state["engine"].step([StepEntry(f"live {i}", ids, [])])


def run(state: dict):
    from hyperion_b200.engine.batch import StepEntry

    engine, case, kind = state["engine"], state["case"], state["case"]["kind"]
    if kind == "generate":
        from hyperion_b200.sampling import SamplingParams

        params = [SamplingParams(temperature=0.8, top_k=20, top_p=0.95, repetition_penalty=1.05, seed=i, max_tokens=case["new"], ignore_eos=True)
                  for i in range(len(state["prompts"]))]
        return np.asarray(engine.generate(state["prompts"], params), dtype=np.int64)
    entries = [StepEntry(f"new {i}", ids, [len(ids) - 1]) for i, ids in enumerate(state["prompts"])]
    if kind in ("decode", "mixed"):
        at = state["pass"] % len(state["said"])
        if state["pass"] and at == 0:  # the conversations have become too long: they start again
            for i in range(case["requests"]):
                engine.finish(f"live {i}")
            _begin(state)
        state["pass"] += 1
        entries += [StepEntry(f"live {i}", [token], [0]) for i, token in enumerate(state["said"][at])]
    logits = engine.step(entries)
    for i in range(len(state["prompts"])):
        engine.finish(f"new {i}")
    return logits


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _layers_of(document: dict) -> list[dict]:
    layers = document["layers"]
    loop = document.get("loop")
    return layers if loop is None else layers[: loop["start"]] + layers[loop["start"] : loop["stop"]] * loop["times"] + layers[loop["stop"] :]


def _layer_needs(layer: dict, width: int) -> tuple[float, float, float, float, float, list]:
    """(dense weights, weights of one expert, experts of a token, operations per token of a recurrence, values of its state,
    [(operations per query and key, cached values per key, window), ...]) of one layer."""
    m, kind = layer["mixer"], layer["type"]
    dense = expert = chosen = recurrent = record = 0.0
    attends = []

    def attention(a, maps=1, gate=True):
        nonlocal dense
        h, g, d, e = a["heads"], a["kv_heads"], a["dim"] * maps, a["vdim"]
        dense += width * (h * d + (g * (d + e) if "kv_from" not in a else 0) + h * e * (2 if gate else 1))
        attends.append((2.0 * h * (d + e * maps), g * (d + e), (a.get("mask") or {}).get("size")))

    def state(heads, d, e, per_entry):
        nonlocal recurrent, record
        recurrent += per_entry * heads * d * e
        record += heads * d * e

    if kind == "parallel" and "decay" in m["right"]:
        attention(m["left"])
        r = m["right"]
        dense += width * r["heads"] * (2 * r["dim"] + 3 * r["vdim"])
        state(r["heads"], r["dim"], r["vdim"], 5)
    elif kind in ("parallel", "parallel_2"):
        attention(m["left"], gate=False)
        r = m["right"]
        dense += width * (r["heads"] * (2 * r["dim"] + 3 * r["vdim"]) if kind == "parallel_2" else r["heads"] * r["vdim"] * 3 + 2 * r["groups"] * r["state"])
        state(r["heads"], r.get("dim", r.get("state")), r["vdim"], 5)
    elif kind == "attention_2":
        attention(m, gate=False)
    elif kind == "attention":
        attention(m, maps=2 if "diff" in m else 1, gate="diff" in m)
    elif kind == "latent_attention":
        h, r = m["heads"], m["kv_rank"]
        dense += width * (m["q_rank"] + r + m["rot_dim"] + h * m["vdim"]) + m["q_rank"] * h * (m["dim"] + m["rot_dim"]) + r * h * (m["dim"] + m["vdim"])
        attends.append((2.0 * h * (m["dim"] + m["rot_dim"] + m["vdim"]), r + m["rot_dim"], None))
    elif kind == "wkv":
        dense += width * (5 * m["heads"] * m["dim"] + 2 * m["decay_rank"])
        state(m["heads"], m["dim"], m["dim"], 5)
    elif kind == "mamba1":
        dense += width * 3 * m["inner"] + m["inner"] * (2 * m["dt_rank"] + 2 * m["state"])
        state(m["inner"], m["state"], 1, 6)
    elif kind == "mamba2":
        dense += width * (3 * m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"])
        state(m["heads"], m["state"], m["vdim"], 5)
    else:  # delta rules, lightning
        keys = m.get("kv_heads", m["heads"]) * m["dim"]
        dense += width * (2 * keys + 2 * m["heads"] * m["vdim"]) + (width * m["heads"] * m["vdim"] if "gate_rank" not in m else 4 * m["gate_rank"] * width)
        state(m["heads"], m["dim"], m["vdim"], 5 if kind == "lightning" else 7)
    mlp = layer.get("mlp")
    if mlp is not None and mlp["kind"] == "dense":
        dense += width * mlp["ff"] * (3 if "limit" in mlp or "softcap" in m else 2)
    elif mlp is not None:
        matrices = 3 if kind in ("parallel", "mamba1") else 2
        expert, chosen = matrices * width * mlp["expert"]["ff"], mlp["router"]["top"]
        dense += matrices * width * mlp.get("shared", {"ff": 0})["ff"]
    return dense, expert, chosen, recurrent, record, attends


def work(case: dict) -> dict:
    document, s = _document(case["model"]), MODELS[case["model"]]
    size = 4 if case["dtype"] == "float32" else 2
    prompts = _prompt_lengths(case) if "tokens" in case else []
    rows = [(0, n) for n in prompts]  # (positions held before, new tokens) of every row
    if case["kind"] == "generate":
        rows = [(0, n + case["new"] - 1) for n in prompts]
    if case["kind"] in ("decode", "mixed"):
        rows += [(c, 1) for c in _contexts(case)]
    tokens = sum(n for _, n in rows)
    wanted = len(rows) * case.get("new", 1)
    if "hidden" in s:
        width, vocab = s["hidden"], s["vocab"]
        per = width * s["dim"] * (2 * s["heads"] + 2 * s["kv_heads"]) + 3 * width * s["ff"]
        layers = [(per, 0.0, 0.0, 0.0, 0.0, [(4.0 * s["heads"] * s["dim"], 2 * s["kv_heads"] * s["dim"], None)])] * s["layers"]
        read = layers
    else:
        width, vocab = s["width"], VOCAB
        layers = [_layer_needs(layer, width) for layer in _layers_of(document)]
        gates = 2 * width * width if s.get("recurrent") and "Tobadra" == document["architecture"] else 0
        layers = [(d + gates, *rest) for d, *rest in layers]
        read = [_layer_needs(layer, width) for layer in document["layers"] if "weights_of" not in layer]
        read = [(d + gates, *rest) for d, *rest in read]
    flops = 2.0 * wanted * width * vocab
    values = width * vocab + wanted * vocab * (4 / size) + tokens * width
    passes = case.get("new", 1)
    for dense, expert, chosen, _, _, _ in read:
        values += passes * (dense + expert * min(EXPERTS, chosen * tokens))
    for dense, expert, chosen, recurrent, record, attends in layers:
        flops += tokens * (2.0 * (dense + expert * chosen) + recurrent)
        values += 2 * record * (4 / size) * len(rows)
        for per_pair, per_key, window in attends:
            for held, new in rows:
                pairs = sum(min(held + i + 1, window or held + i + 1) for i in range(new))
                flops += per_pair * pairs
                values += per_key * (min(held, window or held) + 2 * new)
    values += (passes - 1) * width * vocab
    return {"bytes": float(values * size), "flops": float(flops)}


def tolerance(case: dict):
    if case["kind"] == "generate":
        return {"differ": 0.01}
    if case["dtype"] == "float32":  # 6e-7 from 64 bits
        return {"rel": 1e-5, "max": 1e-4}
    # from 64 bits in bfloat16: 0.007 to 0.012, and 0.001 to 0.003 where tied embeddings carry the stream through to the logits or are large in it
    close = case["model"].split("-")[0] in ("mirovik", "tobadra", "zurevik") or case["model"] == "qwen2-0.5b"
    return {"rel": 0.012, "max": 0.12} if close else {"rel": 0.03, "max": 0.3}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def exact(case: dict, seed: int):
    """The pass's logits in 64-bit arithmetic: every row as one whole sequence, no cache."""
    if case["kind"] == "generate":
        return None
    with torch.no_grad():
        rows = [_ids(case, seed, f"prompt {i}", n) for i, n in enumerate(_prompt_lengths(case))] if "tokens" in case else []
        if case["kind"] in ("decode", "mixed"):
            more = MORE_TOKENS[case["kind"]] if case["requests"] <= 16 else 1024
            said = np.asarray(_ids(case, seed, "said", more * case["requests"])).reshape(more, -1)[0].tolist()
            rows += [_ids(case, seed, f"context {i}", n) + [said[i]] for i, n in enumerate(_contexts(case))]
        out = [None] * len(rows)
        order = sorted(range(len(rows)), key=lambda i: len(rows[i]))
        while order:  # rows of like length side by side, padded at their ends (nothing looks ahead); no more than fit
            most = len(rows[order[-1]])
            group = [i for i in order if 4 * len(rows[i]) >= most][-max(1, 33000 // most) :]
            order = [i for i in order if i not in group]
            ids = torch.zeros(len(group), most, dtype=torch.long, device="cuda")
            for b, i in enumerate(group):
                ids[b, : len(rows[i])] = torch.tensor(rows[i])
            ends = torch.tensor([len(rows[i]) - 1 for i in group], device="cuda")
            logits = _FORWARD[case["model"].split("-")[0]](_Weights(case, seed), _document(case["model"]), ids, ends)
            for b, i in enumerate(group):
                out[i] = logits[b]
        return torch.stack(out)


def _unit(x, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _softplus(x):
    return torch.nn.functional.softplus(x, threshold=1e9)


def _turn(x, dims, freq, pairs=False, sign=1.0, factor=1.0):
    """x [B, T, heads, n]: the first ``dims`` entries turn by position times ``freq``, in neighbouring pairs or in halves."""
    angle = torch.arange(x.shape[1], dtype=torch.float64, device=x.device)[:, None, None] * freq * sign
    c, s = angle.cos() * factor, angle.sin() * factor
    if pairs:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., dims:]], -1)
    u, v = x[..., : dims // 2], x[..., dims // 2 : dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _freq(dims, base):
    return torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device="cuda")


def _seen(tokens, window=None, chunk=None, keep=0):
    i, j = torch.arange(tokens, device="cuda")[:, None], torch.arange(tokens, device="cuda")[None, :]
    near = (j <= i) if window is None else (j <= i) & ((i - j < window) | (j < keep))
    return near if chunk is None else near & (i // chunk == j // chunk)


def _attend(q, k, v, scale, seen, cap=None, sink=None, bias=None):
    """q [B, T, H, d], k [B, T, G, d], v [B, T, G, e] -> [B, T, H, e]; ``scale`` a number or one per head, ``bias`` [H, T, T]."""
    rep, out = q.shape[2] // k.shape[2], []
    for b in range(q.shape[0]):
        heads = []
        for g in range(k.shape[2]):
            mine = slice(g * rep, (g + 1) * rep)
            s = torch.einsum("ihd,jd->hij", q[b, :, mine], k[b, :, g]) * (scale if isinstance(scale, float) else scale[mine, None, None])
            s = s if cap is None else cap * torch.tanh(s / cap)
            s = (s if bias is None else s + bias[mine]).masked_fill(~seen, -math.inf)
            if sink is None:
                p = torch.softmax(s, -1)
            else:
                z = sink[mine, None, None]
                top = torch.maximum(s.amax(-1, keepdim=True), z)
                p = torch.exp(s - top)
                p = p / (p.sum(-1, keepdim=True) + torch.exp(z - top))
            heads.append(torch.einsum("hij,je->ihe", p, v[b, :, g]))
        out.append(torch.cat(heads, 1))
    return torch.stack(out)


def _conv(x, weight, bias=0.0):
    taps = weight.shape[1]
    padded = torch.cat([torch.zeros_like(x[:, : 1]).expand(-1, taps - 1, -1), x], 1)
    return bias + sum(weight[:, j] * padded[:, j : j + x.shape[1]] for j in range(taps))


def _walk(keep, k, v, q, beta=None, bonus=None):
    """S <- keep S (+ rule) + k v^T, out = S^T q, token by token; all [B, T, H, .]; ``beta``: the delta rule; ``bonus``: q sees the
    token itself times ``bonus`` beside the state before it."""
    S = torch.zeros(*k.shape[:1], *k.shape[2:], v.shape[-1], dtype=torch.float64, device=k.device)
    out = torch.empty_like(v)
    for t in range(k.shape[1]):
        if bonus is not None:
            kv = k[:, t, :, :, None] * v[:, t, :, None, :]
            out[:, t] = torch.einsum("bhde,bhd->bhe", S + bonus[:, :, None] * kv, q[:, t])
            S = keep[:, t, :, :, None] * S + kv
            continue
        S = S * keep[:, t, :, :, None]
        u = v[:, t] if beta is None else beta[:, t, :, None] * (v[:, t] - torch.einsum("bhde,bhd->bhe", S, k[:, t]))
        S = S + k[:, t, :, :, None] * u[:, :, None, :]
        out[:, t] = torch.einsum("bhde,bhd->bhe", S, q[:, t])
    return out


def _heads(x, n):
    return x.unflatten(-1, (n, -1))


def _last(x, ends):
    return x[torch.arange(x.shape[0], device=x.device), ends]


def _qwen2(w, c, ids, ends):
    width, n, g, d, ff, eps = (c[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim", "intermediate_size", "rms_norm_eps"))
    x = w("model.embed_tokens.weight", c["vocab_size"], width)[ids]
    freq, seen = _freq(d, c["rope_theta"]), _seen(ids.shape[1])
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        a = _unit(x, eps) * w(p + "input_layernorm.weight", width)
        q, k, v = (_heads(a @ w(f"{p}self_attn.{z}_proj.weight", m * d, width).T + w(f"{p}self_attn.{z}_proj.bias", m * d), m) for z, m in (("q", n), ("k", g), ("v", g)))
        o = _attend(_turn(q, d, freq), _turn(k, d, freq), v, d ** -0.5, seen)
        x = x + o.flatten(2) @ w(p + "self_attn.o_proj.weight", width, n * d).T
        a = _unit(x, eps) * w(p + "post_attention_layernorm.weight", width)
        a = _silu(a @ w(p + "mlp.gate_proj.weight", ff, width).T) * (a @ w(p + "mlp.up_proj.weight", ff, width).T)
        x = x + a @ w(p + "mlp.down_proj.weight", width, ff).T
    x = _unit(_last(x, ends), eps) * w("model.norm.weight", width)
    return x @ w("model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight", c["vocab_size"], width).T


def _mamba2(w, p, m, h, width, eps):
    n, e, states, groups = m["heads"], m["vdim"], m["state"], m["groups"]
    inner = n * e
    z, xbc, dt = torch.split(h @ w(p + "in", 2 * inner + 2 * groups * states + n, width).T, [inner, inner + 2 * groups * states, n], -1)
    xbc = _silu(_conv(xbc, w(p + "conv", inner + 2 * groups * states, m["conv"]), w(p + "conv.b", inner + 2 * groups * states)))
    x, b, q = torch.split(xbc, [inner, groups * states, groups * states], -1)
    x, b, q = _heads(x, n), *(_heads(t, groups).repeat_interleave(n // groups, 2) for t in (b, q))
    dt = _softplus(dt + w(p + "dt_bias", n))
    keep = torch.exp(-torch.exp(w(p + "A_log", n)) * dt)
    y = _walk(keep[..., None], dt[..., None] * b, x, q) + w(p + "D", n)[:, None] * x
    y = y.flatten(2) * _silu(z)
    y = _unit(_heads(y, m["norm_groups"]), eps).flatten(2) * w(p + "norm", inner)
    return y @ w(p + "o", width, inner).T


def _delta(w, p, m, h, width, eps, channel):
    n, g, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (_heads(_silu(_conv(h @ w(p + z, r * s, width).T, w(p + z + ".conv", r * s, m["conv"]))), r) for z, r, s in (("q", g, d), ("k", g, d), ("v", n, e)))
    q = q * torch.rsqrt(q.pow(2).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k * torch.rsqrt(k.pow(2).sum(-1, keepdim=True) + 1e-6)
    q, k = (t.repeat_interleave(n // g, 2) for t in (q, k))
    beta, fade = torch.sigmoid(h @ w(p + "b", n, width).T), torch.exp(w(p + "A_log", n))
    if channel:
        rank = m["decay_rank"]
        pre = (h @ w(p + "a1", rank, width).T) @ w(p + "a2", n * d, rank).T + w(p + "dt_bias", n * d)
        keep = torch.exp(-fade[:, None] * _heads(_softplus(pre), n))
        gate = torch.sigmoid((h @ w(p + "g1", m["gate_rank"], width).T) @ w(p + "g2", n * e, m["gate_rank"]).T)
    else:
        keep = torch.exp(-fade * _softplus(h @ w(p + "a", n, width).T + w(p + "dt_bias", n)))[..., None]
        gate = _silu(h @ w(p + "g", n * e, width).T)
    o = _unit(_walk(keep, k, v, q, beta), eps) * w(p + "norm", e) * _heads(gate, n)
    return o.flatten(2) @ w(p + "o", width, n * e).T


def _nunivik(w, c, ids, ends):
    width, eps, first = c["width"], c["norm"]["eps"], None
    x = w("embed", c["vocab"], width)[ids] * c["embedding"]["scale"]
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        if layer["type"] == "attention":
            n, g, d = m["heads"], m["kv_heads"], m["dim"]
            q, k = (_unit(_heads(x @ w(p + z, r * d, width).T, r), eps) * w(p + z + ".norm", d) for z, r in (("q", n), ("k", g)))
            v, freq = _heads(x @ w(p + "v", g * d, width).T, g), _freq(d, m["rot"]["base"])
            lam = w(p + "vmix")
            first, v = (v, v) if first is None else (first, (1 - lam) * v + lam * first)
            o = _attend(_turn(q, d, freq, True), _turn(k, d, freq, True), v, m["scale"], _seen(ids.shape[1], m["mask"]["size"]), m["softcap"])
            y = o.flatten(2) @ w(p + "o", width, n * d).T
        else:
            y = _delta(w, p, m, x, width, eps, False) if layer["type"] == "delta" else _mamba2(w, p, m, x, width, eps)
        x = x + _unit(y, eps) * w(f"l{i}.norm1", width)
        if layer["mlp"] is not None:
            ff = layer["mlp"]["ff"]
            y = (_silu(x @ w(f"l{i}.mlp.gate", ff, width).T) * (x @ w(f"l{i}.mlp.up", ff, width).T)) @ w(f"l{i}.mlp.down", width, ff).T
            x = x + _unit(y, eps) * w(f"l{i}.norm2", width)
    return (_unit(_last(x, ends), eps) * w("final.norm", width)) @ w("head", c["vocab"], width).T


def _routed(h, scores, weights, expert):
    """Every token through its chosen experts: ``scores`` [B, T, top] indices, ``weights`` their weights, ``expert(e, rows, weights)``."""
    flat, out = h.flatten(0, 1), torch.zeros_like(h).flatten(0, 1)
    chosen, weights = scores.flatten(0, 1), weights.flatten(0, 1)
    for e in range(int(chosen.max()) + 1):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if len(rows):
            out.index_add_(0, rows, expert(e, flat[rows], weights[rows, place][:, None]))
    return out.view_as(h)


def _mirovik(w, c, ids, ends):
    width, eps, T = c["width"], c["norm"]["eps"], ids.shape[1]
    x = w("embed", c["vocab"], width)[ids] * c["embedding"]["scale"]
    index, loop = list(range(len(c["layers"]))), c["loop"]
    assert (loop["start"], loop["stop"]) == (0, len(index))
    steps = w("loop.step", loop["times"], width)
    seen = _seen(T)
    for run, i in enumerate(index * loop["times"]):
        layer, p = c["layers"][i], f"l{i}."

        def norm(y, name, p=p):
            return _unit(y, eps) * (1.0 + w(p + name, width))

        if i == 0:
            x = x + steps[run // len(index)]
        h, m = norm(x, "norm1"), layer["mixer"]
        if layer["type"] == "mamba1":
            inner, n, rank, z = m["inner"], m["state"], m["dt_rank"], p + "mix."
            u, gate = (h @ w(z + "in", 2 * inner, width).T).chunk(2, -1)
            u = _silu(_conv(u, w(z + "conv", inner, m["conv"]), w(z + "conv.b", inner)))
            low, b, q = torch.split(u @ w(z + "x", rank + 2 * n, inner).T, [rank, n, n], -1)
            dt = _softplus(low @ w(z + "dt", inner, rank).T + w(z + "dt.b", inner))
            fade, S, rows = -torch.exp(w(z + "A_log", inner, n)), 0.0, []
            for t in range(T):
                S = torch.exp(dt[:, t, :, None] * fade) * S + (dt[:, t] * u[:, t])[..., None] * b[:, t, None, :]
                rows.append((S * q[:, t, None, :]).sum(-1))
            y = ((torch.stack(rows, 1) + w(z + "D", inner) * u) * _silu(gate)) @ w(z + "o", width, inner).T
        else:
            a, z = m["left"], p + "mix.left."
            n, g, d, buckets = a["heads"], a["kv_heads"], a["dim"], a["buckets"]
            q, k = (_heads(_unit(h @ w(z + s, r * d, width).T, eps) * w(z + s + ".norm", r * d), r) for s, r in (("q", n), ("k", g)))
            half = buckets // 2
            bucket = torch.tensor([s if s < half else min(buckets - 1, half + int(math.floor(math.log(s / half) / math.log(a["bias_max"] / half) * (buckets - half))))
                                   for s in range(T)], device="cuda")
            apart = (torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None, :]).clamp(min=0)
            o = _attend(q, k, _heads(h @ w(z + "v", g * d, width).T, g), a["scale"], seen, bias=w(z + "rel", buckets, n).T[:, bucket[apart]])
            y = m["left_scale"] * ((o.flatten(2) * torch.sigmoid(h @ w(z + "g", n * d, width).T)) @ w(z + "o", width, n * d).T)
            r, z = m["right"], p + "mix.right."
            n, d, e, rot = r["heads"], r["dim"], r["vdim"], r["rot"]
            q, k, v = (_heads(h @ w(z + s, n * t, width).T, n) for s, t in (("q", d), ("k", d), ("v", e)))
            q, k = (_turn(t, rot["dims"], _freq(rot["dims"], rot["base"])) for t in (q, k))
            keep = torch.tensor(r["decay"], dtype=torch.float64, device="cuda")[:, None].expand(*k.shape[:3], 1)
            o = _unit(_walk(keep, k * d ** -0.5, v, q), eps).flatten(2) * _silu(h @ w(z + "g", n * e, width).T)
            y = y + m["right_scale"] * (o @ w(z + "o", width, n * e).T)
        x = x + norm(y, "norm1b")
        h, mlp = norm(x, "norm2"), layer["mlp"]
        if mlp["kind"] == "dense":
            y = _gelu(h @ w(p + "mlp.up", mlp["ff"], width).T) @ w(p + "mlp.down", width, mlp["ff"]).T
        else:
            def gated(z, rows):
                ff = mlp["expert"]["ff"]
                return (_silu(rows @ w(z + "gate", ff, width).T) * (rows @ w(z + "up", ff, width).T)) @ w(z + "down", width, ff).T

            best = torch.sigmoid(h @ w(p + "mlp.router", mlp["router"]["experts"], width).T).topk(mlp["router"]["top"], -1)
            y = gated(p + "mlp.shared.", h) + _routed(h, best.indices, best.values, lambda e, rows, s, p=p: gated(f"{p}mlp.e{e}.", s * rows))
        x = x + norm(y, "norm2b")
    return (_unit(_last(x, ends), eps) * (1.0 + w("final.norm", width))) @ w("embed", c["vocab"], width).T


def _kudazen(w, c, ids, ends):
    width, eps, groups, T = c["width"], c["norm"]["eps"], c["norm"]["groups"], ids.shape[1]

    def norm(x, name):
        return _unit(_heads(x, groups), eps).flatten(-2) * w(name, width)

    x = w("embed", c["vocab"], width)[ids]
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        h, n = norm(x, f"l{i}.norm1"), m["heads"]
        if layer["type"] == "attention":
            g, d = m["kv_heads"], m["dim"]
            q, k, v = (_heads(h @ w(p + z, r * d, width).T, r) for z, r in (("q", n), ("k", g), ("v", g)))
            slope = torch.tensor([2.0 ** (-8.0 * (a + 1) / n) for a in range(n)], dtype=torch.float64, device="cuda")
            at = torch.arange(T, dtype=torch.float64, device="cuda")
            o = _attend(q, k, _unit(v, eps), m["scale"] * w(p + "temp", n), _seen(T, chunk=m["mask"]["size"]), bias=-slope[:, None, None] * (at[:, None] - at[None, :]))
            y = o.flatten(2) @ w(p + "o", width, n * d).T
        elif layer["type"] == "latent_attention":
            d, r, e, R, freq = m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], _freq(m["rot"]["dims"], m["rot"]["base"])
            cq = _unit(h @ w(p + "dq", m["q_rank"], width).T, eps) * w(p + "dq.norm", m["q_rank"])
            q = _heads(cq @ w(p + "uq", n * (d + r), m["q_rank"]).T, n)
            down = h @ w(p + "dkv", R + r, width).T
            latent = _unit(down[..., :R], eps) * w(p + "dkv.norm", R)
            turned = _turn(down[..., None, R:], m["rot"]["dims"], freq, True).expand(-1, -1, n, -1)
            k = torch.cat([_heads(latent @ w(p + "uk", n * d, R).T, n), turned], -1)
            q = torch.cat([q[..., :d], _turn(q[..., d:], m["rot"]["dims"], freq, True)], -1)
            o = _attend(q, k, _heads(latent @ w(p + "uv", n * e, R).T, n), m["scale"], _seen(T), sink=w(p + "sink", n))
            y = o.flatten(2) @ w(p + "o", width, n * e).T
        else:
            d = m["dim"]
            before = torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1)
            r, k, v, gate, low = (h + (before - h) * w(p + "mu." + z, width) for z in "rkvgw")
            r, k, v = (_heads(t @ w(p + z, n * d, width).T, n) for z, t in (("r", r), ("k", k), ("v", v)))
            fade = torch.tanh(low @ w(p + "w1", m["decay_rank"], width).T) @ w(p + "w2", n * d, m["decay_rank"]).T + w(p + "w0", n * d)
            o = _walk(_heads(torch.exp(-torch.exp(fade)), n), k, v, r, bonus=w(p + "u", n, d))
            y = (_unit(o, eps).flatten(2) * w(p + "norm", n * d) * _silu(gate @ w(p + "g", n * d, width).T)) @ w(p + "o", width, n * d).T
        ff, limit = layer["mlp"]["ff"], layer["mlp"]["limit"]
        g = (h @ w(f"l{i}.mlp.gate", ff, width).T).clamp(max=limit)
        u = (h @ w(f"l{i}.mlp.up", ff, width).T).clamp(-limit, limit)
        x = x + y + (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(f"l{i}.mlp.down", width, ff).T
    return norm(_last(x, ends), "final.norm") @ w("embed", c["vocab"], width).T


def _tobadra(w, c, ids, ends):
    width, eps, T = c["width"], c["norm"]["eps"], ids.shape[1]

    def norm(x, name):
        return _unit(x, eps) * w(name, width)

    x = norm(w("embed", c["vocab"], width)[ids], "embed.norm")
    for i, layer in enumerate(c["layers"]):
        l, m, mlp = f"l{layer.get('weights_of', i)}.", layer["mixer"], layer["mlp"]
        p, n = l + "mix.", m["heads"]
        a = norm(x, l + "norm1")
        h = a + _conv(a, w(l + "canon1", width, c["canon"]["taps"]))
        if layer["type"] == "attention":
            g, d, base, dims = m["kv_heads"], m["dim"], m["rot"]["base"], m["rot"]["dims"]
            q, k, v = (_heads(h @ w(p + z, r * d, width).T + w(p + z + ".b", r * d), r) for z, r in (("q", n), ("k", g), ("v", g)))
            q, k, v = _turn(q, dims, _freq(dims, base)), _turn(k, dims, _freq(dims, base)), _turn(v, d, _freq(d, base))
            o = _turn(_attend(q, k, v, m["scale"], _seen(T, m["mask"]["size"])), d, _freq(d, base), sign=-1.0)
            y = o.flatten(2) @ w(p + "o", width, n * d).T + w(p + "o.b", width)
        elif layer["type"] == "lightning":
            d, e = m["dim"], m["vdim"]
            q, k, v = (_heads(_silu(h @ w(p + z, n * s, width).T), n) for z, s in (("q", d), ("k", d), ("v", e)))
            keep = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")[:, None].expand(*k.shape[:3], 1)
            o = _unit(_walk(keep, k, v, q).flatten(2), eps) * w(p + "norm", n * e)
            y = (o * torch.sigmoid(h @ w(p + "g", n * e, width).T)) @ w(p + "o", width, n * e).T
        else:
            y = _delta(w, p, m, h, width, eps, True)
        x = x + norm(y * torch.sigmoid(a @ w(l + "rg1", width, width).T + w(l + "rg1.b", width)), l + "norm1b")
        b, z = norm(x, l + "norm2"), l + "mlp."
        if mlp["kind"] == "dense":
            y = _gelu(b @ w(z + "up", mlp["ff"], width).T) @ w(z + "down", width, mlp["ff"]).T
        else:
            r, ff = mlp["router"], mlp["expert"]["ff"]
            outputs = r["experts"] + r["identity"]
            s = torch.softmax(b @ w(z + "router", outputs, width).T, -1)
            choice = s + w(z + "correction", outputs)
            best = _heads(choice, r["groups"]["count"]).amax(-1)
            kept = torch.zeros_like(best, dtype=torch.bool).scatter_(-1, best.topk(r["groups"]["keep"], -1).indices, True)
            chosen = choice.masked_fill(~kept.repeat_interleave(outputs // r["groups"]["count"], -1), -math.inf).topk(r["top"], -1).indices

            def plain(name, rows):
                return torch.nn.functional.gelu(rows @ w(name + "up", ff, width).T) @ w(name + "down", width, ff).T

            y = _routed(b, chosen, torch.gather(s, -1, chosen) * r["scale"], lambda e, rows, s, z=z: s * (plain(f"{z}e{e}.", rows) if e < r["experts"] else rows))
            y = y + plain(z + "shared.", b) * torch.sigmoid(b @ w(z + "shared.sg", 1, width).T)
        x = x + norm(y * torch.sigmoid(b @ w(l + "rg2", width, width).T + w(l + "rg2.b", width)), l + "norm2b")
    return norm(_last(x, ends), "final.norm") @ w("embed", c["vocab"], width).T * c["logit_scale"]


def _zurevik(w, c, ids, ends):
    width, eps, T, lent = c["width"], c["norm"]["eps"], ids.shape[1], {}
    x = w("embed", c["vocab"], width)[ids] * c["embedding"]["scale"]
    for i, layer in enumerate(c["layers"]):
        p, m, mlp = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        n, g, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        a = _unit(x, eps) * w(f"l{i}.norm1", width)
        if layer["type"] == "attention":
            q, k = (_unit((a @ w(p + z, r * 2 * d, width).T).unflatten(-1, (r, 2, d)), eps) * w(p + z + ".norm", d) for z, r in (("q", n), ("k", g)))
            v, seen = _heads(a @ w(p + "v", g * e, width).T, g), _seen(T, m["mask"]["size"], keep=m["mask"]["keep_first"])
            first, second = (_attend(q[..., s, :], k[..., s, :], v, m["scale"], seen) for s in (0, 1))
            lam = sum(sign * torch.exp((w(p + f"lq{s}", d) * w(p + f"lk{s}", d)).sum()) for s, sign in ((1, 1.0), (2, -1.0))) + m["diff"]
            o = _unit(first - lam * second, eps).flatten(2) * (1.0 - m["diff"]) * torch.sigmoid(a @ w(p + "g", n * e, width).T)
        else:
            q = _heads(a @ w(p + "q", n * d, width).T + w(p + "q.b", n * d), n)
            lent[i] = lent[m["kv_from"]] if "kv_from" in m else tuple(_heads(a @ w(p + z, g * d, width).T + w(p + z + ".b", g * d), g) for z in "kv")
            o = _attend(q, *lent[i], m["scale"], _seen(T, m["mask"]["size"]), sink=w(p + "sink", n))
            o = (o * torch.sigmoid(a @ w(p + "g", n, width).T)[..., None]).flatten(2)
        y = o @ w(p + "o", width, n * e).T
        b, z, ff = _unit(x, eps) * w(f"l{i}.norm2", width), f"l{i}.mlp.", mlp["expert"]["ff"]
        best = (b @ w(z + "router", EXPERTS, width).T + w(z + "router.b", EXPERTS)).topk(mlp["router"]["top"], -1)
        x = x + y + _routed(b, best.indices, torch.softmax(best.values, -1),
                            lambda e, rows, s, z=z, ff=ff: s * (torch.relu(rows @ w(f"{z}e{e}.up", ff, width).T).pow(2) @ w(f"{z}e{e}.down", width, ff).T))
    cap = c["logit_softcap"]
    return cap * torch.tanh((_unit(_last(x, ends), eps) * w("final.norm", width)) @ w("head", c["vocab"], width).T / cap)


def _stretched(rot):
    """(radians per position of every pair, factor on cosine and sine): pairs that turn rarely within the original length are slowed down."""
    freq, s = _freq(rot["dims"], rot["base"]), rot.get("scaling")
    if s is None:
        return freq, 1.0

    def pair(times):
        return rot["dims"] * math.log(s["original"] / (2 * math.pi * times)) / (2 * math.log(rot["base"]))

    low, high = max(math.floor(pair(s["fast"])), 0), min(math.ceil(pair(s["slow"])), rot["dims"] - 1)
    ramp = ((torch.arange(rot["dims"] // 2, dtype=torch.float64, device="cuda") - low) / max(high - low, 0.001)).clamp(0, 1)
    return freq / s["factor"] * ramp + freq * (1 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _biropel(w, c, ids, ends):
    width, eps, T, R, lent = c["width"], c["norm"]["eps"], ids.shape[1], c["streams"], {}
    X = (_unit(w("embed", c["vocab"], width)[ids], eps) * w("embed.norm", width))[None].repeat(R, 1, 1, 1)

    def sublayer(X, l, which, f):
        h = _unit(torch.einsum("r,rbtw->btw", w(f"{l}hc{which}.in", R), X), eps) * w(f"{l}norm{which}", width)
        return torch.einsum("rs,rbtw->sbtw", w(f"{l}hc{which}.mix", R, R), X) + w(f"{l}hc{which}.out", R)[:, None, None, None] * f(h)[None]

    def attention(h, p, m, i, bias, unit):
        n, g, d = m["heads"], m["kv_heads"], m["dim"]

        def project(z, r):
            y = _heads(h @ w(p + z, r * d, width).T + (w(p + z + ".b", r * d) if bias else 0.0), r)
            y = _unit(y, eps) if unit and z != "v" else y
            if z != "v" and "rot" in m:
                freq, factor = _stretched(m["rot"])
                y = _turn(y, m["rot"]["dims"], freq, factor=factor)
            return y

        lent[i] = lent[m["kv_from"]] if "kv_from" in m else (project("k", g), project("v", g))
        q, temp = project("q", n), m.get("q_temp")
        if temp is not None:
            q = q * torch.tensor([1.0 + temp["coef"] * math.log((t + 1) // temp["every"] + 1) for t in range(T)], dtype=torch.float64, device="cuda")[:, None, None]
        o = _attend(q, *lent[i], m["scale"], _seen(T, (m.get("mask") or {}).get("size")), m.get("softcap")).flatten(2)
        return (o * torch.sigmoid(h @ w(p + "g", n * d, width).T) if bias else o) @ w(p + "o", width, n * d).T

    def memory(h, p, m):
        n, d, e, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q, k, v = (_heads(h @ w(p + z, n * s, width).T, n) for z, s in (("q", d), ("k", d), ("v", e)))
        i, f = (cap * torch.tanh((h @ w(p + z, n, width).T + w(p + z + ".b", n)) / cap) for z in "if")
        f, top, keeps, takes, tops = torch.nn.functional.logsigmoid(f), torch.zeros_like(i[:, 0]), [], [], []
        for t in range(T):
            new = torch.maximum(f[:, t] + top, i[:, t])
            keeps.append(torch.exp(f[:, t] + top - new))
            takes.append(torch.exp(i[:, t] - new))
            top = new
            tops.append(new)
        keep, take, top = (torch.stack(z, 1)[..., None] for z in (keeps, takes, tops))
        q = q * d ** -0.5
        both = _walk(keep, take * k, torch.cat([v, torch.ones_like(v[..., :1])], -1), q)
        o = both[..., :e] / (torch.maximum(both[..., e:].abs(), torch.exp(-top)) + 1e-6)
        o = _unit(o, eps).flatten(2) * w(p + "norm", n * e)
        return (o * torch.sigmoid(h @ w(p + "g", n * e, width).T)) @ w(p + "o", width, n * e).T

    for i, layer in enumerate(c["layers"]):
        l, m = f"l{i}.", layer["mixer"]
        p = l + "mix."

        def mix(h, i=i, p=p, m=m, kind=layer["type"]):
            if kind == "attention":
                return attention(h, p, m, i, True, False)
            left = attention(h, p + "left.", m["left"], i, False, kind == "parallel_2")
            right = memory(h, p + "right.", m["right"]) if kind == "parallel_2" else _mamba2(w, p + "right.", m["right"], h, width, eps)
            return 0.5 * (_unit(left, eps) * w(p + "left.out", width) + _unit(right, eps) * w(p + "right.out", width))

        ff = layer["mlp"]["ff"]
        X = sublayer(X, l, 1, mix)
        X = sublayer(X, l, 2, lambda h, l=l, ff=ff: torch.relu(h @ w(l + "mlp.up", ff, width).T).pow(2) @ w(l + "mlp.down", width, ff).T)
    return (_unit(_last(X.sum(0), ends), eps) * w("final.norm", width)) @ w("head", c["vocab"], width).T


_FORWARD = {"qwen2": _qwen2, "nunivik": _nunivik, "mirovik": _mirovik, "kudazen": _kudazen, "tobadra": _tobadra, "zurevik": _zurevik, "biropel": _biropel}
