"""The work that a user of this engine has it do, as cases that can be timed and compared.

A case is one pass through the public step function (`Engine.runner.run` over requests of `Engine.cache`, as the
generation loop, the replay program and the benchmark call it), or one call of the sampler. A pass decodes one token of
each of a number of requests, reads prompts whole or in portions of a token budget, or does both in mixed steps. The
token ids are given (a replay), so that the logits of two implementations can be compared.

Models: Muse-Glimmer of about 1.7 and 8 billion parameters and a tiny one, and two of the other families (Bobarax and
Gisudra), with the sizes of the benchmark and of the tests, and random weights. Gisudra has dense units in the place
of its experts, since a router's choice may fall the other way with any rounding; Bobarax's experts are chosen by a
table.
"""

from __future__ import annotations

import math
import random

import torch

from mlx_omnia_b200.engine.engine import Engine, EngineArgs
from mlx_omnia_b200.engine.step import StepEntry
from mlx_omnia_b200.sampling.batch import sample_rows
from mlx_omnia_b200.sampling.options import SamplingParams

PREFILL_STEP = 8192  # tokens a step at most while `prepare` brings requests to their contexts


# -- models ------------------------------------------------------------------------------------------------------
def _muse(layers, hidden, inner, heads, kv_heads, dim, vocab, tied, **other):
    text = {"hidden_size": hidden, "intermediate_size": inner, "num_hidden_layers": layers, "num_attention_heads": heads,
            "num_key_value_heads": kv_heads, "head_dim": dim, "vocab_size": vocab, "rms_norm_eps": 1e-6,
            "post_norm_eps": 1e-6, "sliding_window": 4096, "qk_scale_factor": 1.0, "output_multiplier": 1.0,
            "final_logit_softcapping": 30.0, "layer_types": ["full_attention"] * layers,
            "layer_rope_theta": [1e6] * layers, "eos_token_id": [], "tie_word_embeddings": tied} | other
    return {"architectures": ["MuseGlimmerForConditionalGeneration"], "model_type": "muse_glimmer", "text_config": text}


def _bobarax():
    heads, dim, width = 16, 128, 2048
    moe = {"kind": "moe", "expert": {"ff": 1536, "limit": 7.0}, "router": {"experts": 32, "top": 4}}
    windowed = {"heads": heads, "kv_heads": 4, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
                "rot": {"base": 100000.0, "dims": dim // 2}, "mask": {"size": 512}}
    decay = [1.0 - 2.0 ** -(3 + 7 * h / (heads - 1)) for h in range(heads)]
    runs = {"heads": heads, "kv_heads": 4, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 30.0, "mask": {"size": 512}}
    layers = []
    for i in range(0, 8, 4):
        layers += [{"type": "attention_2", "mixer": dict(windowed), "mlp": {"kind": "dense", "ff": 8192}},
                   {"type": "lightning", "mixer": {"heads": heads, "dim": dim, "vdim": dim, "decay": decay}, "mlp": moe},
                   {"type": "attention", "mixer": runs, "mlp": moe},
                   {"type": "attention_2", "mixer": dict(windowed, kv_from=i), "mlp": moe}]
    return {"architecture": "Bobarax", "vocab": 32768, "width": width, "residual_mult": 0.5, "logit_scale": 1.0,
            "norm": {"eps": 1e-5}, "layers": layers}


def _gisudra():
    heads, dim, width = 16, 128, 2048
    dense = {"kind": "dense", "ff": 2 * width}
    mamba = {"type": "mamba2", "mixer": {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4,
                                         "norm_groups": 1}, "mlp": dense}
    layers = []
    for _ in range(2):
        layers += [mamba,
                   {"type": "attention", "mixer": {"heads": heads, "kv_heads": 4, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
                                                   "mask": {"size": 512, "keep_first": 64}, "v_mix": True}, "mlp": dense},
                   {"type": "latent_attention", "mixer": {"heads": heads, "dim": dim, "rot_dim": 64, "vdim": dim,
                                                          "kv_rank": 4 * dim, "scale": (dim + 64) ** -0.5, "mask": {"size": 512},
                                                          "rot": {"base": 10000.0, "dims": 64}}, "mlp": dense}, mamba]
    return {"architecture": "Gisudra", "vocab": 32768, "width": width, "norm": {"eps": 1e-5}, "layers": layers}


MODELS = {
    # name: (config.json, engine dtype, tokens a cache page)
    "muse-1.7b": (_muse(28, 2048, 6144, 16, 8, 128, 151936, True), "bfloat16", 16),
    "muse-8b": (_muse(36, 4096, 12288, 32, 8, 128, 151936, False), "bfloat16", 16),
    "muse-tiny": (_muse(3, 96, 320, 8, 1, 24, 1000, False, rms_norm_eps=1e-5, sliding_window=16, qk_scale_factor=1.25,
                        output_multiplier=0.5, final_logit_softcapping=20.0, layer_rope_theta=[1e6, 0.0, 1e6],
                        layer_types=["sliding_attention", "full_attention", "sliding_attention"]), "float32", 8),
    "bobarax": (_bobarax(), "bfloat16", 16),
    "gisudra": (_gisudra(), "bfloat16", 16),
}


def _vocab(raw):
    return raw["text_config"]["vocab_size"] if "text_config" in raw else raw["vocab"]


class _Draw:
    """Random tensors on the GPU from one seed, in a fixed order."""

    def __init__(self, seed, dtype):
        self.generator, self.dtype = torch.Generator(device="cuda").manual_seed(seed), dtype

    def matrix(self, rows, cols, std=None):
        x = torch.randn(rows, cols, generator=self.generator, device="cuda", dtype=self.dtype)
        return x.mul_(cols ** -0.5 if std is None else std)

    def vector(self, size, mean=1.0, std=0.1):
        return torch.randn(size, generator=self.generator, device="cuda") * std + mean


def _weights(model, seed):
    raw, dtype, _ = MODELS[model]
    d = _Draw(seed, getattr(torch, dtype))
    return {"muse_glimmer": _muse_weights, "Bobarax": _bobarax_weights, "Gisudra": _gisudra_weights}[
        raw.get("model_type") or raw["architecture"]](raw, d)


def _muse_weights(raw, d):
    c = raw["text_config"]
    D, q, kv, inner = (c["hidden_size"], c["num_attention_heads"] * c["head_dim"], c["num_key_value_heads"] * c["head_dim"],
                       c["intermediate_size"])
    p = "model.language_model."
    out = {p + "embed_tokens.weight": d.matrix(c["vocab_size"], D, 0.02), p + "norm.weight": d.vector(D, 1.0, 0.01)}
    for i in range(c["num_hidden_layers"]):
        for name, rows, cols in (("self_attn.q_proj", q, D), ("self_attn.k_proj", kv, D), ("self_attn.v_proj", kv, D),
                                 ("self_attn.gate_proj", q, D), ("self_attn.o_proj", D, q), ("mlp.gate_proj", inner, D),
                                 ("mlp.up_proj", inner, D), ("mlp.down_proj", D, inner)):
            out[f"{p}layers.{i}.{name}.weight"] = d.matrix(rows, cols, 0.02)
        for name in ("input_layernorm", "post_attention_layernorm", "pre_feedforward_layernorm", "post_feedforward_layernorm"):
            out[f"{p}layers.{i}.{name}.weight"] = d.vector(D, 0.0, 0.01)
    if not c["tie_word_embeddings"]:
        out["lm_head.weight"] = d.matrix(c["vocab_size"], D, 0.02)
    return out


def _bobarax_weights(raw, d):
    D = raw["width"]
    gain = 2.0 * D ** -0.5
    out = {"embed": d.matrix(raw["vocab"], D, 1.0), "final.norm": d.vector(D, 0.0)}
    for i, layer in enumerate(raw["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]
        H, dk, dv = m["heads"], m["dim"], m["vdim"]
        for name in ("norm1", "norm1b", "norm2", "norm2b"):
            out[p + name] = d.vector(D, 0.0)
        out[p + "mix.q"], out[p + "mix.o"] = d.matrix(H * dk, D, gain), d.matrix(D, H * dv)
        if layer["type"] == "lightning":
            out[p + "mix.k"], out[p + "mix.v"] = d.matrix(H * dk, D, gain), d.matrix(H * dv, D, gain)
            out[p + "mix.norm"] = d.vector(H * dv)
        else:
            out[p + "mix.q.norm"] = d.vector(H * dk, 1.0, 0.2)
            if m.get("kv_from") is None:
                out[p + "mix.k"], out[p + "mix.v"] = d.matrix(m["kv_heads"] * dk, D, gain), d.matrix(m["kv_heads"] * dv, D, gain)
                out[p + "mix.k.norm"] = d.vector(m["kv_heads"] * dk, 1.0, 0.2)
        if layer["type"] != "attention":
            out[p + "mix.g"] = d.matrix(H * dv, D)
        units, ff = [p + "mlp."], f.get("ff")
        if f["kind"] == "moe":
            experts, top, ff = f["router"]["experts"], f["router"]["top"], f["expert"]["ff"]
            units = [f"{p}mlp.e{e}." for e in range(experts)]
            order = torch.rand(raw["vocab"], experts, generator=d.generator, device="cuda").argsort(dim=1)
            out[p + "mlp.table"] = order[:, :top].to(torch.int32).contiguous()
        for unit in units:
            out[unit + "gate"], out[unit + "up"], out[unit + "down"] = d.matrix(ff, D, gain), d.matrix(ff, D, gain), d.matrix(D, ff)
    return out


def _gisudra_weights(raw, d):
    D = raw["width"]
    out = {"embed": d.matrix(raw["vocab"], D, 1.0), "head": d.matrix(raw["vocab"], D), "final.norm": d.vector(D)}
    for i, layer in enumerate(raw["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        H, dv = m["heads"], m["vdim"]
        out[f"l{i}.norm1"], out[f"l{i}.norm2"] = d.vector(D), d.vector(D)
        if layer["type"] == "mamba2":
            channels = H * dv + 2 * m["groups"] * m["state"]
            out[p + "in"] = d.matrix(H * dv + channels + H, D, 1.5 * D ** -0.5)
            out[p + "conv"] = d.vector((channels, m["conv"]), 0.0, 0.5 * m["conv"] ** -0.5)
            out[p + "conv"][:, -1] += 0.7
            out[p + "conv.b"], out[p + "dt_bias"], out[p + "A_log"] = (d.vector(channels, 0.0, 0.2), d.vector(H, -2.0, 1.0),
                                                                       d.vector(H, 0.0, 0.7))
            out[p + "D"], out[p + "norm"] = d.vector(H, 0.0, 0.5), d.vector(H * dv)
        elif layer["type"] == "attention":
            G, dk = m["kv_heads"], m["dim"]
            out[p + "q"], out[p + "k"], out[p + "v"] = d.matrix(H * dk, D), d.matrix(G * dk, D), d.matrix(G * dv, D)
            out[p + "q.norm"], out[p + "k.norm"] = d.vector(dk), d.vector(dk)
            out[p + "vmix"] = d.vector(1, 0.4, 0.2)[0]
        else:
            dk, rot, rank = m["dim"], m["rot_dim"], m["kv_rank"]
            out[p + "q"], out[p + "dkv"] = d.matrix(H * (dk + rot), D, 2.0 * D ** -0.5), d.matrix(rank + rot, D)
            out[p + "dkv.norm"] = d.vector(rank)
            out[p + "uk"], out[p + "uv"] = d.matrix(H * dk, rank, 2.0 * rank ** -0.5), d.matrix(H * dv, rank)
        if layer["type"] != "mamba2":
            out[p + "g"] = d.matrix(H * dv, D)
        out[p + "o"] = d.matrix(D, H * dv)
        for name, rows, cols in (("gate", layer["mlp"]["ff"], D), ("up", layer["mlp"]["ff"], D), ("down", D, layer["mlp"]["ff"])):
            out[f"l{i}.mlp.{name}"] = d.matrix(rows, cols)
    return out


# -- the cases ---------------------------------------------------------------------------------------------------
def _decode(model, batch, context, ragged=False):
    """`batch` requests that hold up to `context` positions decode a token each. ragged: as many as that only for
    the longest, down to a sixteenth for others, as requests of many lengths that run together."""
    return {"kind": "step", "model": model, "batch": batch, "context": context, "ragged": ragged, "prompts": "", "portion": 0,
            "all_logits": False}


def _prefill(model, *prompts, portion=0):
    """Prompts of these lengths are read from their first token to their last, all of them whole in one step, or in
    portions of `portion` tokens."""
    return {"kind": "step", "model": model, "batch": 0, "context": 0, "ragged": False, "prompts": ",".join(map(str, prompts)),
            "portion": portion, "all_logits": False}


def _sample(batch, vocab, top_k=0, top_p=1.0, min_p=0.0, penalty=1.0, temperature=0.8):
    return {"kind": "sample", "batch": batch, "vocab": vocab, "temperature": temperature, "top_k": top_k, "top_p": top_p,
            "min_p": min_p, "penalty": penalty}


def listed():
    return [
        # A check of the engine in true 32 bits: a tiny model, three requests that decode while two prompts are read
        # in portions of eight, the logits of every token wanted. Launches and host work are all there is.
        dict(_decode("muse-tiny", 3, 40), prompts="31,17", portion=8, all_logits=True, name="replay-tiny-float32"),
        # The draw of the next token for 64 requests with a user's usual options.
        dict(_sample(64, 151936, top_k=50, top_p=0.95), name="sample-64"),
        # One user, a long conversation: the latency of a token.
        dict(_decode("muse-1.7b", 1, 4096), name="decode-1"),
        # A small group of users with long contexts.
        dict(_decode("muse-1.7b", 8, 4096), name="decode-8"),
        # A full server: 64 requests of many lengths.
        dict(_decode("muse-1.7b", 64, 2304, ragged=True), name="decode-64-ragged"),
        # One prompt of ordinary length, whole: the time to the first token.
        dict(_prefill("muse-1.7b", 2048), name="prefill-2048"),
        # Short prompts of several users that arrive together.
        dict(_prefill("muse-1.7b", 37, 211, 5, 700, 129), name="prefill-ragged"),
        # Continuous batching: eight requests decode while a prompt is read beside them in portions.
        dict(_decode("muse-1.7b", 8, 4096, ragged=True), prompts="700", portion=256, name="mixed-8"),
        # A long document read by the larger model in portions of a token budget.
        dict(_prefill("muse-8b", 8192, portion=2048), name="portions-8b"),
        # Linear attention, windows and experts: a prompt, and a decode step.
        dict(_prefill("bobarax", 2048), name="bobarax-prefill"),
        dict(_decode("bobarax", 8, 4096), name="bobarax-decode"),
        # State-space recurrence, windows with kept first tokens, latent attention: prompts of unequal lengths.
        dict(_prefill("gisudra", 1201, 433, 97), name="gisudra-prefill"),
    ]


def draw(rng):
    def log(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    def lengths(count, most):
        left, out = most, []
        for _ in range(count):
            out.append(min(log(5, most), left - (count - len(out) - 1) * 5))
            left -= out[-1]
        return out

    kind = rng.choice(["tiny", "sample", "decode", "decode", "decode-8b", "prefill", "prefill", "portions", "mixed", "other-prefill",
                       "other-decode"])
    if kind == "tiny":
        prompts = lengths(rng.randint(1, 4), 90)
        return dict(_decode("muse-tiny", rng.randint(1, 6), rng.randint(20, 90)), prompts=",".join(map(str, prompts)),
                    portion=max(8, -(-max(prompts) // 4)), all_logits=True)
    if kind == "sample":
        option = rng.choice([{"temperature": 0.0}, {}, {"top_k": log(2, 400)}, {"top_p": round(rng.uniform(0.5, 0.99), 3)},
                             {"min_p": round(rng.uniform(0.01, 0.3), 3)}, {"penalty": 1.1, "top_p": 0.9}])
        return _sample(log(1, 64), rng.choice([32768, 151936]), **option)
    if kind == "decode":
        return _decode("muse-1.7b", log(1, 64), log(100, 3000), rng.random() < 0.5)
    if kind == "decode-8b":
        return _decode("muse-8b", log(1, 24), log(100, 3000), rng.random() < 0.5)
    if kind == "prefill":
        return _prefill("muse-1.7b", *lengths(rng.randint(1, 6), log(60, 4096)))
    if kind == "portions":
        return _prefill("muse-1.7b", log(1000, 8192), portion=log(128, 2048))
    if kind == "mixed":
        prompt = log(60, 1500)
        return dict(_decode("muse-1.7b", log(1, 15), log(100, 4096), True), prompts=str(prompt), portion=max(64, -(-prompt // rng.randint(1, 6))))
    model = rng.choice(["bobarax", "gisudra"])
    if kind == "other-prefill":
        return _prefill(model, *lengths(rng.randint(1, 4), log(60, 4096)))
    return _decode(model, log(1, 32), log(100, 4096), rng.random() < 0.5)


def _layout(case):
    """(positions that each decoding request holds in whole pages, and those behind them in its last page; the prompts'
    lengths; tokens of a portion; steps of a pass). The same for every seed."""
    page = MODELS[case["model"]][2]
    prompts = [int(n) for n in case["prompts"].split(",")] if case["prompts"] else []
    portion = case["portion"] or max(prompts, default=1)
    steps = max((-(-n // portion) for n in prompts), default=1)
    rng = random.Random(case["context"] * 1000 + case["batch"])
    bulk, tail = [], []
    for i in range(case["batch"]):
        context = case["context"] if i == 0 or not case["ragged"] else rng.randint(-(-case["context"] // 16), case["context"])
        tail.append(1 + (context + 3 * i) % max(1, page - 2 - steps))
        bulk.append(max(1, (context - steps) // page) * page)
    return bulk, tail, prompts, portion, steps


# -- a pass ------------------------------------------------------------------------------------------------------
def _sample_params(case):
    return SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], min_p=case["min_p"],
                          repetition_penalty=case["penalty"], seed=1)


def _ids(count, vocab, seed):
    return torch.randint(0, vocab, (count,), generator=torch.Generator().manual_seed(seed)).tolist()


def _tokens(case, seed):
    """Token ids: of each decoding request (its context and one more for each step), and of each prompt."""
    vocab = _vocab(MODELS[case["model"]][0])
    bulk, tail, prompts, _, steps = _layout(case)
    return ([_ids(b + t + steps, vocab, seed * 1000 + i) for i, (b, t) in enumerate(zip(bulk, tail))],
            [_ids(n, vocab, seed * 1000 + 500 + i) for i, n in enumerate(prompts)])


def _states(engine, count):
    """The per-request state of requests in the first `count` slots, entry by entry."""
    held = [engine.cache.state[e] for e in sorted(engine.cache.state)]
    return [t[:count] for s in held for t in ([s[k] for k in sorted(s)] if isinstance(s, dict) else [s])]


def prepare(case, seed):
    if case["kind"] == "sample":
        g = torch.Generator(device="cuda").manual_seed(seed)
        logits = torch.randn(case["batch"], case["vocab"], generator=g, device="cuda") * 2.5
        histories = [_ids(20, case["vocab"], seed * 1000 + i) if case["penalty"] != 1.0 else [] for i in range(case["batch"])]
        return {"logits": logits, "params": [_sample_params(case)] * case["batch"],
                "seeds": [seed * 1000 + i for i in range(case["batch"])], "draws": list(range(case["batch"])), "histories": histories}
    raw, dtype, page = MODELS[case["model"]]
    bulk, tail, prompts, portion, steps = _layout(case)
    contexts, texts = _tokens(case, seed)
    pages = lambda n: -(-n // page)  # noqa: E731
    tail_pages, text_pages = len(bulk), sum(pages(n) for n in prompts)
    total = sum(pages(b) for b in bulk) + tail_pages + text_pages
    engine = Engine.from_tensors(raw, _weights(case["model"], seed),
                                 EngineArgs(dtype=dtype, page_size=page, cache_tokens=total * page, max_requests=len(bulk) + len(prompts)))
    requests = [engine.cache.open(f"decoding-{i}") for i in range(len(bulk))]
    while any(r.tokens < b for r, b in zip(requests, bulk)):  # in steps, as long prompts are read
        room, entries = PREFILL_STEP, []
        for r, b, ids in zip(requests, bulk, contexts):
            n = min(b - r.tokens, room)
            if n > 0:
                entries.append(StepEntry(r, ids[r.tokens: r.tokens + n]))
                room -= n
        engine.runner.run(entries)
    if requests:
        engine.runner.run([StepEntry(r, ids[b: b + t]) for r, b, t, ids in zip(requests, bulk, tail, contexts)])
    state = {"engine": engine, "requests": requests, "held": [b + t for b, t in zip(bulk, tail)], "contexts": contexts, "texts": texts,
             "portion": portion, "steps": steps, "all_logits": case["all_logits"], "states": _states(engine, len(bulk) + len(prompts)),
             "cache": []}
    groups = engine.cache.groups
    if len(groups) == 1 and not groups[0].spec.forgets:
        # Every page that a pass writes to: the decoding requests' last ones, and the prompts'.
        first = sum(pages(b) for b in bulk)
        state["cache"] = [groups[0].pages[:, first:]]
    if requests and not texts:  # a program that decodes has decoded before
        saved = [t.clone() for t in state["states"]]
        run(state)
        for t, s in zip(state["states"], saved):
            t.copy_(s)
    return state


def run(state):
    if "logits" in state:
        return sample_rows(state["logits"], state["params"], state["seeds"], state["draws"], state["histories"])
    engine, portion, logits = state["engine"], state["portion"], []
    for request, held in zip(state["requests"], state["held"]):
        request.tokens = held  # back to where the pass begins: no page has been taken since
    readers = [engine.cache.open(f"prompt-{i}") for i in range(len(state["texts"]))]
    for step in range(state["steps"]):
        entries = [StepEntry(r, [ids[h + step]], [0]) for r, h, ids in zip(state["requests"], state["held"], state["contexts"])]
        for r, ids in zip(readers, state["texts"]):
            part = ids[step * portion: (step + 1) * portion]
            if part:
                ends = (step + 1) * portion >= len(ids)
                entries.append(StepEntry(r, part, list(range(len(part))) if state["all_logits"] else [len(part) - 1] if ends else []))
        logits.append(engine.runner.run(entries))
    for r in reversed(readers):
        engine.cache.close(r.request_id)
    return {"logits": logits, "cache": state["cache"], "states": state["states"]}


# -- what a pass cannot do without ------------------------------------------------------------------------------
def _layers(raw):
    """Per layer: (weights read whatever the tokens, weights of one expert, experts, chosen of them, query heads x (key and
    value width), cache elements a position, positions in sight or None, state elements, its operations a token)."""
    if "text_config" in raw:
        c = raw["text_config"]
        D, q, kv = c["hidden_size"], c["num_attention_heads"] * c["head_dim"], c["num_key_value_heads"] * c["head_dim"]
        for kind in c["layer_types"]:
            yield (D * (3 * q + 2 * kv) + 3 * D * c["intermediate_size"], 0, 0, 0, 2 * q, 2 * kv,
                   c["sliding_window"] if kind == "sliding_attention" else None, 0, 0)
        return
    D = raw["width"]
    for layer in raw["layers"]:
        m, f = layer["mixer"], layer["mlp"]
        H, dk, dv = m["heads"], m.get("dim", 0), m["vdim"]
        window = m["mask"]["size"] if "mask" in m else None
        score, cache, state, ops = H * (dk + dv), 0, 0, 0
        if layer["type"] == "lightning":
            w, score, state, ops = D * H * (2 * dk + 3 * dv), 0, H * dk * dv, 4 * H * dk * dv
        elif layer["type"] == "mamba2":
            rows, inner = m["state"], H * dv
            w, score, state, ops = D * (3 * inner + 2 * rows * m["groups"] + H), 0, H * rows * dv, 5 * H * rows * dv
        elif layer["type"] == "latent_attention":
            score, cache = H * (dk + m["rot_dim"] + dv), m["kv_rank"] + m["rot_dim"]
            w = D * (H * (dk + m["rot_dim"]) + cache + 2 * H * dv) + m["kv_rank"] * H * (dk + dv)
        else:
            kv = m["kv_heads"] * (dk + dv)
            gate = 0 if layer["type"] == "attention" and raw["architecture"] == "Bobarax" else H * dv
            w, cache = D * (H * dk + H * dv + gate + (kv if m.get("kv_from") is None else 0)), kv
        if f["kind"] == "moe":
            yield w, 3 * D * f["expert"]["ff"], f["router"]["experts"], f["router"]["top"], score, cache, window, state, ops
        else:
            yield w + 3 * D * f["ff"], 0, 0, 0, score, cache, window, state, ops


def work(case):
    if case["kind"] == "sample":
        values = case["batch"] * case["vocab"]
        return {"bytes": 4 * values, "flops": 2 * values}
    raw, dtype, _ = MODELS[case["model"]]
    size = 2 if dtype == "bfloat16" else 4
    bulk, tail, prompts, _, steps = _layout(case)
    spans = [(b + t, b + t + steps) for b, t in zip(bulk, tail)] + [(0, n) for n in prompts]  # positions computed, by request
    tokens = sum(hi - lo for lo, hi in spans)
    rows = len(bulk) * steps + (sum(prompts) if case["all_logits"] else len(prompts))
    head = _vocab(raw) * (raw["text_config"]["hidden_size"] if "text_config" in raw else raw["width"])
    read, flops = size * head + 4 * rows * _vocab(raw), 2 * rows * head
    for fixed, expert, experts, top, score, cache, window, state, ops in _layers(raw):
        touched = experts * (1 - (1 - top / experts) ** tokens) if experts else 0
        read += size * (fixed + expert * touched)
        flops += tokens * (2 * (fixed + top * expert) + ops)
        read += len(spans) * 2 * 4 * state
        for lo, hi in spans:
            if cache:  # the positions in sight when it starts are read, the new ones written and read
                read += size * cache * (min(lo, window or lo) + 2 * (hi - lo))
            if score:  # sum of the positions in sight of each new one
                w = window or hi
                seen = lambda n: n * (n + 1) / 2 if n <= w else w * (w + 1) / 2 + (n - w) * w  # noqa: E731
                flops += 2 * score * (seen(hi) - seen(lo))
    return {"bytes": float(read), "flops": float(flops)}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["model"] == "muse-tiny":  # 32 bits: 8e-7 from the result in 64 bits
        return {"rel": 5e-6, "max": 1e-4}
    return {"rel": 0.03, "max": 0.3}  # bfloat16 through 8 to 36 layers: 0.6 to 1.5 % from the result in 64 bits


# -- the same in 64 bits ------------------------------------------------------------------------------------------
def _rms(x, eps, weight=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight.double()


def _lin(x, weight):
    return x @ weight.double().T


def _softmax_attention(q, k, v, scale, window=None, run=None, keep_first=0, softcap=None):
    """q [T, H, dk], k [T, G, dk], v [T, G, dv] -> [T, H * dv], some rows of queries at a time."""
    T, H, dk = q.shape
    G = k.shape[1]
    qs, ks, vs = q.view(T, G, H // G, dk).permute(1, 2, 0, 3), k.permute(1, 2, 0).contiguous(), v.permute(1, 0, 2).contiguous()
    out = torch.empty(G, H // G, T, v.shape[2], dtype=q.dtype, device=q.device)
    for r0 in range(0, T, 1024):
        r1 = min(T, r0 + 1024)
        i, j = torch.arange(r0, r1, device=q.device)[:, None], torch.arange(r1, device=q.device)[None, :]
        sees = j <= i
        if window is not None:
            sees &= (i - j < window) | (j < keep_first)
        if run is not None:
            sees &= torch.div(i, run, rounding_mode="floor") == torch.div(j, run, rounding_mode="floor")
        n = r1 - r0
        s = torch.bmm(qs[:, :, r0:r1].reshape(G, -1, dk), ks[:, :, :r1]).view(G, H // G, n, r1).mul_(scale)
        if softcap is not None:
            s = s.div_(softcap).tanh_().mul_(softcap)
        s = torch.softmax(s.masked_fill_(~sees, -math.inf), dim=-1)
        out[:, :, r0:r1] = torch.bmm(s.view(G, -1, r1), vs[:, :r1]).view(G, H // G, n, -1)
    return out.permute(2, 0, 1, 3).reshape(T, -1)


def _rotate(x, dims, base, pairs):
    """x [T, heads, d], row t at position t: dims (2i, 2i + 1) turn together, or (i, i + dims / 2)."""
    f = base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=x.device) / dims)
    angle = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * f
    c, s = torch.cos(angle), torch.sin(angle)
    y = x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, dims // 2), slice(dims // 2, dims))
    y[..., a], y[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return y


def _sequences(x, lengths):
    return torch.split(x, lengths)


def _muse_exact(raw, W, ids, lengths, rows):
    """-> (logits of `rows`, per layer the keys and values of every token [tokens, 2, G, d], no states)."""
    c, p = raw["text_config"], "model.language_model."
    eps, post, H, G, d = c["rms_norm_eps"], c["post_norm_eps"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
    x, kept = _rms(W[p + "embed_tokens.weight"][ids].double(), eps), []
    for i, (kind, theta) in enumerate(zip(c["layer_types"], c["layer_rope_theta"])):
        w = lambda name: W[f"{p}layers.{i}.{name}.weight"]  # noqa: B023, E731
        h = _rms(x, eps, 1.0 + w("input_layernorm").double())
        q, k = (_rms(_lin(h, w(f"self_attn.{n}_proj")).view(len(ids), -1, d), eps) for n in "qk")
        v = _lin(h, w("self_attn.v_proj")).view(len(ids), G, d)
        if theta:
            q, k = (torch.cat([_rotate(s, d, theta, False) for s in _sequences(t, lengths)]) for t in (q, k))
        out = torch.cat([_softmax_attention(*s, c["qk_scale_factor"] * d ** -0.5,
                                            c["sliding_window"] if kind == "sliding_attention" else None)
                         for s in zip(*(_sequences(t, lengths) for t in (q, k, v)))])
        kept.append(torch.stack([k, v], dim=1))
        out = _lin(out * torch.sigmoid(_lin(h, w("self_attn.gate_proj"))), w("self_attn.o_proj"))
        x = x + _rms(out, post, 1.0 + w("post_attention_layernorm").double())
        h = _rms(x, eps, 1.0 + w("pre_feedforward_layernorm").double())
        gate = _lin(h, w("mlp.gate_proj"))
        out = _lin(gate * torch.sigmoid(gate) * _lin(h, w("mlp.up_proj")), w("mlp.down_proj"))
        x = x + _rms(out, post, 1.0 + w("post_feedforward_layernorm").double())
    head = W[p + "embed_tokens.weight"] if c["tie_word_embeddings"] else W["lm_head.weight"]
    logits = _lin(_rms(x[rows], eps, W[p + "norm.weight"]), head) * c["output_multiplier"]
    return torch.tanh(logits / c["final_logit_softcapping"]) * c["final_logit_softcapping"], kept, []


def _recur(decay, k, v, q):
    """S <- decay_t S + k_t v_t^T, o_t = S^T q_t from zeros. decay [T, H], k and q [T, H, dk], v [T, H, dv] -> (o, S)."""
    S, out = torch.zeros(*k.shape[1:], v.shape[2], dtype=v.dtype, device=v.device), torch.empty_like(v)
    for t in range(len(k)):
        S = torch.baddbmm(S * decay[t][:, None, None], k[t][:, :, None], v[t][:, None, :])
        out[t] = torch.bmm(q[t][:, None, :], S)[:, 0]
    return out, S


def _bobarax_exact(raw, W, ids, lengths, rows):
    eps, mult = raw["norm"]["eps"], raw["residual_mult"]
    x, held, states = W["embed"][ids].double(), {}, []
    for i, layer in enumerate(raw["layers"]):
        w = lambda name: W[f"l{i}.{name}"]  # noqa: B023, E731
        m, f = layer["mixer"], layer["mlp"]
        H, dk, dv, T = m["heads"], m["dim"], m["vdim"], len(ids)
        h = _rms(x, eps, 1.0 + w("norm1").double())
        if layer["type"] == "lightning":
            q, k, v = (torch.nn.functional.silu(_lin(h, w("mix." + n))).view(T, H, -1) for n in "qkv")
            decay = torch.tensor(m["decay"], dtype=torch.float64, device=x.device).expand(T, H)
            parts = [_recur(*s) for s in zip(*(_sequences(t, lengths) for t in (decay, k, v, q)))]
            out = _rms(torch.cat([o for o, _ in parts]).reshape(T, -1), eps, w("mix.norm"))
            states.append(torch.stack([S for _, S in parts]))
        else:
            rot = m.get("rot")
            turn = lambda t: torch.cat([_rotate(s, rot["dims"], rot["base"], True) for s in _sequences(t, lengths)]) if rot else t  # noqa: B023, E731
            q = turn(_rms(_lin(h, w("mix.q")), eps, w("mix.q.norm")).view(T, H, dk))
            if m.get("kv_from") is None:
                k = turn(_rms(_lin(h, w("mix.k")), eps, w("mix.k.norm")).view(T, -1, dk))
                held[i] = (k, _lin(h, w("mix.v")).view(T, -1, dv))
            kv = held[m.get("kv_from", i)]
            size = m["mask"]["size"]
            mask = {"window": size} if rot else {"run": size, "softcap": m.get("softcap")}
            out = torch.cat([_softmax_attention(*s, m["scale"], **mask) for s in zip(*(_sequences(t, lengths) for t in (q, *kv)))])
        if layer["type"] != "attention":
            out = out * torch.sigmoid(_lin(h, w("mix.g")))
        x = x + mult * _rms(_lin(out, w("mix.o")), eps, 1.0 + w("norm1b").double())
        h = _rms(x, eps, 1.0 + w("norm2").double())
        if f["kind"] == "dense":
            out = _lin(torch.relu(_lin(h, w("mlp.gate"))) * _lin(h, w("mlp.up")), w("mlp.down"))
        else:
            out, limit, chosen = torch.zeros_like(h), f["expert"]["limit"], w("mlp.table")[ids].long()
            for e in range(f["router"]["experts"]):
                at = (chosen == e).any(dim=1).nonzero()[:, 0]
                g = _lin(h[at], w(f"mlp.e{e}.gate")).clamp(max=limit)
                u = _lin(h[at], w(f"mlp.e{e}.up")).clamp(-limit, limit)
                out[at] += _lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), w(f"mlp.e{e}.down")) / f["router"]["top"]
        x = x + mult * _rms(out, eps, 1.0 + w("norm2b").double())
    return _lin(_rms(x[rows], eps, 1.0 + W["final.norm"].double()), W["embed"]) * raw["logit_scale"], [], states


def _gisudra_exact(raw, W, ids, lengths, rows):
    eps, T, first, states = raw["norm"]["eps"], len(ids), None, []
    x = W["embed"][ids].double()
    for i, layer in enumerate(raw["layers"]):
        w = lambda name: W[f"l{i}.{name}"].double()  # noqa: B023, E731
        m, H, dv = layer["mixer"], layer["mixer"]["heads"], layer["mixer"]["vdim"]
        h = _rms(x, eps, w("norm1"))
        if layer["type"] == "mamba2":
            N, inner, taps = m["state"], H * dv, m["conv"]
            z, xbc, dt = torch.split(_lin(h, w("mix.in")), [inner, inner + 2 * N, H], dim=-1)
            parts, kept = [], []
            for u, step in zip(_sequences(xbc, lengths), _sequences(dt, lengths)):
                padded = torch.nn.functional.pad(u, (0, 0, taps - 1, 0))
                conv = w("mix.conv.b") + sum(padded[j: j + len(u)] * w("mix.conv")[:, j] for j in range(taps))
                v, b, c = torch.split(torch.nn.functional.silu(conv), [inner, N, N], dim=-1)
                step = torch.nn.functional.softplus(step + w("mix.dt_bias"))
                v, heads = v.view(-1, H, dv), (len(u), H, N)
                y, S = _recur(torch.exp(-torch.exp(w("mix.A_log")) * step), b[:, None].expand(heads), step[..., None] * v, c[:, None].expand(heads))
                parts.append(y + w("mix.D")[:, None] * v)
                kept.append((S, padded[len(u):]))
            states += [torch.stack([S for S, _ in kept]), torch.stack([conv for _, conv in kept])]
            out = _rms(torch.cat(parts).reshape(T, inner) * torch.nn.functional.silu(z), eps, w("mix.norm"))
        elif layer["type"] == "attention":
            q, k = (_rms(_lin(h, w("mix." + n)).view(T, -1, m["dim"]), eps, w(f"mix.{n}.norm")) for n in "qk")
            v = _lin(h, w("mix.v")).view(T, -1, dv)
            first, v = (v, v) if first is None else (first, (1.0 - w("mix.vmix")) * v + w("mix.vmix") * first)
            out = torch.cat([_softmax_attention(*s, m["scale"], m["mask"]["size"], keep_first=m["mask"]["keep_first"])
                             for s in zip(*(_sequences(t, lengths) for t in (q, k, v)))])
        else:
            dk, rank, rot = m["dim"], m["kv_rank"], m["rot"]
            turn = lambda t: torch.cat([_rotate(s, rot["dims"], rot["base"], True) for s in _sequences(t, lengths)])  # noqa: B023, E731
            q, down = _lin(h, w("mix.q")).view(T, H, -1), _lin(h, w("mix.dkv"))
            latent = _rms(down[:, :rank], eps, w("mix.dkv.norm"))
            q = torch.cat([q[..., :dk], turn(q[..., dk:])], dim=-1)
            k = torch.cat([_lin(latent, w("mix.uk")).view(T, H, dk), turn(down[:, None, rank:]).expand(T, H, -1)], dim=-1)
            v = _lin(latent, w("mix.uv")).view(T, H, dv)
            out = torch.cat([_softmax_attention(*s, m["scale"], m["mask"]["size"]) for s in zip(*(_sequences(t, lengths) for t in (q, k, v)))])
        if layer["type"] != "mamba2":
            out = out * torch.sigmoid(_lin(h, w("mix.g")))
        x = x + _lin(out, w("mix.o"))
        h = _rms(x, eps, w("norm2"))
        x = x + _lin(torch.nn.functional.gelu(_lin(h, w("mlp.gate")), approximate="tanh") * _lin(h, w("mlp.up")), w("mlp.down"))
    return _lin(_rms(x[rows], eps, W["final.norm"]), W["head"]), [], states


def exact(case, seed):
    if case["kind"] == "sample":
        return None  # token ids
    raw, _, page = MODELS[case["model"]]
    bulk, tail, prompts, portion, steps = _layout(case)
    contexts, texts = _tokens(case, seed)
    sequences = contexts + texts
    lengths = [len(s) for s in sequences]
    head = _vocab(raw) * (raw["text_config"]["hidden_size"] if "text_config" in raw else raw["width"])
    weights = sum(fixed + top * expert for fixed, expert, _, top, *_ in _layers(raw))
    recurrent = sum(1 for layer in _layers(raw) if layer[7])
    if 2 * weights * sum(lengths) + 2 * head * len(lengths) > 3.5e14 or recurrent * sum(lengths) > 200000:
        return None
    starts = [sum(lengths[:i]) for i in range(len(lengths))]
    rows, per_step = [], []  # rows of all sequences whose logits a pass wants, step after step
    for step in range(steps):
        wanted = [starts[i] + b + t + step for i, (b, t) in enumerate(zip(bulk, tail))]
        for start, n in zip(starts[len(bulk):], prompts):
            lo, hi = step * portion, min(n, (step + 1) * portion)
            if lo < hi:
                wanted += list(range(start + lo, start + hi)) if case["all_logits"] else [start + hi - 1] if hi == n else []
        rows += wanted
        per_step.append(len(wanted))
    W = _weights(case["model"], seed)
    forward = {"muse_glimmer": _muse_exact, "Bobarax": _bobarax_exact, "Gisudra": _gisudra_exact}[
        raw.get("model_type") or raw["architecture"]]
    logits, kept, states = forward(raw, W, torch.tensor(sum(sequences, []), device="cuda"), lengths, torch.tensor(rows, device="cuda"))
    cache = []
    if kept and all(window is None for *_, window, _, _ in _layers(raw)):
        taken, first = [], len(bulk)  # (sequence, its first position, the place of its page) of every page a pass writes to
        taken += [(i, b, i) for i, b in enumerate(bulk)]
        for step in range(steps):  # the prompts take theirs as they are read
            for i, n in enumerate(prompts):
                lo, hi = (-(-min(n, s * portion) // page) for s in (step, step + 1))
                taken += [(len(bulk) + i, at * page, first + at - lo) for at in range(lo, hi)]
                first += hi - lo
        out = torch.zeros(len(kept), first, 2, kept[0].shape[2], page, kept[0].shape[3], dtype=torch.float64, device="cuda")
        for layer, kv in enumerate(kept):
            for i, at, place in taken:
                rows_ = kv[starts[i] + at: starts[i] + min(at + page, lengths[i])]
                out[layer, place, :, :, : len(rows_)] = rows_.permute(1, 2, 0, 3)
        cache = [out]
    return {"logits": list(torch.split(logits, per_step)), "cache": cache, "states": states}
