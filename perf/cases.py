"""What this engine is used for, as cases whose time can be taken and whose results can be checked.

A case names a model shape (the shapes of ``bench.py`` and ``xyntetik_runner_b200/measure_designs.py``), what one pass does
with it, and the sizes:

* ``prefill``: `requests` prompts of `tokens` tokens in all, each new to the engine, in ONE step that wants the logits behind
  every prompt; the requests end behind it.
* ``decode``: one token of each of `requests` requests that hold about `context` tokens already (really run, in ``prepare``).
  The step is given back at the end of the pass, so that every pass has the same positions.
* ``mixed``: a portion of `tokens` tokens of a prompt that is half run, beside one token of each of `requests` other requests.
* ``score``: ``Runner.score`` of one text of `tokens` tokens.

Weights are bfloat16, drawn from the seed, scaled as in trained models: a stream of about unit size to which every sublayer adds
a little, recurrences that remember hundreds of tokens, and routers that are decided.  The last is done by giving every token's
embedding the directions of the experts that it uses: with rows drawn independently, several layers' choices would hang on the
last bit of a sum, and two correct results could not be told from a wrong one.
"""
from __future__ import annotations

import math
import zlib

import torch

DEVICE = "cuda:0"

# ---- the shapes --------------------------------------------------------------------------------------------------------


def _llama(hidden, layers, heads, kv_heads, head_dim, inter, vocab, theta, scaling=None, tied=False):
    return {"architectures": ["LlamaForCausalLM"], "hidden_size": hidden, "num_hidden_layers": layers, "num_attention_heads": heads,
            "num_key_value_heads": kv_heads, "head_dim": head_dim, "intermediate_size": inter, "vocab_size": vocab, "rms_norm_eps": 1e-5,
            "rope_theta": theta, "rope_scaling": scaling, "max_position_embeddings": 8192, "tie_word_embeddings": tied,
            "torch_dtype": "bfloat16"}


def _turudra(W, la, ml, E, top, ff, sff):
    mlp = {"kind": "moe", "router": {"experts": E, "top": top}, "expert": {"ff": ff, "limit": 7.0}, "shared": {"ff": sff, "limit": 7.0}}
    latent = {"type": "latent_attention", "mlp": mlp,
              "mixer": dict(la, scale=(la["dim"] + la["rot_dim"]) ** -0.5, rot={"base": 10000.0, "dims": la["rot_dim"]})}
    mlstm = {"type": "mlstm", "mlp": mlp, "mixer": dict(ml, gate_cap=15.0)}
    return {"architecture": "Turudra", "vocab": 32000, "width": W, "embedding": {"scale": 1.0}, "residual_mult": 1.0,
            "norm": {"eps": 1e-5}, "logit_softcap": 30.0, "layers": [mlstm, latent, mlstm, latent], "loop": {"start": 1, "stop": 3, "times": 2}}


def _besolix(W, at, dl, la, ff):
    mlp = {"kind": "dense", "ff": ff}
    window = {"size": 1024}
    attention = {"type": "attention", "mlp": mlp,
                 "mixer": dict(at, scale=at["dim"] ** -0.5, rot={"base": 20000.0, "dims": at["dim"] // 2, "scaling": {"factor": 4.0}}, mask=window)}
    delta = {"type": "delta", "mlp": mlp, "mixer": dict(dl, conv=4)}
    lm = dict(la, scale=(la["dim"] + la["rot_dim"]) ** -0.5, rot={"base": 10000.0, "dims": la["rot_dim"]}, mask=window)
    return {"architecture": "Besolix", "vocab": 32000, "width": W, "norm": {"eps": 1e-5},
            "layers": [delta, {"type": "latent_attention", "mlp": mlp, "mixer": lm}, attention, delta,
                       {"type": "latent_attention", "mlp": mlp, "mixer": dict(lm, kv_from=1)}, attention]}


def _pitolix(W, H, G, every, ff):
    mlp = {"kind": "dense", "ff": ff}
    sizes = {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
    rotary = {"type": "attention_2", "mlp": mlp, "mixer": dict(sizes, rot={"base": 10000.0, "dims": 64})}
    sink = {"type": "attention", "mlp": mlp, "mixer": dict(sizes, q_temp={"coef": 0.1, "every": every})}
    return {"architecture": "Pitolix", "vocab": 32000, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5},
            "layers": [rotary, sink, rotary, sink], "loop": {"start": 1, "stop": 3, "times": 2}}


def _decays(heads):
    return [1.0 - 2.0 ** -(3 + 5.0 * h / max(heads - 1, 1)) for h in range(heads)]


def _buzarax(W, H, G, rh, R, B, ff, eff):
    dense = {"kind": "dense", "ff": ff, "limit": 7.0}
    moe = {"kind": "moe", "router": {"experts": 16, "top": 2}, "expert": {"ff": eff}}
    par = {"type": "parallel", "mixer": {
        "left": {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
                 "rot": {"base": 100000.0, "dims": 64, "scaling": {"factor": 16.0, "original": 8192, "fast": 16.0, "slow": 2.0}}},
        "right": {"heads": rh, "dim": 128, "vdim": 128, "decay": _decays(rh)}, "left_scale": 0.7, "right_scale": 0.9}}
    rec = {"type": "rglru", "mixer": {"width": R, "blocks": B, "conv": 4}}
    layers = [dict(par, mlp=dense), dict(rec, mlp=moe), dict(par, mlp=moe), dict(rec, mlp=dense), dict(par, mlp=dense), dict(rec, mlp=moe)]
    return {"architecture": "Buzarax", "vocab": 32000, "width": W, "norm": {"eps": 1e-5}, "logit_softcap": 30.0,
            "embedding": {"bigram": {"buckets": 65521, "mul_prev": 257, "mul_cur": 13}}, "layers": layers}


def _semesun(W, H, G, mh, ff, eff):
    dense = {"kind": "dense", "ff": ff}
    moe = {"kind": "moe", "router": {"experts": 12, "identity": 4, "top": 2, "groups": {"count": 4, "keep": 2}, "scale": 2.0},
           "expert": {"ff": eff, "limit": 7.0}}
    att = {"type": "attention", "mixer": {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "bias_max": 512,
                                          "v_mix": True, "mask": {"size": 1024, "keep_first": 4}}}
    rec = {"type": "mamba2", "mixer": {"heads": mh, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}}
    layers = [dict(att, mlp=dense), dict(rec, mlp=moe), dict(att, mlp=moe), dict(rec, mlp=dense), dict(att, mlp=dense), dict(rec, mlp=moe)]
    return {"architecture": "Semesun", "vocab": 32000, "width": W, "norm": {"eps": 1e-5}, "layers": layers}


def _lilalorn(W, H, G, rh, gh, eff):
    moe = {"kind": "moe", "router": {"experts": 16, "top": 2}, "expert": {"ff": eff}, "shared": {"ff": eff}}
    par = {"type": "parallel", "mlp": moe, "mixer": {
        "left": {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                 "rot": {"base": 200000.0, "dims": 128, "scaling": {"factor": 16.0, "low": 1.0, "high": 8.0, "original": 4096}}},
        "right": {"heads": rh, "dim": 128, "vdim": 128, "decay": _decays(rh)}, "left_scale": 0.7, "right_scale": 0.9}}
    gla = {"type": "gla", "mlp": moe, "mixer": {"heads": gh, "dim": 128, "vdim": 256, "tau": 12.0}}
    return {"architecture": "Lilalorn", "vocab": 32000, "width": W, "norm": {"eps": 1e-5}, "residual_mult": 0.7, "logit_scale": 0.8,
            "layers": [par, gla, par, gla, par, gla]}


_LLAMA3 = {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}
MODELS = {
    "llama-3-8b": _llama(4096, 32, 32, 8, 128, 14336, 128256, 500000.0),
    "llama-3.2-1b": _llama(2048, 16, 32, 8, 64, 8192, 128256, 500000.0, _LLAMA3, True),
    "turudra-w1024": _turudra(1024, dict(heads=8, dim=64, rot_dim=32, vdim=64, kv_rank=256), dict(heads=4, dim=128, vdim=256), 16, 2, 512, 1024),
    "turudra-w2048": _turudra(2048, dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512), dict(heads=8, dim=128, vdim=256), 64, 6, 1408, 2816),
    "besolix-w1024": _besolix(1024, dict(heads=8, kv_heads=2, dim=64, vdim=128), dict(heads=4, kv_heads=2, dim=128, vdim=128),
                              dict(heads=8, dim=64, rot_dim=32, vdim=64, kv_rank=256, q_rank=384), 2816),
    "besolix-w2048": _besolix(2048, dict(heads=16, kv_heads=4, dim=128, vdim=128), dict(heads=8, kv_heads=4, dim=128, vdim=256),
                              dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512, q_rank=768), 5632),
    "pitolix-w1024": _pitolix(1024, 8, 2, 512, 2816),
    "pitolix-w2048": _pitolix(2048, 16, 4, 1024, 5632),
    "buzarax-w1024": _buzarax(1024, 8, 2, 4, 1280, 5, 2816, 1408),
    "buzarax-w2048": _buzarax(2048, 16, 4, 8, 2560, 10, 5632, 2816),
    "semesun-w1024": _semesun(1024, 8, 2, 32, 4096, 1408),
    "semesun-w2048": _semesun(2048, 16, 4, 64, 8192, 2816),
    "lilalorn-w1024": _lilalorn(1024, 8, 2, 4, 4, 1408),
    "lilalorn-w2048": _lilalorn(2048, 16, 4, 8, 8, 2816),
}

# ---- the cases ---------------------------------------------------------------------------------------------------------


def _case(name, model, kind, tokens=0, requests=1, context=0, dtype="bfloat16"):
    c = {"name": name, "model": model, "kind": kind, "tokens": tokens, "requests": requests, "context": context, "dtype": dtype}
    return c if name else {k: v for k, v in c.items() if k != "name"}


def listed():
    return [
        # one conversation with a small model: latency, every launch counts
        _case("lilalorn-w1024-decode-1", "lilalorn-w1024", "decode", requests=1, context=300),
        _case("llama-3.2-1b-decode-1", "llama-3.2-1b", "decode", requests=1, context=640),
        # a server's step: a few long conversations, the benchmark's own workload
        _case("llama-3-8b-decode-8", "llama-3-8b", "decode", requests=8, context=8128),
        # a busy server's step with a recurrent model: many requests of different lengths
        _case("buzarax-w2048-decode-32", "buzarax-w2048", "decode", requests=32, context=640),
        # a server's step with experts and latent attention
        _case("turudra-w2048-decode-8", "turudra-w2048", "decode", requests=8, context=2000),
        # a long prompt in one step: the benchmark's prompt, the largest case
        _case("llama-3-8b-prefill-2048", "llama-3-8b", "prefill", tokens=2048),
        # the same for models of the other designs; several prompts at once, odd lengths
        _case("turudra-w2048-prefill-2048", "turudra-w2048", "prefill", tokens=2048),
        _case("buzarax-w2048-prefill-1901", "buzarax-w2048", "prefill", tokens=1901, requests=3),
        _case("semesun-w1024-prefill-777", "semesun-w1024", "prefill", tokens=777),
        _case("lilalorn-w2048-prefill-2048", "lilalorn-w2048", "prefill", tokens=2048),
        # a portion of a prompt beside requests that generate: what a scheduler's step looks like under load
        _case("besolix-w2048-mixed-512", "besolix-w2048", "mixed", tokens=505, requests=7, context=900),
        # scoring a text in true 32 bit: what a model's outputs are checked with
        _case("pitolix-w1024-score-float32", "pitolix-w1024", "score", tokens=300, dtype="float32"),
    ]


def draw(rng):
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    kind = rng.choice(["prefill", "prefill", "decode", "decode", "mixed", "score"])
    model = rng.choice([m for m in MODELS if m != "llama-3-8b" or kind != "score"])
    dtype = "float32" if kind == "score" and model.endswith("w1024") and rng.random() < 0.5 else "bfloat16"
    tokens, requests, context = log(24, 2040), log(1, 48), log(40, 4000)
    if kind == "decode":
        return _case(None, model, kind, requests=requests, context=min(context, 40000 // requests))
    if kind == "mixed":
        return _case(None, model, kind, tokens=tokens, requests=min(requests, 12), context=min(context, 1500))
    if kind == "score":
        return _case(None, model, kind, tokens=min(tokens, 600 if dtype == "bfloat16" else 320))
    return _case(None, model, kind, tokens=tokens, requests=min(requests, 1 + tokens // 40))


def _lengths(total, n):
    """`total` cut into `n` parts of different lengths, the same for every seed."""
    share = [1.0 + 0.9 * math.sin(2.4 * (i + 1)) for i in range(n)]
    out = [max(1, int(total * s / sum(share))) for s in share]
    out[-1] += total - sum(out)
    return out if min(out) >= 1 else [total // n + (i < total % n) for i in range(n)]


def _contexts(case):
    n = case["requests"]
    return [max(8, int(case["context"] * (1.0 - 0.4 * ((0.618 * i) % 1.0)))) for i in range(n)]


def _sequences(case, seed):
    """(what the requests hold before the pass, what the pass runs), lists of token lists."""
    vocab = _vocab(case["model"])
    g = torch.Generator().manual_seed(seed * 1000003 + 17)
    make = lambda n: torch.randint(0, vocab, (n,), generator=g).tolist()
    if case["kind"] in ("prefill", "score"):
        lens = _lengths(case["tokens"], case["requests"])
        return [[] for _ in lens], [make(n) for n in lens]
    held, run = [make(n) for n in _contexts(case)], [make(1) for _ in range(case["requests"])]
    if case["kind"] == "mixed":
        held, run = [make(case["tokens"])] + held, [make(case["tokens"])] + run
    return held, run


def _vocab(model):
    c = MODELS[model]
    return c.get("vocab") or c["vocab_size"]


def _width(model):
    c = MODELS[model]
    return c.get("width") or c["hidden_size"]


# ---- weights -----------------------------------------------------------------------------------------------------------


def _experts(config):
    """(router outputs, chosen) of the layers with experts, or None: the same in all of a model's layers."""
    for lay in config.get("layers", []):
        r = (lay.get("mlp") or {}).get("router")
        if r:
            return r["experts"] + r.get("identity", 0), r["top"]
    return None


class Weights:
    """The tensors of a model by name, each drawn from (seed, name) when it is asked for."""

    def __init__(self, model, seed):
        self.config, self.seed, self.width = MODELS[model], seed, _width(model)
        e = _experts(self.config)
        if e:
            self.outputs, self.top = e
            u = self._normal("directions", (self.outputs, self.width))
            self.directions = u / u.norm(dim=1, keepdim=True)
            coef = torch.linspace(1.0, 0.6, self.top, device=DEVICE)
            self.coef = 0.8 * coef / coef.norm() * self.width ** 0.5

    def _normal(self, name, shape):
        g = torch.Generator(device=DEVICE).manual_seed(zlib.crc32(("%d:%s" % (self.seed, name)).encode()))
        return torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32)

    def __call__(self, name, shape):
        last = name.rsplit(".", 1)[-1]
        x = self._normal(name, shape)
        if "norm" in last:
            one_plus = self.config.get("architecture") in ("Besolix", "Pitolix") and last in ("norm1", "norm2") or (
                self.config.get("architecture") in ("Besolix", "Pitolix") and name == "final.norm")
            x = 0.05 * x + (0.0 if one_plus else 1.0)
            if len(shape) == 0 and name != "final.norm":
                x = x * 0.15                                   # the norm behind a sublayer: what it adds to the stream
        elif last in ("layernorm", "input_layernorm", "post_attention_layernorm") or name.endswith("norm.weight") or "layernorm" in name:
            x = 1.0 + 0.05 * x
        elif name in ("embed", "model.embed_tokens.weight"):
            if _experts(self.config):
                which = self._normal("experts of tokens", (shape[0], self.outputs)).argsort(dim=1)[:, :self.top]
                x = 0.6 * x
                for j in range(self.top):
                    x += self.coef[j] * self.directions[which[:, j]]
            if self.config.get("tie_word_embeddings"):
                x = x * self.width ** -0.5 * 4.0               # (the head reads it too)
        elif name == "bigram":
            x = 0.2 * x
        elif last == "router":
            layer = int(name[1:].split(".")[0])
            x = 0.02 * x * self.width ** -0.5 + torch.roll(self.directions, layer, 0) * 6.0 / self.coef[0]
        elif name == "loop.in":
            eye = torch.eye(self.width, device=DEVICE)
            x = 0.1 * x * shape[1] ** -0.5 + torch.cat([0.6 * eye, 0.4 * eye], dim=1)
        elif last == "dwa":
            x = 0.02 * x + torch.tensor([0.1 / (shape[0] - 1)] * (shape[0] - 1) + [0.9], device=DEVICE)
        elif last == "A_log":
            x = 0.5 * x
        elif last in ("dt_bias", "lam"):
            x = 0.5 * x - 4.0
        elif name.endswith("f.b"):
            x = x + 4.0
        elif name.endswith("a2.b"):
            x = x + 2.0
        elif last == "D":
            x = 1.0 + 0.1 * x
        elif last == "vmix":
            x = 0.3 + 0.05 * x
        elif last == "conv":
            x = 0.5 * x
        elif last in ("b", "correction", "step", "rel", "sink"):
            x = {"b": 0.1, "correction": 0.01, "step": 0.1, "rel": 0.3, "sink": 0.5}[last] * x
        else:
            fan = shape[-1]
            gain = 0.4 if last in ("o", "down") or name.endswith(("o_proj.weight", "down_proj.weight")) else 2.0 if name in ("head", "lm_head.weight") else 1.0
            x = x * gain * fan ** -0.5
        return x.to(torch.bfloat16)


def _plan(model):
    from xyntetik_runner_b200.config import registry
    from xyntetik_runner_b200 import architectures  # noqa: F401  (registers them)
    c = MODELS[model]
    arch = registry.resolve(c.get("architecture") or c["architectures"][0])
    config = arch.config_from_dict(c)
    return config, arch.build_plan(config)


_SHAPES = {}


def _shapes(model):
    """{tensor name: shape} that the model's checkpoint holds."""
    if model not in _SHAPES:
        _SHAPES[model] = {n: tuple(s.shape) for n, s in _plan(model)[1].tensor_specs().items() if not s.optional}
    return _SHAPES[model]


# ---- a pass ------------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    from xyntetik_runner_b200 import Engine, EngineParams, Runner, StepEntry
    from xyntetik_runner_b200.weights.loader import TensorSource
    shapes, weights = _shapes(case["model"]), Weights(case["model"], seed)

    class Source(TensorSource):
        where = "drawn weights"

        def listing(self):
            return {n: (torch.bfloat16, s) for n, s in shapes.items()}

        def fetch(self, name, device):
            return weights(name, shapes[name]).to(device)

    config, _ = _plan(case["model"])
    held, run = _sequences(case, seed)
    longest = max(len(a) + len(b) for a, b in zip(held, run)) + 64
    pages = sum((len(a) + len(b) + 63) // 64 + 1 for a, b in zip(held, run))
    engine = Engine(params=EngineParams(dtype=case["dtype"], max_tokens=64 * pages, page_size=64, max_requests=len(run),
                                        max_request_tokens=(longest + 63) // 64 * 64, max_step_tokens=2048), config=config, source=Source())
    if case["kind"] == "score":
        return {"runner": Runner(engine=engine), "text": run[0]}
    for i, h in enumerate(held):
        for at in range(0, len(h), 2048):
            engine.step([StepEntry(i, h[at:at + 2048])])
    return {"engine": engine, "entries": [StepEntry(i, t, [len(t) - 1]) for i, t in enumerate(run)], "new": case["kind"] == "prefill"}


def run(state):
    if "runner" in state:
        return torch.tensor(state["runner"].score(state["text"]))
    engine, entries = state["engine"], state["entries"]
    if state["new"]:
        logits = engine.step(entries)
        for e in entries:
            engine.end(e.request)
        return logits
    logits = engine.step(entries, commit=False)
    engine.cancel_step(entries)
    return logits


# ---- what a pass cannot do without -------------------------------------------------------------------------------------


def _attention_layers(c):
    """(heads, key elements, value elements, cached elements a token, window) per run of an attention layer."""
    if "hidden_size" in c:
        H, G, D = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        return [(H, D, D, 2 * G * D, None)] * c["num_hidden_layers"]
    out = []
    for i in _order(c):
        lay = c["layers"][i]
        m = lay["mixer"].get("left", lay["mixer"])
        window = (m.get("mask") or {}).get("size")
        if lay["type"] == "latent_attention":
            out.append((m["heads"], m["dim"] + m["rot_dim"], m["vdim"], m["kv_rank"] + m["rot_dim"], window))
        elif lay["type"] in ("attention", "attention_2", "parallel"):
            out.append((m["heads"], m["dim"], m["vdim"], m["kv_heads"] * (m["dim"] + m["vdim"]), window))
    return out


def _states(c):
    """State elements (32 bit) of every run of a recurrent layer."""
    out = []
    for i in _order(c) if "layers" in c else []:
        lay = c["layers"][i]
        m = lay["mixer"]
        m = m.get("right", m)
        if lay["type"] in ("mlstm", "delta", "gla", "parallel"):
            out.append(m["heads"] * m["dim"] * m["vdim"])
        elif lay["type"] == "mamba2":
            out.append(m["heads"] * m["vdim"] * m["state"])
        elif lay["type"] == "rglru":
            out.append(m["width"])
    return out


def _order(c):
    """Layers in the order they run."""
    n, loop = len(c["layers"]), c.get("loop")
    if not loop:
        return list(range(n))
    a, b = loop["start"], loop["stop"]
    return list(range(a)) + list(range(a, b)) * loop["times"] + list(range(b, n))


def work(case):
    c, W, vocab = MODELS[case["model"]], _width(case["model"]), _vocab(case["model"])
    held, run_ = _sequences(case, 1)
    T = sum(len(t) for t in run_)
    rows = T - 1 if case["kind"] == "score" else len(run_)
    times = {i: _order(c).count(i) for i in range(len(c["layers"]))} if "layers" in c else {}
    e = _experts(c)
    nbytes = T * 8 + T * W * 2 + rows * (4 if case["kind"] == "score" else vocab * 4)
    flops = 2.0 * rows * vocab * W
    tied = c.get("tie_word_embeddings")
    for name, shape in _shapes(case["model"]).items():
        n = math.prod(shape)
        if name in ("embed", "bigram") or name == "model.embed_tokens.weight" and not tied:
            continue
        if name in ("head", "lm_head.weight", "model.embed_tokens.weight"):
            nbytes += 2 * n
            continue
        again = times.get(int(name[1:].split(".")[0]), 1) if name[0] == "l" and name[1].isdigit() else 1
        part = name.split(".")
        if e and len(part) > 2 and part[1] == "mlp" and part[2][0] == "e" and part[2][1:].isdigit():
            nbytes += 2 * n * min(1.0, T * e[1] / e[0])
            flops += again * 2.0 * n * T * e[1] / e[0]
            continue
        nbytes += 2 * n
        if len(shape) > 1:
            flops += again * 2.0 * n * T
    for H, D, V, kept, window in _attention_layers(c):
        for a, b in zip(held, run_):
            see = lambda p: min(p + 1, window or p + 1)
            flops += 2.0 * H * (D + V) * sum(see(len(a) + i) for i in range(len(b)))
            nbytes += (min(len(a), (window or len(a)) + len(b)) + len(b)) * kept * (2 if case["dtype"] == "bfloat16" else 4)
    for n in _states(c):
        flops += 4.0 * n * T
        nbytes += 4 * n * len(run_) * (1 if case["kind"] in ("prefill", "score") else 2)
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    # Four times what the outputs are off the 64-bit results: 0.002 to 0.004 for the six-layer models with bfloat16 activations, up
    # to 0.008 behind the 16 and 32 layers of the Llamas, 1e-7 to 4e-7 in 32 bit.
    if case["dtype"] == "float32":
        return {"rel": 2e-6, "max": 2e-5}
    return {"rel": 0.03, "max": 0.15} if case["model"].startswith("llama") else {"rel": 0.015, "max": 0.1}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------


def exact(case, seed):
    c = MODELS[case["model"]]
    held, run_ = _sequences(case, seed)
    T = sum(len(a) + len(b) for a, b in zip(held, run_))
    params = sum(math.prod(s) for n, s in _shapes(case["model"]).items() if "embed" not in n and n != "bigram")
    e = _experts(c)
    if T * params * 2.0 > 8e13 * (e[0] / e[1] if e else 1) or T * len(_states(c)) > 60000:
        return None                                       # over 20 seconds
    w = Weights(case["model"], seed)
    model = _Exact(c, w, _shapes(case["model"]), case["model"])
    texts = [a + b for a, b in zip(held, run_)]
    if case["kind"] == "score":
        logits = model.logits(texts[:1], [list(range(len(texts[0]) - 1))])
        return torch.log_softmax(logits, -1).gather(1, torch.tensor(texts[0][1:], device=DEVICE)[:, None])[:, 0].cpu()
    return model.logits(texts, [[len(t) - 1] for t in texts])


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _softplus(z):
    return torch.logaddexp(z, torch.zeros_like(z))


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _turn(v, freq, mult=1.0, adjacent=False, back=False):
    """v [T, heads, D]: the first 2 len(freq) elements in pairs (i, i + half) or (2i, 2i + 1), turned by position * freq."""
    half = len(freq)
    ang = torch.arange(v.shape[0], device=DEVICE, dtype=v.dtype)[:, None, None] * freq
    cos, sin = torch.cos(ang) * mult, torch.sin(ang) * (-mult if back else mult)
    out = v.clone()
    i = torch.arange(half, device=DEVICE)
    a, b = (2 * i, 2 * i + 1) if adjacent else (i, i + half)
    out[..., a] = v[..., a] * cos - v[..., b] * sin
    out[..., b] = v[..., b] * cos + v[..., a] * sin
    return out


def _freq(dims, base, dtype=torch.float64):
    return base ** (-2.0 * torch.arange(dims // 2, device=DEVICE, dtype=dtype) / dims)


def _yarn(dims, base, s):
    f = _freq(dims, base)
    where = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    lo, hi = max(math.floor(where(s["fast"])), 0), min(math.ceil(where(s["slow"])), dims - 1)
    ramp = torch.clamp((torch.arange(dims // 2, device=DEVICE) - lo) / max(hi - lo, 0.001), 0, 1)
    return f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _long_waves(f, factor, low, high, original):
    """Frequencies that turn fewer than `low` times over `original` positions divided by `factor`, more than `high` kept."""
    turns = original * f / (2 * math.pi)
    s = ((turns - low) / (high - low)).clamp(0, 1)
    return (1 - s) * f / factor + s * f


def _attend(q, k, v, scale, window=None, keep=0, sink=None, cap=None, bias=None):
    """q [T, H, D], k [T, G, D], v [T, G, V] -> [T, H, V], queries in blocks.  `sink` [H]: exp of it joins the denominator;
    `bias` [H, T]: added by distance."""
    T, H = q.shape[:2]
    rep = H // k.shape[1]
    out = []
    j = torch.arange(T, device=DEVICE)
    for at in range(0, T, 512):
        i = torch.arange(at, min(T, at + 512), device=DEVICE)
        o = []
        for h in range(H):
            s = (q[i, h] @ k[:, h // rep].T) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            far = i[:, None] - j[None, :]
            if bias is not None:
                s = s + bias[h][far.clamp(min=0)]
            see = far >= 0
            if window:
                see &= (far < window) | (j[None, :] < keep)
            s = s.masked_fill(~see, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[h].expand(len(i), 1)], dim=1)
            o.append(torch.softmax(s, dim=-1)[:, :T] @ v[:, h // rep])
        out.append(torch.stack(o, dim=1))
    return torch.cat(out)


def _walk(q, k, v, decay):
    """S <- decay S + k v^T, o = S^T q.  q, k [T, H, D], v [T, H, V], decay [T, H, 1] or [T, H, D]."""
    S = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=q.dtype, device=DEVICE)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S.mul_(decay[t][:, :, None]).baddbmm_(k[t][:, :, None], v[t][:, None, :])
        torch.bmm(q[t][:, None, :], S, out=out[t][:, None, :])
    return out


def _conv(z, taps, bias=None):
    T, K = z.shape[0], taps.shape[1]
    out = torch.zeros_like(z) if bias is None else bias.expand(T, -1).clone()
    for j in range(min(K, T)):
        out[j:] += z[:T - j] * taps[:, K - 1 - j]
    return out


class _Exact:
    """The seven decoders on whole sequences, in float64, from their definitions."""

    def __init__(self, c, weights, shapes, model):
        self.c, self.weights, self.shapes, self.W = c, weights, shapes, _width(model)
        self.arch = c.get("architecture", "Llama")
        self.eps = c["rms_norm_eps"] if "hidden_size" in c else c["norm"]["eps"]

    def w(self, name):
        return self.weights(name, self.shapes[name]).double()

    def lin(self, h, name):
        return h @ self.w(name).T

    def norm(self, x, name):
        one_plus = self.arch in ("Besolix", "Pitolix") and (name.endswith(("norm1", "norm2")) or name == "final.norm")
        return _unit(x, self.eps) * (self.w(name) + (1.0 if one_plus else 0.0))

    def logits(self, texts, wanted):
        """All texts go through a layer together, so that its weights are drawn once."""
        c = self.c
        ids = [torch.tensor(t, device=DEVICE) for t in texts]
        at = [0]
        for t in texts:
            at.append(at[-1] + len(t))
        self.spans = list(zip(at[:-1], at[1:]))
        table = self.weights("model.embed_tokens.weight" if self.arch == "Llama" else "embed",
                             self.shapes["model.embed_tokens.weight" if self.arch == "Llama" else "embed"])
        x = table[torch.cat(ids)].double()
        if self.arch == "Buzarax":
            pair, b = self.weights("bigram", self.shapes["bigram"]), c["embedding"]["bigram"]
            n = pair.shape[0] - 1
            rows = [torch.cat([torch.tensor([n], device=DEVICE), (t[:-1] * b["mul_prev"] + t[1:] * b["mul_cur"]) % n]) for t in ids]
            x = x + pair[torch.cat(rows)].double()
            del pair
        del table
        if self.arch == "Llama":
            for i in range(c["num_hidden_layers"]):
                x = self.llama_layer(x, i)
        else:
            x = self.layers(x)
        rows = torch.cat([torch.tensor([a + p for p in ps], device=DEVICE) for (a, _), ps in zip(self.spans, wanted)])
        name = ("model.embed_tokens.weight" if c.get("tie_word_embeddings") else "lm_head.weight") if self.arch == "Llama" else "head"
        out = self.lin(self.norm(x[rows], "model.norm.weight" if self.arch == "Llama" else "final.norm"), name) * c.get("logit_scale", 1.0)
        cap = c.get("logit_softcap")
        return cap * torch.tanh(out / cap) if cap else out

    def by_text(self, fn, *tensors):
        return torch.cat([fn(*(t[a:b] for t in tensors)) for a, b in self.spans])

    def layers(self, x):
        c, x0, self.kept = self.c, x, {}
        streams, seen = [x], {}
        for n, i in enumerate(_order(c)):
            lay, p, mult = c["layers"][i], "l%d." % i, c.get("residual_mult", 1.0)
            loop = c.get("loop")
            if loop and i == loop["start"]:
                t = seen.get(i, 0)
                seen[i] = t + 1
                if self.arch == "Turudra":
                    x = self.lin(torch.cat([x, x0], dim=1), "loop.in")
                else:
                    x = x + (x0 if t > 0 else 0.0) + self.w("loop.step")[t]
            mix = getattr(self, lay["type"])
            if self.arch == "Turudra":
                h = self.norm(x, p + "norm1")
                x = x + mult * (mix(h, p + "mix.", lay["mixer"]) + self.feed(h, p + "mlp.", lay["mlp"]))
            elif self.arch == "Pitolix":
                x = x + mix(self.norm(x, p + "norm1"), p + "mix.", lay["mixer"]) + self.feed(self.norm(x, p + "norm2"), p + "mlp.", lay["mlp"])
            elif self.arch == "Buzarax":
                x = x + self.norm(mix(x, p + "mix.", lay["mixer"]), p + "norm1")
                x = x + self.norm(self.feed(x, p + "mlp.", lay["mlp"]), p + "norm2")
                streams.append(x)
                x = sum(a * s for a, s in zip(self.w(p + "dwa"), streams))
            else:
                x = x + mult * mix(self.norm(x, p + "norm1"), p + "mix.", lay["mixer"])
                x = x + mult * self.feed(self.norm(x, p + "norm2"), p + "mlp.", lay["mlp"])
        return x

    def llama_layer(self, x, i):
        c, p = self.c, "model.layers.%d." % i
        H, G, D = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        f, s = _freq(D, c["rope_theta"]), c["rope_scaling"]
        if s:
            f = _long_waves(f, s["factor"], s["low_freq_factor"], s["high_freq_factor"], s["original_max_position_embeddings"])
        h = self.norm(x, p + "input_layernorm.weight")
        q, k, v = (self.lin(h, p + "self_attn.%s_proj.weight" % n).view(len(h), -1, D) for n in "qkv")
        o = self.by_text(lambda q, k, v: _attend(_turn(q, f), _turn(k, f), v, D ** -0.5), q, k, v)
        x = x + self.lin(o.reshape(len(h), H * D), p + "self_attn.o_proj.weight")
        h = self.norm(x, p + "post_attention_layernorm.weight")
        return x + self.lin(_silu(self.lin(h, p + "mlp.gate_proj.weight")) * self.lin(h, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight")

    # mixers
    def heads(self, h, p, m, names="qkv"):
        G = m.get("kv_heads", m["heads"])
        sizes = {"q": (m["heads"], m["dim"]), "k": (G, m["dim"]), "v": (G, m["vdim"])}
        return [self.lin(h, p + n).view(len(h), *sizes[n]) for n in names]

    def attention(self, h, p, m):
        q, k, v = self.heads(h, p, m)
        T, window = len(h), (m.get("mask") or {}).get("size")
        if self.arch == "Pitolix":
            q, k, t = _unit(q, self.eps), _unit(k, self.eps), m["q_temp"]
            def one(q, k, v):
                pos = torch.arange(len(q), device=DEVICE)
                temp = 1.0 + t["coef"] * torch.log(((pos + 1) // t["every"]).double() + 1.0)
                return _attend(q * temp[:, None, None], k, v, m["scale"], sink=self.w(p + "sink"))
            o = self.by_text(one, q, k, v).reshape(T, -1)
            return self.lin(o * torch.sigmoid(self.lin(h, p + "g")), p + "o")
        q, k = self.norm(q, p + "q.norm"), self.norm(k, p + "k.norm")
        if self.arch == "Besolix":
            r = m["rot"]
            f = _freq(r["dims"], r["base"]) / r["scaling"]["factor"]
            o = self.by_text(lambda q, k, v: _attend(_turn(q, f, adjacent=True), _turn(k, f, adjacent=True), v, m["scale"], window), q, k, v)
            return self.lin(o.reshape(T, -1), p + "o")
        if "v" not in self.kept:
            self.kept["v"] = v
        else:
            lam = self.w(p + "vmix")
            v = (1.0 - lam) * v + lam * self.kept["v"]
        rel = self.w(p + "rel")
        n, half = rel.shape[0], rel.shape[0] // 2
        far = torch.arange(max(b - a for a, b in self.spans), device=DEVICE)
        step = torch.log(far.clamp(min=1).double() / half) / math.log(m["bias_max"] / half) * (n - half) + 1e-9
        bias = rel[torch.where(far < half, far, (half + step.floor().long()).clamp(max=n - 1))].T
        o = self.by_text(lambda q, k, v: _attend(q, k, v, m["scale"], window, m["mask"]["keep_first"], bias=bias), q, k, v)
        return self.lin(o.reshape(T, -1), p + "o")

    def attention_2(self, h, p, m):
        q, k, v = (t + self.w(p + n + ".b").view(t.shape[1:]) for t, n in zip(self.heads(h, p, m), "qkv"))
        f = _freq(m["rot"]["dims"], m["rot"]["base"])
        o = self.by_text(lambda q, k, v: _attend(_turn(q, f), _turn(k, f), v, m["scale"]), q, k, v)
        return self.lin((o * torch.sigmoid(self.lin(h, p + "g"))[:, :, None]).reshape(len(h), -1), p + "o")

    def latent_attention(self, h, p, m):
        T, C, D, adjacent = len(h), m["kv_rank"], m["dim"], self.arch == "Besolix"
        f, window = _freq(m["rot"]["dims"], m["rot"]["base"]), (m.get("mask") or {}).get("size")
        q = self.lin(h, p + "q") if not adjacent else self.lin(self.norm(self.lin(h, p + "dq"), p + "dq.norm"), p + "uq")
        q = q.view(T, m["heads"], -1)
        if m.get("kv_from") is None:
            down = self.lin(h, p + "dkv")
            self.kept["rows"] = self.norm(down[:, :C], p + "dkv.norm"), down[:, C:]
        latent, kr = self.kept["rows"]
        k, v = self.lin(latent, p + "uk").view(T, m["heads"], D), self.lin(latent, p + "uv").view(T, m["heads"], -1)
        def one(q, k, kr, v):
            kr = _turn(kr[:, None, :], f, adjacent=adjacent).expand(-1, m["heads"], -1)
            q = torch.cat([q[..., :D], _turn(q[..., D:], f, adjacent=adjacent)], dim=-1)
            return _attend(q, torch.cat([k, kr], dim=-1), v, m["scale"], window)
        o = self.by_text(one, q, k, kr, v)
        g = torch.sigmoid(self.lin(h, p + "g"))
        o = o * (g.view(o.shape) if adjacent else g[:, :, None])
        return self.lin(o.reshape(T, -1), p + "o")

    def mlstm(self, h, p, m):
        T, H, cap = len(h), m["heads"], m["gate_cap"]
        q, k, v = self.heads(h, p, m)
        q = q * m["dim"] ** -0.5
        ig = cap * torch.tanh((self.lin(h, p + "i") + self.w(p + "i.b")) / cap)
        fg = -_softplus(-cap * torch.tanh((self.lin(h, p + "f") + self.w(p + "f.b")) / cap))
        def one(q, k, v, ig, fg):
            mx, dec, inp, tops = torch.zeros(H, device=DEVICE, dtype=q.dtype), [], [], []
            for t in range(len(q)):
                new = torch.maximum(fg[t] + mx, ig[t])
                dec.append(torch.exp(fg[t] + mx - new))
                inp.append(torch.exp(ig[t] - new))
                tops.append(new)
                mx = new
            # the value 1 beside v carries the normaliser's sum
            k, v = k * torch.stack(inp)[:, :, None], torch.cat([v, torch.ones_like(v[..., :1])], dim=-1)
            o = _walk(q, k, v, torch.stack(dec)[:, :, None])
            return o[..., :-1] / (torch.maximum(o[..., -1:].abs(), torch.exp(-torch.stack(tops))[:, :, None]) + 1e-6)
        o = _unit(self.by_text(one, q, k, v, ig, fg), self.eps).reshape(T, -1) * self.w(p + "norm")
        return self.lin(o * torch.sigmoid(self.lin(h, p + "g")), p + "o")

    def delta(self, h, p, m):
        T, H, G, D, V = len(h), m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (self.by_text(lambda z: _silu(_conv(z, self.w(p + n + ".conv"))), self.lin(h, p + n)) for n in "qkv")
        q, k = (z.view(T, G, D) / torch.sqrt((z.view(T, G, D) ** 2).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        q, k, v = (q * D ** -0.5).repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1), v.view(T, H, V)
        beta = torch.sigmoid(self.lin(h, p + "b"))
        decay = torch.exp(-torch.exp(self.w(p + "A_log")) * _softplus(self.lin(h, p + "a") + self.w(p + "dt_bias")))
        def one(q, k, v, beta, decay):
            S, out = torch.zeros(H, D, V, dtype=q.dtype, device=DEVICE), torch.empty_like(v)
            for t in range(len(q)):
                S.mul_(decay[t][:, None, None])
                u = beta[t][:, None, None] * (v[t][:, None, :] - torch.bmm(k[t][:, None, :], S))
                S.baddbmm_(k[t][:, :, None], u)
                torch.bmm(q[t][:, None, :], S, out=out[t][:, None, :])
            return out
        o = self.by_text(one, q, k, v, beta, decay)
        o = _unit(o, self.eps) * self.w(p + "norm") * _silu(self.lin(h, p + "g")).view(T, H, V)
        return self.lin(o.reshape(T, H * V), p + "o")

    def parallel(self, h, p, m):
        T, l, r = len(h), m["left"], m["right"]
        q, k, v = self.heads(h, p + "left.", l)
        rot = l["rot"]
        if self.arch == "Buzarax":
            f, mult = _yarn(rot["dims"], rot["base"], rot["scaling"])
            vf = _freq(l["vdim"], rot["base"])
            def one(q, k, v):
                q, k = _unit(_turn(q, f, mult), self.eps), _unit(_turn(k, f, mult), self.eps)
                sink = torch.zeros(l["heads"], dtype=q.dtype, device=DEVICE)
                return _turn(_attend(q, k, _turn(v, vf), l["scale"], sink=sink, cap=l["softcap"]), vf, back=True)
        else:
            s = rot["scaling"]
            f = _long_waves(_freq(rot["dims"], rot["base"]), s["factor"], s["low"], s["high"], s["original"])
            def one(q, k, v):
                return _attend(_turn(q, f), _turn(k, f), v, l["scale"])
        left = self.lin(self.by_text(one, q, k, v).reshape(T, -1), p + "left.o")
        q, k, v = self.heads(h, p + "right.", r)
        g = self.lin(h, p + "right.g")
        q, k, v = (_silu(q), _silu(k), _silu(v)) if self.arch == "Buzarax" else (q, k * r["dim"] ** -0.5, v)
        decay = torch.tensor(r["decay"], dtype=h.dtype, device=DEVICE)[None, :, None].expand(T, -1, -1)
        o = self.by_text(_walk, q, k, v, decay)
        if self.arch == "Buzarax":
            o = self.norm(o.reshape(T, -1), p + "right.norm") * torch.sigmoid(g)
        else:
            o = _unit(o, self.eps).reshape(T, -1) * _silu(g)
        return m["left_scale"] * left + m["right_scale"] * self.lin(o, p + "right.o")

    def gla(self, h, p, m):
        q, k, v = self.heads(h, p, m)
        z = self.lin(self.lin(h, p + "a1"), p + "a2") + self.w(p + "a2.b")
        decay = torch.exp(-_softplus(-z) / m["tau"]).view(q.shape)
        o = self.norm(self.by_text(_walk, q * m["dim"] ** -0.5, k, v, decay), p + "norm").reshape(len(h), -1)
        return self.lin(o * _silu(self.lin(h, p + "g")), p + "o")

    def rglru(self, h, p, m):
        T, R, B = len(h), m["width"], m["blocks"]
        y = _gelu(self.lin(h, p + "y") + self.w(p + "y.b"))
        u = self.by_text(lambda z: _conv(z, self.w(p + "conv"), self.w(p + "conv.b")), self.lin(h, p + "x") + self.w(p + "x.b"))
        r, i = (torch.sigmoid(torch.einsum("boi,tbi->tbo", self.w(p + n), u.view(T, B, -1)) + self.w(p + n + ".b")).reshape(T, R) for n in ("ra", "ri"))
        a = torch.exp(-8.0 * r * _softplus(self.w(p + "lam")))
        inp = torch.sqrt(1.0 - a * a) * i * u
        def one(a, inp):
            S, out = torch.zeros(R, dtype=a.dtype, device=DEVICE), torch.empty_like(a)
            for t in range(len(a)):
                S = torch.addcmul(inp[t], a[t], S, out=out[t])
            return out
        return self.lin(self.by_text(one, a, inp) * y, p + "o")

    def mamba2(self, h, p, m):
        T, H, V, N, G = len(h), m["heads"], m["vdim"], m["state"], m["groups"]
        z, xbc, dt = torch.split(self.lin(h, p + "in"), [H * V, H * V + 2 * G * N, H], dim=-1)
        xbc = self.by_text(lambda t: _silu(_conv(t, self.w(p + "conv"), self.w(p + "conv.b"))), xbc)
        x, b, q = torch.split(xbc, [H * V, G * N, G * N], dim=-1)
        x, b, q = x.view(T, H, V), b.view(T, G, N).repeat_interleave(H // G, 1), q.view(T, G, N).repeat_interleave(H // G, 1)
        dt = _softplus(dt + self.w(p + "dt_bias"))
        a = torch.exp(-torch.exp(self.w(p + "A_log")) * dt)
        y = self.by_text(_walk, q, b * dt[:, :, None], x, a[:, :, None]) + self.w(p + "D")[:, None] * x
        y = (y.reshape(T, -1) * _silu(z)).view(T, m["norm_groups"], -1)
        return self.lin(_unit(y, self.eps).reshape(T, -1) * self.w(p + "norm"), p + "o")

    # feed-forwards
    def clamped(self, h, p, limit):
        g, u = self.lin(h, p + "gate").clamp(max=limit), self.lin(h, p + "up").clamp(-limit, limit)
        return self.lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), p + "down")

    def relu2(self, h, p):
        return self.lin(torch.relu(self.lin(h, p + "up")) ** 2, p + "down")

    def gated(self, h, p, act):
        return self.lin(act(self.lin(h, p + "gate")) * self.lin(h, p + "up"), p + "down")

    def feed(self, h, p, f):
        if f["kind"] == "dense":
            if self.arch == "Buzarax":
                return self.clamped(h, p, f["limit"])
            return self.relu2(h, p) if self.arch == "Semesun" else self.gated(h, p, _gelu if self.arch == "Besolix" else _silu)
        r = f["router"]
        z = self.lin(h, p + "router")
        if self.arch == "Turudra":
            best, chosen = torch.topk(z, r["top"], dim=-1)
            weight = torch.softmax(best, dim=-1)
        elif self.arch == "Buzarax":
            s = torch.sigmoid(z)
            chosen = torch.topk(s + self.w(p + "correction"), r["top"], dim=-1).indices
            weight = s.gather(1, chosen)
        elif self.arch == "Semesun":
            s, g = torch.softmax(z, dim=-1), r["groups"]
            by = s + self.w(p + "correction")
            best = torch.topk(by.view(len(h), g["count"], -1).max(dim=-1).values, g["keep"], dim=-1).indices
            allowed = torch.zeros(len(h), g["count"], dtype=torch.bool, device=DEVICE).scatter_(1, best, True)
            chosen = torch.topk(by.masked_fill(~allowed.repeat_interleave(by.shape[1] // g["count"], 1), float("-inf")), r["top"], dim=-1).indices
            weight = s.gather(1, chosen) * r["scale"]
        else:
            s = torch.softmax(z, dim=-1)
            weight, chosen = torch.topk(s, r["top"], dim=-1)
            weight = weight / (weight.sum(dim=-1, keepdim=True) + 1e-20)
        out = torch.zeros_like(h)
        for e in range(r["experts"] + r.get("identity", 0)):
            t, j = (chosen == e).nonzero(as_tuple=True)
            if len(t) == 0:
                continue
            q = p + "e%d." % e
            if e >= r["experts"]:
                y = h[t]
            elif self.arch == "Buzarax":
                y = self.gated(h[t], q, _silu)
            else:
                y = self.relu2(h[t], q) if self.arch == "Lilalorn" else self.clamped(h[t], q, f["expert"]["limit"])
            out.index_add_(0, t, weight[t, j][:, None] * y)
        if self.arch == "Turudra":
            out = out + self.clamped(h, p + "shared.", f["shared"]["limit"])
        elif self.arch == "Lilalorn":
            out = out + torch.sigmoid(self.lin(h, p + "shared.sg")) * self.relu2(h, p + "shared.")
        return out
