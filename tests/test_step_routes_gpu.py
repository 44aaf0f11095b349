"""The routes that a step's size chooses between, through the engine: recurrences in chunks or token by token, latent attention over expanded
keys or over the latent rows, experts on pairs of CTAs or on padded tiles, the choice of experts of a few tokens in one launch or in four.

A step that mixes single tokens, short portions and one long portion, then steps of single tokens, run once with the new route and once with
the other; both against the true 32-bit engine on the same weights.  The route changes where bfloat16 roundings fall, so its error may
differ from the other's, but a wrong row, slice or buffer moves an output by its own size.  Every expert is chosen (`top` = experts), so that
no rounding turns a choice."""
import numpy as np
import pytest
import torch

from xyntetik_runner_b200 import kernels
from xyntetik_runner_b200.config import registry
from xyntetik_runner_b200.engine.engine import EngineParams, StepEntry, random_engine
from xyntetik_runner_b200.parts import chunks, latent_attention, moe

pytestmark = pytest.mark.gpu

LATENT = dict(heads=8, dim=64, rot_dim=32, vdim=64, kv_rank=256, scale=0.1)
MOE = {"kind": "moe", "router": {"experts": 2, "top": 2}, "expert": {"ff": 64, "limit": 7.0}, "shared": {"ff": 64, "limit": 7.0}}
DENSE = {"kind": "dense", "ff": 64}


def turudra():
    return {"architecture": "Turudra", "vocab": 300, "width": 128, "embedding": {"scale": 1.0}, "residual_mult": 1.0, "norm": {"eps": 1e-5},
            "logit_softcap": 30.0, "loop": None,
            "layers": [{"type": "latent_attention", "mlp": MOE, "mixer": dict(LATENT, rot={"base": 10000.0, "dims": 32})},
                       {"type": "mlstm", "mlp": MOE, "mixer": dict(heads=2, dim=64, vdim=64, gate_cap=15.0)},
                       {"type": "latent_attention", "mlp": None, "mixer": dict(LATENT, rot={"base": 10000.0, "dims": 32})}]}


def besolix():
    """An output gate an element, a window, and a layer that reads the rows of another through a longer one."""
    m = dict(LATENT, q_rank=96, rot={"base": 10000.0, "dims": 32})
    return {"architecture": "Besolix", "vocab": 300, "width": 128, "norm": {"eps": 1e-5},
            "layers": [{"type": "latent_attention", "mlp": DENSE, "mixer": dict(m, mask={"size": 700})},
                       {"type": "latent_attention", "mlp": DENSE, "mixer": dict(m, mask={"size": 900}, kv_from=0)},
                       {"type": "attention", "mlp": DENSE,
                        "mixer": dict(heads=2, kv_heads=1, dim=64, vdim=64, scale=0.1, rot={"base": 10000.0, "dims": 32}, mask={"size": 400})}]}


def lilalorn():
    m = {"kind": "moe", "router": {"experts": 2, "top": 2}, "expert": {"ff": 64}, "shared": {"ff": 64}}
    par = {"left": {"heads": 2, "kv_heads": 1, "dim": 64, "vdim": 64, "scale": 0.1, "rot": {"base": 10000.0, "dims": 64}},
           "right": {"heads": 2, "dim": 64, "vdim": 64, "decay": [0.97, 0.995]}, "left_scale": 0.7, "right_scale": 0.9}
    return {"architecture": "Lilalorn", "vocab": 300, "width": 128, "norm": {"eps": 1e-5}, "residual_mult": 0.7, "logit_scale": 0.8,
            "layers": [{"type": "parallel", "mlp": m, "mixer": par}, {"type": "gla", "mlp": m, "mixer": dict(heads=2, dim=64, vdim=128, tau=12.0)}]}


# what is counted, what turns the route off
ROUTES = {
    "expanded keys": (lambda c: c["flat"], lambda p: p.setattr(latent_attention, "USE_FLAT", False)),
    "chunks": (lambda c: c["chunks"], lambda p: p.setattr(chunks, "CHUNKED_FROM", {k: 1 << 30 for k in chunks.CHUNKED_FROM})),
    "pairs": (lambda c: c["pairs"], lambda p: p.setattr(moe, "PAIRS_FROM", 1 << 20)),
    "few": (lambda c: c["few"], lambda p: p.setattr(moe, "FEW_TOKENS", 0)),
}
CASES = [("turudra", "expanded keys"), ("turudra", "chunks"), ("turudra", "pairs"), ("turudra", "few"), ("besolix", "expanded keys"),
         ("lilalorn", "chunks"), ("lilalorn", "pairs"), ("lilalorn", "few")]
MODELS = {"turudra": turudra, "besolix": besolix, "lilalorn": lilalorn}


def run(model, dtype, monkeypatch=None):
    """Logits of the mixed step and of four steps of single tokens behind it, and how often each route was taken."""
    c = MODELS[model]()
    arch = registry.resolve(c["architecture"])
    eng = random_engine(arch.config_from_dict(c), 5, EngineParams(dtype=dtype, max_tokens=64 * 80, page_size=64, max_requests=8, max_request_tokens=2048,
                                                                  max_step_tokens=2048), std=0.08)
    rng = np.random.RandomState(1)
    tok = lambda n: [int(t) for t in rng.randint(0, 300, n)]
    taken = {"flat": -latent_attention.counters["flat"], "chunks": 0, "pairs": 0, "few": 0}
    if monkeypatch is not None:
        def count(name, key, when):
            fn = getattr(kernels, name)
            monkeypatch.setattr(kernels, name, lambda *a, **k: (taken.__setitem__(key, taken[key] + bool(when(k))), fn(*a, **k))[1])
        for name in ("mlstm", "decay_attention", "key_decay_attention"):
            count(name, "chunks", lambda k: k.get("scratch") is not None)
        count("gemm_tc_grouped_pairs", "pairs", lambda k: True)
        count("route_few", "few", lambda k: True)
    held = {"s0": 90, "long": 300, "s1": 5, "short": 150, "s2": 400}
    for r, n in held.items():
        eng.step([StepEntry(r, tok(n))])
    out = [eng.step([StepEntry("s0", tok(1), [0]), StepEntry("long", tok(1000), [0, 63, 64, 500, 999]), StepEntry("s1", tok(1), [0]),
                     StepEntry("short", tok(20), [0, 19]), StepEntry("s2", tok(1), [0])]).clone()]
    for _ in range(4):
        out.append(eng.step([StepEntry(r, tok(1), [0]) for r in held]).clone())
    eng.check_status()
    taken["flat"] += latent_attention.counters["flat"]
    return torch.cat(out).double().cpu(), taken


_exact = {}


@pytest.mark.parametrize("model,route", CASES)
def test_either_route_through_the_engine(model, route, monkeypatch):
    if model not in _exact:
        _exact[model] = run(model, "float32")[0]
    want = _exact[model]
    counted, off = ROUTES[route]
    if route == "pairs" and not kernels.pairs_available():
        pytest.skip("no pairs of CTAs on this device")
    with monkeypatch.context() as p:
        got, taken = run(model, "bfloat16", p)
    with monkeypatch.context() as p:
        off(p)
        other, other_taken = run(model, "bfloat16", p)
    assert counted(taken) > 0 and counted(other_taken) == 0, (taken, other_taken)
    assert got.shape == want.shape == (10 + 20, 300)
    # row by row, against the row's own size: a route's roundings are as many and as large as the other's, and no row is worse than a few times
    # the worst of either
    err = lambda x: (x - want).norm(dim=1) / want.norm(dim=1)
    assert err(other).max() < 0.05 and err(got).max() < 0.05
    assert err(got).median() < 1.5 * err(other).median() + 1e-4
