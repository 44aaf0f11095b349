"""What a step works out once.

A step whose capture made a buffer runs again plainly: work that a step does once (a sum that starts at zero) was only recorded
by the capture and must be done by the run that counts.  And an answer
of None is an answer: no layer works it out again."""
import contextlib

import torch

from xyntetik_runner_b200.engine.engine import Engine, StepContext


def test_a_discarded_capture_leaves_nothing_behind(monkeypatch):
    class Graph:
        def replay(self):
            raise AssertionError("a graph with a stale address was replayed")

    monkeypatch.setattr(torch.cuda, "CUDAGraph", Graph)
    monkeypatch.setattr(torch.cuda, "graph", lambda g: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    eng = object.__new__(Engine)
    eng.device, eng._graphs, eng._graph_launches, eng._buf_generation, eng.graph_replays = "cpu", {}, {}, 0, 0
    ctx = object.__new__(StepContext)
    ctx.n = ctx.n_rows = ctx.max_kv_len = 1
    ctx.token_feed, ctx._memo, ctx._pending, ctx.stream_cast = None, {}, {}, None
    eng._graph_seen = {(1, 1, 1, None): 1}                  # the second step of its shape: it is captured
    sums = torch.full((4,), 7.0)
    x = torch.zeros(4)
    runs = []

    def forward(c):
        runs.append("capture" if not runs else "plain")
        assert c.take_pending(x) is None and c.stream_cast is None
        if runs[-1] == "capture":
            eng._buf_generation += 1                         # a buffer is replaced ...
            c.once("zeroed", lambda: True)                   # ... and the zeroing is recorded, not done
            c.set_pending(x, object())
            c.stream_cast = x.data_ptr()
        else:
            c.once("zeroed", lambda: (sums.zero_(), True)[1])
        return sums

    eng._forward = forward
    assert eng._forward_graphed(ctx).abs().sum() == 0
    assert runs == ["capture", "plain"] and not eng._graphs


def test_an_answer_of_none_is_kept():
    ctx = object.__new__(StepContext)
    ctx._memo = {}
    asked = []
    for _ in range(3):
        assert ctx.once("plan", lambda: asked.append(1)) is None
    assert len(asked) == 1
