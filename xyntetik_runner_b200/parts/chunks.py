"""When a recurrence over a matrix memory runs in chunks (csrc/chunked.cuh) instead of token by token."""
from __future__ import annotations

import math

import torch

from .. import kernels

# The longest portion must have at least so many tokens: below, the chunks' five to eight launches cost as much as the walk.
CHUNKED_FROM = {"head": 640, "key": 768, "mlstm": 192}

# What the scratch of one step may take: it stays allocated beside the cached keys, and the walk needs none.
MOST_BYTES = 1 << 28

# Both sides' times in microseconds (``costs``).  walk: a launch, a token of the longest portion, the same where a warp takes twice the
# columns (wide), a token of a block's work on one multiprocessor, and the share of these with keys of 64.  chunks: launches, a
# million elements of a chunk's memory, a million of its scores, a thousand blocks' look through a portion.
_WALK = {"head": (5.6, 0.062, 0.134, 0.091, 0.75, 0.675), "key": (13.4, 0.078, 0.162, 0.128, 0.70, 0.59), "mlstm": (11.2, 0.479, 0.479, 0.236, 0.89, 0.65)}
_CHUNKS = {"head": (32.0, 13.4, 0.5, 1.5), "key": (44.6, 15.0, 5.1, 1.1), "mlstm": (46.0, 15.9, 13.0, 0.8)}
_SMS, _MARGIN = 148, 1.1


def costs(kind: str, lens, H: int, D: int, V: int):
    """(walk, chunks): what a step with portions of `lens` tokens takes either way.  The walk goes through all portions side by side: the
    longest one's chain, or the work of all blocks over the machine, whichever is larger.  The chunks' time grows with all tokens and
    heads, and every portion, a single token too, is a chunk with a memory of its own, whose blocks look for their portion among all.
    Fitted to 1,080 steps on one B200 (1 to 129 portions of 1 to 2,048 tokens, 4 to 32 heads of 64 x 64 to 128 x 256), walk / chunks, 8 heads,
    us: constant decay, 128 x 128: 2,048 tokens 167 / 74, 3 x 680 88 / 77, 10 x 700 226 / 245, 800 beside 8 single tokens 103 / 86, beside
    128 110 / 1,002; decay per key channel, 128 x 256: 1,500 168 / 116, 3 x 680 175 / 157, 10 x 700 440 / 641, 800 + 8 130 / 161; mLSTM,
    128 x 256: 192 106 / 69, 3 x 200 160 / 92, 10 x 200 226 / 238, 200 + 32 117 / 278.  (The state-space recurrence of Mamba-2, whose heads
    have 64 values and fill the machine, is as fast walked at every size up to 2,048.)"""
    longest, n, S = max(lens), sum(lens), len(lens)
    c0, chain, chain_wide, work, d64_chain, d64_work = _WALK[kind]
    wide = kind != "mlstm" and -(-V // 16) * H * S > 2 * _SMS
    blocks = H * -(-V // (16 if kind != "mlstm" and not wide else 32))
    walk = c0 + math.hypot((chain_wide if wide else chain) * (d64_chain if D <= 64 else 1.0) * longest,
                           work * (d64_work if D <= 64 else 1.0) * n * blocks / _SMS)
    launches, memory, scores, look = _CHUNKS[kind]
    chunks = sum(-(-m // 64) for m in lens) * H
    return walk, launches + chunks * D * (memory * V + scores * 64) * 1e-6 + look * S * chunks * V / 64 * 1e-3


def chunk_scratch(ctx, kind: str, H: int, D: int, V: int):
    """The scratch that sends this step's recurrence through the chunked kernels, or None for the walk: where the chunks do not pay (by
    less than what ``costs`` is off by), scratch beyond MOST_BYTES, sizes the chunked kernels do not take, and the true 32-bit path, which
    promises the same bits however portions are cut."""
    if ctx.act_dtype != torch.bfloat16:
        return None
    floats = ctx.once(("chunked_floats", kind, H, D, V), lambda: _floats(ctx, kind, H, D, V))
    if floats == 0:
        return None
    # (a power of two: a buffer that grows invalidates the step graphs)
    return ctx.buf("chunk_scratch", (1 << (floats - 1).bit_length(),), torch.float32)


def _floats(ctx, kind: str, H: int, D: int, V: int) -> int:
    lens = ctx.host["seg_len"]
    if int(lens.max()) < CHUNKED_FROM[kind]:
        return 0
    floats = kernels.chunked_floats(ctx.n, ctx.n_seg, H, D, V, kind)
    if floats == 0 or 4 << (floats - 1).bit_length() > MOST_BYTES:
        return 0
    walk, chunks = costs(kind, lens.tolist(), H, D, V)
    return floats if _MARGIN * chunks < walk else 0
