"""When a recurrence over a matrix memory runs in chunks (csrc/chunked.cuh) instead of token by token."""
from __future__ import annotations

import torch

from .. import kernels

# Portions of at least so many tokens.  The walk takes about 0.1 us a token whatever stands beside it (mLSTM's 0.4); the chunks take
# five to eight launches of a few microseconds each.  8 heads, us, walk / chunks: constant decay 512 tokens 45 / 44, 777 66 / 58; decay
# per key channel 512 tokens 68 / 81, 777 96 / 88; mLSTM 128 tokens 64 / 73, 192 92 / 73.  (The state-space recurrence of Mamba-2,
# whose heads have 64 values and fill the machine, is as fast walked at every size up to 2,048.)
CHUNKED_FROM = {"head": 640, "key": 768, "mlstm": 192}


def chunk_scratch(ctx, kind: str, H: int, D: int, V: int):
    """The scratch that sends this step's recurrence through the chunked kernels, or None for the walk: steps without a long portion,
    sizes the chunked kernels do not take, and the true 32-bit path, which promises the same bits however portions are cut."""
    if ctx.act_dtype != torch.bfloat16:
        return None
    if ctx.once("longest_portion", lambda: int(ctx.host["seg_len"].max())) < CHUNKED_FROM[kind]:
        return None
    n = ctx.n
    floats = ctx.once(("chunked_floats", kind, H, D, V), lambda: kernels.chunked_floats(n, ctx.n_seg, H, D, V, kind))
    if floats == 0:
        return None
    # (a power of two: a buffer that grows invalidates the step graphs)
    return ctx.buf("chunk_scratch", (1 << (floats - 1).bit_length(),), torch.float32)
