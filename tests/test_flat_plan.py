"""Which steps expand the keys of a latent attention layer (LatentAttention._flat_plan): when it pays, what is left to the other order,
how much memory it may take.  No GPU: the plan is arithmetic on a step's portions."""
import time
import types

import numpy as np
import pytest

from xyntetik_runner_b200.parts.latent_attention import LatentAttention


def plan(portions, H=16, D=128, R=64, V=128, C=512, window=0):
    """portions: (position of the first token, tokens) each, in the order of the step."""
    lens = np.array([m for _, m in portions], dtype=np.int32)
    ctx = types.SimpleNamespace(host={"seg_len": lens, "seg_pos0": np.array([p for p, _ in portions], dtype=np.int32),
                                      "seg_start": np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.int32)})
    return LatentAttention._flat_plan(types.SimpleNamespace(H=H, D=D, R=R, V=V, C=C, window=window), ctx, int(lens.sum()))


def test_what_is_expanded_and_what_is_left():
    assert plan([(0, 2048)]) == (2048, 16, [])
    # single tokens and short portions keep the other order, neighbours together
    keys, tiles, rest = plan([(900, 1), (901, 1), (100, 500), (5, 31), (300, 1), (0, 700)])
    assert (keys, tiles, rest) == (600 + 700, 4 + 6, [[0, 2], [502, 534]])
    # only what a window's first token sees, down to a tile's border
    assert plan([(5000, 512)], window=1024)[0] == 5512 - (5000 - 1023) // 128 * 128
    # steps of single tokens, small layers, portions scattered between many others
    assert plan([(3000, 1)] * 8) is None
    assert plan([(0, 64)], H=2, D=64, R=32, V=64, C=64) is None
    assert plan([(0, 512), (9, 1)] * 6) is None


@pytest.mark.parametrize("H", [16, 32, 128])
@pytest.mark.parametrize("at", [0, 7000, 30000, 65000, 200000])
def test_memory_is_bounded(H, at):
    """Whatever the reach, what is gathered and expanded takes at most half a gigabyte: the step could run without."""
    got = plan([(at, 512)] * 3, H=H)
    if got is not None:
        room = 1 << (got[0] - 1).bit_length()                      # (buffers for a power of two of keys)
        assert got[0] == 3 * (at + 512) and room * (H * 256 + 576) * 2 <= 1 << 29
    else:
        assert H * at > 16 * 7000


BIG, SMALL, WINDOW = (dict(H=16, D=128, R=64, V=128, C=512), dict(H=8, D=64, R=32, V=64, C=256), dict(H=16, D=128, R=64, V=128, C=512, window=1024))
# keys held, tokens of the portion, single tokens at 600 keys beside it; microseconds a layer on one B200: over the latent rows, expanded
MEASURED = [
    (BIG, 0, 32, 0, 59, 44),
    (BIG, 0, 512, 16, 216, 114),
    (BIG, 0, 2048, 0, 1365, 137),
    (BIG, 500, 64, 16, 105, 111),
    (BIG, 2000, 32, 0, 92, 95),
    (BIG, 2000, 48, 0, 135, 98),
    (BIG, 2000, 48, 16, 124, 152),
    (BIG, 2000, 96, 16, 249, 162),
    (BIG, 8000, 32, 16, 221, 335),
    (BIG, 8000, 48, 16, 286, 336),
    (BIG, 8000, 200, 16, 1188, 346),
    (BIG, 30000, 32, 16, 644, 902),
    (BIG, 30000, 128, 0, 2754, 512),
    (WINDOW, 0, 256, 0, 138, 84),
    (WINDOW, 2000, 48, 16, 110, 142),
    (WINDOW, 2000, 64, 16, 136, 152),
    (WINDOW, 2000, 200, 16, 249, 154),
    (WINDOW, 8000, 64, 16, 137, 143),
    (SMALL, 0, 1024, 16, 301, 96),
    (SMALL, 2000, 32, 16, 87, 120),
    (SMALL, 8000, 32, 0, 155, 203),
    (SMALL, 8000, 32, 16, 198, 278),
    (SMALL, 8000, 48, 16, 260, 276),
    (SMALL, 8000, 128, 0, 413, 131),
]


@pytest.mark.parametrize("sizes,held,tokens,singles,over_latents,expanded", MEASURED)
def test_the_faster_order_is_taken(sizes, held, tokens, singles, over_latents, expanded):
    """Never expanded where that takes a tenth longer, always where it takes two thirds at most."""
    got = plan([(held, tokens)] + [(600, 1)] * singles, **sizes)
    if expanded > 1.1 * over_latents:
        assert got is None
    if 1.5 * expanded < over_latents:
        assert got is not None


def test_a_plan_takes_little_of_a_steps_host_time():
    """A portion beside 255 single tokens: the plan is made anew for every step with a portion, and nothing hides its time.  (0.1 ms here;
    array operations a portion took 1.0.)"""
    portions = [(505, 505)] + [(700, 1)] * 255
    took = []
    for _ in range(20):
        t0 = time.perf_counter()
        assert plan(portions) is not None
        took.append(time.perf_counter() - t0)
    assert min(took) < 0.5e-3
