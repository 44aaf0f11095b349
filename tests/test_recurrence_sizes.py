"""Sizes that the gated linear recurrence (xr_rglru) takes and refuses, by its answer alone: without a device nothing is launched, and an
accepted call answers that the launch was refused."""
import pytest
import torch

from xyntetik_runner_b200 import kernels

REFUSED, NO_DEVICE = -1, -2


def answer(n, R, B, taps=4):
    p = 1 << 12
    return kernels._c.xr_rglru(p, 2 * R, 0, R, p, p, p, p, p, p, p, p, R * taps, p, p, p, p, p, p, p, p, kernels.BF16, n, 1, R, B, taps, 8.0, 0)


@pytest.mark.skipif(torch.cuda.is_available(), reason="the addresses are made up: only where nothing can be launched")
def test_sizes():
    assert answer(1901, 2560, 10) == NO_DEVICE and answer(1, 48, 2) == NO_DEVICE
    assert answer(900_000, 2560, 10) == NO_DEVICE               # more than 2^31 elements
    assert answer(17, 6400, 1) == answer(1, 6400, 1) == NO_DEVICE and answer(17, 6408, 1) == answer(1, 6408, 1) == REFUSED
    assert answer(17, 48, 5) == REFUSED and answer(0, 48, 2) == REFUSED and answer(17, 48, 2, taps=17) == REFUSED


@pytest.mark.skipif(torch.cuda.is_available(), reason="the addresses are made up: only where nothing can be launched")
@pytest.mark.parametrize("kind", ["head", "key"])
def test_scratch_of_chunks(kind):
    """The chunked kernels read and write their scratch 16 bytes at a time: one off that border, or too small, is refused ahead of any launch."""
    n, H, D, V, p = 700, 2, 64, 64, 1 << 12
    floats = kernels.chunked_floats(n, 1, H, D, V, kind)

    def ask(scratch, room):
        ld, st = 2 * H * D + H * V + 8, H * D * V
        if kind == "head":
            return kernels._c.xr_decay_attention(p, ld, 0, H * D, 2 * H * D, p, p, st, p, p, p, p, n, 1, H, D, V, 1, 1.0, scratch, room, 0)
        return kernels._c.xr_key_decay_attention(p, ld, 0, H * D, 2 * H * D, 2 * H * D + H * V, p, p, 8, 1.0, p, p, st, p, p, p, p, n, 1, H, D, V, 1.0,
                                                 scratch, room, 0)
    assert ask(1 << 16, floats) == NO_DEVICE and ask(None, 0) == NO_DEVICE
    assert ask((1 << 16) + 4, floats) == REFUSED and ask((1 << 16) + 8, floats) == REFUSED and ask(1 << 16, floats // 2) == REFUSED
