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
