"""The library's entry points as a caller of its own reaches them: the arguments they take and what they answer, without a device."""
import ctypes

import pytest
import torch

from xyntetik_runner_b200 import kernels

REFUSED, NOT_LAUNCHED = -1, (-2, -3)             # (-3: no tensor map can be made without a driver)
without_device = pytest.mark.skipif(torch.cuda.is_available(), reason="the addresses are made up: only where nothing can be launched")
P = 1 << 12


@without_device
def test_grouped_products():
    """Seventeen arguments, the status word second to last; sizes of the rows that are anybody's have an entry of their own."""
    head = lambda bn=16, n=64: (P, P, P, kernels.BF16, kernels.EPI_STORE, 0, 0.0, n, 256, 128, 128, 256, bn, P, 4)
    assert kernels._c.xr_gemm_tc_grouped(*head(), P, 0) in NOT_LAUNCHED
    assert kernels._c.xr_gemm_tc_grouped(*head(17), P, 0) == REFUSED and kernels._c.xr_gemm_tc_grouped(*head(16, 63), P, 0) == REFUSED
    live = kernels._c.xr_gemm_tc_grouped_live
    assert live(*head(), 1, 4, P, 0) in NOT_LAUNCHED and live(*head(), 0, 0, P, 0) in NOT_LAUNCHED
    assert live(*head(), 17, 4, P, 0) == REFUSED and live(*head(), -1, 4, P, 0) == REFUSED
