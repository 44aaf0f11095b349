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


@without_device
@pytest.mark.parametrize("n,n_out,k", [(1, 1024, 1024), (2, 4096, 1024), (1, 2048, 4096), (8, 1024, 4096)])
def test_slices_that_a_product_leaves(n, n_out, k):
    """What xr_gemm_tc says of a product whose sum is left to the caller: how many slices lie in the scratch, within the room it was given.  That one
    slice of a product that is not cut may lie there is said to callers of xr_gemm_tc_uncut alone."""
    lib, room = kernels.lib(), 16 * n * n_out
    said = []
    for entry in (lib.xr_gemm_tc, lib.xr_gemm_tc_uncut):
        slices = ctypes.c_int(-7)
        rc = entry(P, P, None, P, kernels.F32, kernels.EPI_ADD, 0, 0.0, 1.0, n, n_out, k, k, n_out, P, room, P, 0, 1, ctypes.byref(slices), 1, None)
        assert rc in NOT_LAUNCHED
        said.append(slices.value)
    if n <= 2:                                    # (on CUDA cores: nothing is cut)
        assert said == [1, kernels.ONE_DEFERRED]
    else:                                         # (no tensor map, no answer)
        assert set(said) <= {-7} | set(range(1, 17))


def test_what_a_products_grid_does_not_hold_goes_by_another():
    """Sizes beyond the grid, or beyond the addresses, of the products in pieces stay with the float32 FMA kernel, which takes them (storage on no device:
    only sizes are looked at)."""
    rows = lambda n, ld, k=256, dtype=torch.float32: torch.empty_strided((n, k), (ld, 1), dtype=dtype, device="meta")
    assert kernels.split_rows_ok(rows(300, 256)) and kernels.split_rows_ok(rows(65535 * 64, 256)) and kernels.split_rows_ok(rows(7, (1 << 31) + 4))
    assert not kernels.split_rows_ok(rows(65535 * 64 + 1, 256)) and not kernels.split_rows_ok(rows(9, 1 << 31)) and not kernels.split_rows_ok(rows(3, 258))
    matrix = lambda r, k: torch.empty(r, k, dtype=torch.bfloat16, device="meta")
    assert kernels.split_shape_ok(matrix(65535 * 128, 256)) and not kernels.split_shape_ok(matrix(65535 * 128 + 1, 256))
    assert not kernels.split_shape_ok(matrix(100, 248)) and not kernels.split_shape_ok(matrix(100, 260))


@without_device
def test_a_recurrence_of_more_blocks_than_the_products_grid_holds():
    """20,000 blocks of 256 channels: four tiles each are more than the grid of the products in pieces holds, and the FMA kernel takes them."""
    R, B = 256 * 20000, 20000
    p = P
    for n in (17, 64):
        args = (p, 2 * R, 0, R, p, p, p, p, p, p, p, p, p, R * 4, p, p, p, p, p, p, p, p, kernels.F32, n, 1, R, B, 4, 8.0, p, 0)
        assert kernels._c.xr_rglru_gates(*args) == -2            # (the products in pieces would ask for a tensor map first)
