"""The launchers through the generated extension (csrc/calls.py) and through ctypes: the same answers, and which of the two it is."""
import ctypes

import pytest
import torch

from xyntetik_runner_b200 import kernels
from xyntetik_runner_b200.csrc import build, calls


@pytest.fixture
def elsewhere(monkeypatch, tmp_path):
    """Nothing is built yet, as on a fresh clone (the CUDA library itself is taken from where it is)."""
    kernels.lib()
    monkeypatch.setattr(build, "library_path", lambda build=True, p=build.library_path(build=False): p)
    monkeypatch.setattr(build, "_build_dirs", lambda: [str(tmp_path)])
    monkeypatch.setattr(kernels, "_c", kernels._Calls())


SIZES = [(700, 3, 8, 128, 256, 2), (700, 3, 8, 96, 256, 2), (65, 1, 2, 64, 64, 1)]


def test_without_a_compiler_ctypes_gives_the_same_answers(elsewhere, monkeypatch):
    want = build.calls(build.library_path())            # (built here, in the empty folder)
    monkeypatch.setattr(build, "_build_dirs", lambda: ["/nowhere"])
    monkeypatch.setattr(build.shutil, "which", lambda name: None)
    assert kernels._c.xr_moe_tile_rows() == want.xr_moe_tile_rows()
    assert isinstance(kernels._c, kernels._CtypesCalls)
    assert [kernels._c.xr_chunked_floats(*s) for s in SIZES] == [want.xr_chunked_floats(*s) for s in SIZES]
    assert kernels._c.xr_chunked_floats(1 << 20, 1, 64, 128, 256, 2) > 1 << 31


def test_a_compiler_that_rejects_the_source_is_an_error(elsewhere, monkeypatch):
    monkeypatch.setattr(calls, "source", lambda: "this is not C++\n")
    with pytest.raises(build.BuildError, match="C\\+\\+ compiler failed"):
        kernels._c.xr_moe_tile_rows()


def test_an_int_set_through_a_pointer_is_returned():
    fn = lambda a, out, b: (ctypes.cast(out, ctypes.POINTER(ctypes.c_int)).__setitem__(0, 5), a + b)[1]
    assert kernels._CtypesCalls._setting(fn, 1)(2, -2) == 5 and kernels._CtypesCalls._setting(fn, 1)(-1, 0) == -1


@pytest.mark.gpu
def test_a_cut_product_through_either(monkeypatch):
    g = torch.Generator().manual_seed(3)
    x, w = (torch.randn(s, generator=g).bfloat16().cuda() for s in ((5, 2048), (256, 2048)))
    got = []
    kernels.lib()
    for way in (build.calls(build.library_path(build=False)), kernels._CtypesCalls(kernels.lib())):
        monkeypatch.setattr(kernels, "_c", way)
        out = torch.empty(5, 256, device="cuda")
        got.append((kernels.gemm_tc(x, w, out), out))
        with pytest.raises(kernels.KernelError):
            kernels.gemm_tc(x, w, out, epilogue=7)
    assert got[0][0] == got[1][0] > 1 and torch.equal(got[0][1], got[1][1])
    a, b = x.double().cpu(), w.double().cpu().T
    assert ((got[0][1].double().cpu() - a @ b).abs() <= 2048 * 2.0 ** -24 * (a.abs() @ b.abs())).all()
