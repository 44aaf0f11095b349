"""Products of float32 rows with a bfloat16 matrix in three exact pieces on the tensor cores (csrc/split_product.cuh)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# rows of W off and on the tiles' 128 (64 gated), tokens around every tile's 16, 32 and 64, K off its blocks of 64, of one slice and of eight
SIZES = [(1, 8, 256), (15, 129, 264), (17, 128, 1024), (33, 127, 328), (64, 1000, 512), (65, 64, 4096), (129, 6000, 256), (300, 257, 2816), (300, 5001, 1024)]


def _inputs(n, rows, k, seed=0):
    g = torch.Generator().manual_seed(n * 7 + rows + k + seed)
    x = torch.randn(n, k, generator=g) * torch.exp(2.0 * torch.randn(n, 1, generator=g))
    return x, (torch.randn(rows, k, generator=g) * k ** -0.5).to(torch.bfloat16)


@pytest.mark.parametrize("n,n_out,k", SIZES)
def test_products_in_pieces(n, n_out, k):
    """Stored behind a factor, a bias and an activation, added, gated, with strided rows; against float64.  A sum of k products rounded to
    float32 at every step is off by at most (k + 2) 2^-24 times the sum of their sizes; as a whole it is no further off than the FMA
    kernel's.  A token alone gives the same bits."""
    from xyntetik_runner_b200 import kernels
    x, w = _inputs(n, n_out, k)
    xs = torch.full((n, k + 4), float("nan"), device=DEV)
    xs[:, :k] = x.to(DEV)
    xd, wd = xs[:, :k], w.to(DEV)
    assert kernels.split_weight_ok(wd) and kernels.split_rows_ok(xd)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    bound = size * (k + 2) * 2.0 ** -24
    got, fma = (torch.empty(n, n_out, device=DEV) for _ in range(2))
    kernels.gemm_split(xd, wd, got)
    assert ((got.cpu().double() - want).abs() <= bound).all()
    kernels.gemm_simt(xd, wd, fma)
    off = lambda y: float(((y.cpu().double() - want) / size).square().mean().sqrt())
    assert off(got) <= off(fma) * (1.0 if n * n_out > 2000 else 1.5), (off(got), off(fma))
    for t in {0, n // 2, n - 1}:
        one = torch.empty(1, n_out, device=DEV)
        kernels.gemm_split(xd[t:t + 1], wd, one)
        assert torch.equal(one[0], got[t]), t
    bias, base = torch.randn(n_out, device=DEV), torch.randn(n, n_out + 3, device=DEV)
    out = base.clone()[:, :n_out]
    kernels.gemm_split(xd, wd, out, bias, True, -0.3)
    assert torch.equal(out, base[:, :n_out] + (-0.3 * got + bias)) or (out - (base[:, :n_out] + (-0.3 * got + bias))).abs().max() <= 2e-6 * (got.abs().max() + 5)
    kernels.gemm_split(xd, wd, out, bias, False, 0.5, kernels.ACT_SILU)
    assert torch.allclose(out, torch.nn.functional.silu(0.5 * got + bias), rtol=2e-6, atol=2e-6)
    F = n_out // 2
    pair = torch.empty(n, F, device=DEV)
    for act, limit in ((kernels.ACT_SILU, 0.0), (kernels.ACT_SWISH_CLAMP, 1.5)):
        ref = torch.empty(n, F, device=DEV)
        kernels.gemm_split(xd, wd[:2 * F], pair, act=act, gated=True, limit=limit)
        kernels.act_mul(got[:, :2 * F].contiguous(), ref, act, True, limit)
        assert torch.allclose(pair, ref, rtol=1e-6, atol=1e-7)


def test_values_that_are_no_numbers_and_the_smallest():
    """An infinite value makes its sums infinite, one that is no number makes them none, other rows stay; values near both ends of the range."""
    from xyntetik_runner_b200 import kernels
    x, w = _inputs(40, 200, 320)
    x[3, 7], x[4, 8], x[5, 9], x[6] = float("inf"), float("-inf"), float("nan"), 3.0e38 * (torch.arange(320) == 11)
    x[7] *= 1e-33
    x[8, 1] = torch.tensor(0x7f800001, dtype=torch.int32).view(torch.float32)          # no number by its last bit alone
    out, fma = (torch.empty(40, 200, device=DEV) for _ in range(2))
    kernels.gemm_split(x.to(DEV), w.to(DEV), out)
    kernels.gemm_simt(x.to(DEV), w.to(DEV), fma)
    assert torch.equal(out.isnan(), fma.isnan()) and torch.equal(out.isinf(), fma.isinf())
    # both are within (k + 2) 2^-24 of the products' sizes; pieces below 2^-126 may count as zero
    x = torch.where(x.isfinite(), x, 0.0).double()
    bound = x.abs() @ w.double().abs().T * (2 * 322 * 2.0 ** -24) + 320 * 2.0 ** -126
    live = fma.isfinite().cpu()
    assert ((out.cpu().double() - fma.cpu().double()).abs() <= bound)[live].all()
    w[0, 0] = float("inf")
    assert not kernels.split_weight_ok(w.to(DEV))


@pytest.mark.parametrize("n,R,B", [(63, 512, 2), (64, 768, 3), (65, 2560, 10), (200, 1320, 5), (777, 576, 2)])
def test_recurrences_gates_in_pieces(n, R, B):
    """The gates' products on the tensor cores beside the FMA kernel's: the recurrence's outputs and state from both, against float64."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + R)
    Bs, taps = R // B, 4
    dev = lambda t: t.to(DEV)
    proj = dev(torch.randn(n, 2 * R, generator=g))
    conv_w, conv_b = dev(torch.randn(R, taps, generator=g) * 0.5), dev(torch.randn(R, generator=g) * 0.1)
    both = dev((torch.randn(2 * R, Bs, generator=g) * Bs ** -0.5).to(torch.bfloat16))
    wa, wi = (both[i * R:(i + 1) * R].float().reshape(B, Bs, Bs).contiguous() for i in range(2))
    ba, bi, lam = (dev(torch.randn(R, generator=g) * 0.5 - s) for s in (0.0, 0.0, 4.0))
    ints = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)
    seg = torch.zeros(n, dtype=torch.int32, device=DEV)
    got = []
    for gates in (None, both):
        state = torch.zeros(1, kernels.rglru_state_floats(R, taps), device=DEV)
        a, b, u, p = torch.empty(n, R, device=DEV), torch.empty(n, R, device=DEV), torch.empty(n, R, device=DEV), proj.clone()
        out = torch.empty(n, R, device=DEV)
        kernels.rglru(p, conv_w, conv_b, None, None, wa, wi, ba, bi, lam, state, seg, ints(0), ints(n), ints(0), a, b, u, out, 1, R, B, taps, 8.0, gates)
        ud = u.double().view(n, B, Bs)
        r, i = (torch.sigmoid(torch.einsum("tbi,boi->tbo", ud, w.double()).reshape(n, R) + c.double()) for w, c in ((wa, ba), (wi, bi)))
        la = -8.0 * r * torch.nn.functional.softplus(lam.double())
        want = torch.exp(la), torch.sqrt(-torch.expm1(2.0 * la)) * i * u.double()
        got.append([float((x.double() - y).square().mean().sqrt()) for x, y in zip((a, b), want)] + [out, state, p])
    for off, fma in zip(got[1][:2], got[0][:2]):
        assert off <= 1.02 * fma + 1e-9
    for x, y in zip(got[1][2:], got[0][2:]):
        assert (x - y).abs().max() <= 2e-5 * y.abs().max()


@pytest.mark.parametrize("R,B", [(512, 2), (1320, 5)])
def test_a_recurrence_in_32_bits_cut_anywhere(R, B):
    """The true 32-bit path with bfloat16 gate matrices, portions of more than sixteen tokens: outputs and state are the same bits whatever
    portions a text is cut into (around every width of the products' token tiles, and the 64 tokens that serving steps go by) and whatever stands
    beside one."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(R)
    n, Bs, taps = 200, R // B, 4
    dev = lambda t: t.to(DEV)
    proj = dev(torch.randn(n, 2 * R, generator=g))
    conv_w, conv_b = dev(torch.randn(R, taps, generator=g) * 0.5), dev(torch.randn(R, generator=g) * 0.1)
    gates = dev((torch.randn(2 * R, Bs, generator=g) * Bs ** -0.5).to(torch.bfloat16))
    assert kernels.split_weight_ok(gates)
    wa, wi = (gates[i * R:(i + 1) * R].float().reshape(B, Bs, Bs).contiguous() for i in range(2))
    ba, bi, lam = (dev(torch.randn(R, generator=g) * 0.5 - s) for s in (0.0, 0.0, 4.0))
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)

    def step(rows, lengths, state):
        m = rows.shape[0]
        a, b, u, out = (torch.empty(m, R, device=DEV) for _ in range(4))
        seg = ints([i for i, k in enumerate(lengths) for _ in range(k)])
        starts = [sum(lengths[:i]) for i in range(len(lengths))]
        kernels.rglru(rows.clone(), conv_w, conv_b, None, None, wa, wi, ba, bi, lam, state, seg, ints(starts), ints(lengths), ints(list(range(len(lengths)))), a, b, u, out,
                      len(lengths), R, B, taps, 8.0, gates)
        return out

    def text(cuts):
        state = torch.zeros(1, kernels.rglru_state_floats(R, taps), device=DEV)
        outs, at = [], 0
        for k in cuts:
            outs.append(step(proj[at:at + k], [k], state))
            at += k
        return torch.cat(outs), state
    whole, state = text([200])
    for cuts in ([100, 100], [17, 63, 64, 56], [40, 33, 65, 62], [136, 32, 32]):
        got, st = text(cuts)
        assert torch.equal(got, whole) and torch.equal(st, state), cuts
    two = torch.zeros(2, kernels.rglru_state_floats(R, taps), device=DEV)
    beside = step(torch.cat([proj[:40], proj]), [40, 200], two)
    assert torch.equal(beside[:40], whole[:40]) and torch.equal(beside[40:], whole) and torch.equal(two[1:], state)


@pytest.mark.parametrize("n,n_out,k", [(1, 129, 1024), (3, 33, 2048), (20, 161, 4096), (40, 255, 2816), (70, 97, 512), (300, 1, 1024)])
def test_rows_that_part_a_warp(n, n_out, k):
    """Outputs that end inside a warp's 32, K in slices and whole, activations with branches that lanes take apart: what every warp does as one behind
    them (the cluster's barrier, tensor memory's release) still comes to its end, twice over, with the same bits."""
    from xyntetik_runner_b200 import kernels
    x, w = _inputs(n, n_out, k)
    x *= 60.0                                          # (SiLU below and above -80)
    xd, wd = x.to(DEV), w.to(DEV)
    want = x.double() @ w.double().T
    bound = x.double().abs() @ w.double().abs().T * (k + 2) * 2.0 ** -24
    for act, ref in ((kernels.ACT_SILU, torch.nn.functional.silu(want)), (kernels.ACT_RELU2, want.clamp(min=0) ** 2)):
        out, again = (torch.empty(n, n_out, device=DEV) for _ in range(2))
        kernels.gemm_split(xd, wd, out, act=act)
        kernels.gemm_split(xd, wd, again, act=act)
        # an error e of the sum: 1.1 e of SiLU (its largest slope), 2 |sum| e + e^2 of the square; functions and the last rounding 2^-20 of the value
        slope = 1.1 * bound if act == kernels.ACT_SILU else 2 * want.abs() * bound + bound * bound
        assert ((out.cpu().double() - ref).abs() <= slope + ref.abs() * 2.0 ** -20 + 1e-30).all()
        assert torch.equal(out, again)
    assert int(kernels.workspace(torch.device(DEV)).status.sum()) == 0


def test_the_switch_reaches_a_recurrences_gates(monkeypatch):
    """With the tensor cores switched off to bisect a difference, the gates go to the FMA kernel too."""
    from types import SimpleNamespace
    from xyntetik_runner_b200.parts import linear_tc
    from xyntetik_runner_b200.parts.rglru import GatedLinearRecurrence
    for on in (True, False):
        monkeypatch.setattr(linear_tc, "ENABLED", on)
        part = GatedLinearRecurrence(64, 512, 2, 4, "")
        part.bind({name: torch.randn(spec.shape, device=DEV).to(torch.bfloat16) for name, spec in part.tensors().items()}, SimpleNamespace(act_dtype=torch.bfloat16))
        assert (part.gates is not None) == on and (part.out.packed is not None) == on
