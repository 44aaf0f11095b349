"""Row kernels with several columns a thread beside what they stand for: borders that allow it and borders that do not, widths with remainders."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,width", [(1, 8), (3, 12), (5, 2048), (2, 1030), (70001, 8)])
def test_concat_cast(dtype, n, width):
    from xyntetik_runner_b200 import kernels
    a, b = (torch.randn(n, width, device=DEV) for _ in range(2))
    out = torch.empty(n, 2 * width, dtype=dtype, device=DEV)
    kernels.concat_cast(a, b, out)
    assert torch.equal(out, torch.cat([a, b], 1).to(dtype))


@pytest.mark.parametrize("n,H,V,skip", [(1, 1, 4, 0), (3, 4, 64, 0), (3, 4, 64, 1), (5, 2, 132, 4), (7, 3, 256, 0), (2, 2, 260, 0), (2, 1, 512, 0), (2, 2, 516, 0), (9, 8, 102, 2)])
@pytest.mark.parametrize("dtype,gate_dtype,silu", [(torch.float32, torch.float32, True), (torch.bfloat16, torch.bfloat16, False), (torch.bfloat16, torch.float32, True)])
def test_head_norm_gate(n, H, V, skip, dtype, gate_dtype, silu):
    """Heads of one, two and four accesses a lane and of more values than that, gates off the borders."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + H * V)
    o, w = torch.randn(n, H * V, generator=g), 1 + 0.1 * torch.randn(H * V, generator=g)
    gate = torch.randn(n, H * V + 8, generator=g).to(gate_dtype)
    y = torch.empty(n, H * V, dtype=dtype, device=DEV)
    kernels.head_norm_gate(o.to(DEV), gate.to(DEV), skip, w.to(DEV), y, H, V, 1e-5, True, silu)
    od, z = o.double().view(n, H, V), gate[:, skip:skip + H * V].double()
    want = (od / torch.sqrt((od * od).mean(-1, keepdim=True) + 1e-5)).view(n, -1) * w.double() * torch.sigmoid(z) * (z if silu else 1.0)
    # float32 sums of V squares and a few functions: 1e-5 of the value; stored once
    assert ((y.double().cpu() - want).abs() <= want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 1e-5) + 1e-6).all()


@pytest.mark.parametrize("n,width,groups,skip", [(1, 4, 1, 0), (3, 512, 1, 0), (3, 516, 1, 0), (2, 2048, 1, 4), (777, 2048, 1, 0), (4, 2048, 4, 0), (2, 2048, 1, 1), (2, 8192, 1, 0), (2, 8196, 1, 0), (3, 30, 3, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_silu_gate_norm(n, width, groups, skip, dtype):
    """Groups of one and of four accesses a thread, wider ones, gates off the borders."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + width)
    o, gate, w = torch.randn(n, width, generator=g), torch.randn(n, width + 8, generator=g), 1 + 0.1 * torch.randn(width, generator=g)
    y = torch.empty(n, width, dtype=dtype, device=DEV)
    kernels.silu_gate_norm(o.to(DEV), gate.to(DEV), skip, w.to(DEV), y, groups, 1e-5)
    z = (o.double() * torch.nn.functional.silu(gate[:, skip:skip + width].double())).view(n, groups, -1)
    want = (z / torch.sqrt((z * z).mean(-1, keepdim=True) + 1e-5)).view(n, -1) * w.double()
    assert ((y.double().cpu() - want).abs() <= want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 1e-5) + 1e-6).all()
