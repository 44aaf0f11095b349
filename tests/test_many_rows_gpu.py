"""The kernels and dispatch branches that take steps of many tokens, at the edges of their tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


# ---- float32 attention -----------------------------------------------------------------------------------------------
@pytest.mark.parametrize("H,K,hd,page,extra", [(8, 2, 128, 16, ""), (4, 4, 64, 8, "sink"), (16, 1, 64, 64, "cap"), (6, 3, 256, 32, "bias"), (4, 1, 128, 64, "short")])
def test_float32_attention_of_packed_rows_gives_the_same_bits(H, K, hd, page, extra):
    """Portions that begin inside a chunk of 32 keys and end on either side of one, several in a tile of tokens, against the
    kernel that takes a row alone; the cache holds what is no number behind every portion's last key."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(hd + H)
    specs = [(0, 33), (31, 1), (5, 64), (100, 29)] if extra != "short" else [(0, 40)]
    mp = -(-max(p + n for p, n in specs) // page)
    pages = mp * len(specs)
    cache = torch.full((pages, 1, 2, K, page, hd), float("nan"))
    bt = torch.randperm(pages, generator=g).view(len(specs), mp).int()
    for s, (p0, n) in enumerate(specs):
        for j in range(p0 + n):
            cache[bt[s, j // page], 0, :, :, j % page] = torch.randn(2, K, hd, generator=g)
    n = sum(m for _, m in specs)
    qkv = torch.randn(n, (H + 2 * K) * hd, generator=g).to(DEV)
    positions = _i32([p + i for p, m in specs for i in range(m)])
    tok_seg = _i32([s for s, (_, m) in enumerate(specs) for _ in range(m)])
    cache, bt = cache.to(DEV), bt.to(DEV)
    opt = {"sink": dict(sink=torch.randn(H, generator=g).to(DEV)), "cap": dict(softcap=5.0),
           "bias": dict(bias=torch.randn(H, 20, generator=g).to(DEV))}.get(extra, {})
    outs = []
    for portions in (0, len(specs)):
        out = torch.full((n, H * hd), 7.0, device=DEV)
        kernels.attention_simt(qkv, qkv.shape[1], out, cache.data_ptr(), positions, tok_seg, bt, cache.stride(0), cache.stride(2), H, K, hd, mp, page,
                               0, hd ** -0.5, portions=portions, **opt)
        outs.append(out)
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1])
