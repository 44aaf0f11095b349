"""Products of one token or two on CUDA cores (csrc/gemv.cuh): the entry points' other road for so few."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _close(got, want, size, k, dtype):
    """A sum of k exact products rounded to float32 at every step, then once to `dtype`."""
    bound = size * (k + 4) * 2.0 ** -24 + (want.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else 0.0) + 1e-6
    assert ((got.double().cpu() - want).abs() <= bound).all()


# rows off a unit's 8 (4 features) and a tile's 128, K off its blocks of 64, one block, fewer than warps, more than are held ahead, more units than
# are walked at once
@pytest.mark.parametrize("n", [1, 2, 3])
@pytest.mark.parametrize("n_out,k", [(1, 8), (7, 72), (130, 64), (129, 1000), (2048, 1024), (500, 4096), (96, 2504), (300, 4104), (28411, 64), (20003, 320)])
def test_products_of_a_few_tokens(n, n_out, k):
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n * 31 + n_out + k)
    x = torch.randn(n, k, generator=g).to(torch.bfloat16)
    wide = torch.full((n, k + 8), float("nan"), dtype=torch.bfloat16, device=DEV)      # (rows apart, what lies between is nobody's)
    wide[:, :k] = x.to(DEV)
    xd = wide[:, :k]
    w = (torch.randn(n_out, k, generator=g) * k ** -0.5).to(torch.bfloat16)
    bias = torch.randn(n_out, generator=g)
    packed = kernels.pack_weight(w.to(DEV))
    torch.cuda.synchronize()                    # (weights are at rest when a product is launched)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    for dtype in (torch.float32, torch.bfloat16):
        out = torch.empty(n, n_out, dtype=dtype, device=DEV)
        kernels.gemm_tc(xd, packed, out, bias.to(DEV), packed_rows=n_out, alpha=-0.5)
        _close(out, -0.5 * want + bias.double(), size + bias.double().abs(), k, dtype)
        kernels.gemm_tc(xd, packed, out, None, packed_rows=n_out, act=kernels.ACT_RELU2)
        _close(out, want.clamp(min=0) ** 2, 2 * size * size + size, k, dtype)
    base = torch.randn(n, n_out + 3, generator=g)
    acc = base.to(DEV)[:, :n_out]
    kernels.gemm_tc(xd, packed, acc, bias.to(DEV), kernels.EPI_ADD, packed_rows=n_out)
    _close(acc, base[:, :n_out].double() + want + bias.double(), size + base[:, :n_out].double().abs() + bias.double().abs(), k, torch.float32)
    # left to the next kernel
    x0 = torch.randn(n, n_out, generator=g)
    rows = x0.to(DEV)
    sums = kernels.gemm_tc_deferred(xd, packed, rows, bias.to(DEV), kernels.EPI_ADD, packed_rows=n_out)
    if sums is not None:                         # (None: the product was not left to anyone)
        assert torch.equal(rows.cpu(), x0)
        kernels.finish_plain(sums.partial, sums.splits, bias.to(DEV), rows, True)
        sums.release()
    _close(rows, x0.double() + want + bias.double(), size + x0.double().abs() + bias.double().abs(), k, torch.float32)
    assert kernels.workspace(torch.device(DEV)).live == 0
    # gated: gate rows, then up rows
    F = (n_out + 1) // 2
    pair = (torch.randn(2 * F, k, generator=g) * k ** -0.5).to(torch.bfloat16)
    gate, up = (x.double() @ pair[i * F:(i + 1) * F].double().T for i in range(2))
    out = torch.empty(n, F, dtype=torch.bfloat16, device=DEV)
    both = kernels.pack_weight(pair.to(DEV), 2)
    torch.cuda.synchronize()
    kernels.gemm_tc(xd, both, out, None, kernels.EPI_GATED, packed_rows=F)
    ref = torch.nn.functional.silu(gate) * up
    assert ((out.double().cpu() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-5 * (gate.abs() + 1) * (up.abs() + 1)).all()


@pytest.mark.parametrize("n,E,top,width,inner", [(1, 16, 2, 1024, 1408), (2, 64, 6, 264, 72), (2, 5, 3, 136, 200), (1, 12, 1, 64, 128)])
def test_experts_products_of_a_few_tokens(n, E, top, width, inner):
    """The rows of the first tiles alone, every one by its tile's matrix, against plain products; other rows stay as they are."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + E)
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(n)])
    used = sorted(set(ids.reshape(-1).tolist()))
    tiles, bn = len(used) + 2, 16
    group = torch.tensor(used + [-1, -1], dtype=torch.int32, device=DEV)
    x = torch.randn(tiles * bn, width, generator=g).to(torch.bfloat16)
    up = (torch.randn(E, inner, width, generator=g) * width ** -0.5).to(torch.bfloat16)
    out = torch.full((tiles * bn, inner), 7.0, device=DEV)
    packed = kernels.pack_weight_groups(up.to(DEV))
    torch.cuda.synchronize()
    kernels.gemm_tc_grouped(x.to(DEV), packed, out, group, bn, inner, kernels.EPI_STORE, kernels.ACT_RELU2, live_rows=n, live_tiles=n * top)
    got = out.cpu().double().view(tiles, bn, inner)
    for t, e in enumerate(used):
        want = (x.view(tiles, bn, width)[t, :n].double() @ up[e].double().T).clamp(min=0) ** 2
        assert ((got[t, :n] - want).abs() <= 1e-4 * (want + 1)).all()
    assert (got[:, n:] == 7).all() and (got[len(used):] == 7).all()


@pytest.mark.parametrize("n,ctx,chunk,page,skew", [(1, 33, 128, 8, 0), (3, 700, 128, 8, 0), (2, 1030, 512, 16, 2), (40, 300, 128, 64, 0), (9, 2000, 128, 64, 0), (1, 2100, 2112, 8, 0)])
def test_latent_attention_by_stages_and_pages(n, ctx, chunk, page, skew):
    """Both depths of the ring (every CTA an SM to itself or not), more pages a split than are kept in shared memory, queries off 16-byte borders, tiles
    that end early; against float64 of the same bfloat16 numbers.  Probabilities are rounded to bfloat16: 2^-8 of the values' size."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + ctx)
    H, C, R = 16, 128, 32
    W, mp = C + R, -(-ctx // page)
    cache = torch.randn(n * mp + 1, page, W, generator=g).to(torch.bfloat16)
    bt = torch.arange(n * mp).reshape(n, mp).flip(1).contiguous()
    pos = torch.tensor([max(0, ctx - 1 - 17 * (i % 5)) for i in range(n)])
    wide = torch.randn(n, H * R + 8, generator=g).to(torch.bfloat16)
    ql = torch.randn(n, H * C, generator=g).to(torch.bfloat16)
    splits = -(-ctx // chunk)
    dev = lambda t, d=torch.int32: t.to(d).to(DEV)
    out = torch.full((n, H * C), float("nan"), device=DEV)
    po, pm = torch.empty(n * splits * 16 * C, device=DEV), torch.empty(n * splits * 32, device=DEV)
    cd = cache.to(DEV)
    kernels.latent_attention_mma(ql.to(DEV), wide.to(DEV), skew, R, out, po, pm, cd.data_ptr(), page * W, dev(pos), dev(torch.arange(n)), dev(bt), H, C, R, mp, page,
                                 0.1, chunk, splits)
    for t in range(n):
        rows = torch.cat([cache[b] for b in bt[t]])[:int(pos[t]) + 1].double()
        q = torch.cat([ql[t].view(H, C), wide[t, skew:skew + H * R].view(H, R)], 1).double()
        want = torch.softmax(0.1 * q @ rows.T, -1) @ rows[:, :C]
        assert (out[t].cpu().double().view(H, C) - want).abs().max() <= 2.0 ** -7 * rows[:, :C].abs().max()


@pytest.mark.parametrize("n,top,E", [(1, 1, 3), (300, 6, 64), (4096, 4, 7), (4097, 4, 16), (6000, 6, 64)])
def test_plan_of_many_pairs(n, top, E):
    """Pairs around and beyond what a thread keeps (16,384 in all), rows of identity experts among them: every pair has a row of its own among its
    expert's, the tiles cover every expert's rows, and the gather brings every row its token, rows of four blocks and a remainder."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + E)
    ids = torch.stack([torch.randperm(E + 2, generator=g)[:top] for _ in range(n)]).int()
    pairs = n * top
    max_tiles, rows = kernels.moe_tiles_room(pairs, E)
    row_src, pair_row, tiles = (torch.full((m,), -7, dtype=torch.int32, device=DEV) for m in (rows, pairs, 1 + 3 * max_tiles))
    kernels.moe_plan_tiles(ids.to(DEV), row_src, pair_row, tiles, E)
    src, at, table = row_src.cpu(), pair_row.cpu().long(), tiles.cpu()
    flat = ids.reshape(-1).long()
    real = flat < E
    assert (at[~real] == -1).all() and at[real].unique().numel() == int(real.sum())
    assert torch.equal(src[at[real]].long(), torch.arange(pairs)[real]) and int((src >= 0).sum()) == int(real.sum())
    owner = torch.full((rows,), -1, dtype=torch.long)
    for e, first, count in table[1:1 + 3 * int(table[0])].view(-1, 3).tolist():
        assert (owner[first:first + count] == -1).all()
        owner[first:first + count] = e
    assert torch.equal(owner[at[real]], flat[real]) and int((owner >= 0).sum()) == int(real.sum())
    h = torch.randn(n, 40, generator=g).to(torch.bfloat16)
    xs = torch.full((rows, 40), 7.0, dtype=torch.bfloat16, device=DEV)
    kernels.moe_gather(h.to(DEV), xs, row_src, None, top)
    want = torch.where((src >= 0)[:, None], h[src.clamp(min=0).long() // top], torch.tensor(7.0, dtype=torch.bfloat16))
    assert torch.equal(xs.cpu(), want)


def test_a_token_meets_an_expert_once():
    """Scores that leave nothing to choose by (one token's are no numbers, or fewer outputs than are chosen have a finite correction): the choices
    of a token still differ, so an expert has as many rows as there are tokens at most, and the other token's rows are all computed."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(4)
    n, E, top, width, inner, align = 2, 12, 3, 64, 136, 16
    z = torch.randn(n, E, generator=g)
    z[0, 5], z[1, 0] = float("nan"), 6.0                        # (expert 0 is the other token's)
    few = torch.full((E,), float("-inf"))
    few[7] = 0.0
    for correction in (None, few):
        cd = None if correction is None else correction.to(DEV)
        ids, w = torch.empty(n, top, dtype=torch.int32, device=DEV), torch.empty(n, top, device=DEV)
        kernels.route_groups(z.to(DEV), ids, w, top, cd, 4, 2, 1.0)
        assert all(len(set(r)) == top and 0 <= min(r) and max(r) < E for r in ids.tolist()), ids
    h = torch.randn(n, width, generator=g).to(torch.bfloat16)
    up = (torch.randn(E, inner, width, generator=g) * width ** -0.5).to(torch.bfloat16)
    tiles = kernels.moe_max_tiles(n * top, E, align)
    pair_row, group = (torch.full((m,), -7, dtype=torch.int32, device=DEV) for m in (n * top, tiles))
    wts, xs = torch.empty(n, top, device=DEV), torch.zeros(tiles * align, width, dtype=torch.bfloat16, device=DEV)
    zs = z.to(DEV)
    kernels.route_few(zs, 1, zs, E, E, top, wts, pair_row, group, align, h.to(DEV), xs, 2, None, 4, 2, 1.0)
    out = torch.full((tiles * align, inner), 7.0, device=DEV)
    packed = kernels.pack_weight_groups(up.to(DEV))
    torch.cuda.synchronize()
    kernels.gemm_tc_grouped(xs, packed, out, group, align, inner, live_rows=n, live_tiles=n * top)
    rows, of = pair_row.cpu().view(n, top)[1].tolist(), group.cpu()
    assert int(of[rows[0] // align]) == 0
    for r in rows:
        want = h[1].double() @ up[int(of[r // align])].double().T
        assert (out[r].cpu().double() - want).abs().max() <= 1e-4


@pytest.mark.parametrize("n,n_out,k,few", [(1, 1024, 4096, True), (1, 1024, 4104, False), (1, 2504, 64, True), (2, 2048, 1536, True), (2, 2048, 1544, False),
                                           (2, 16, 8, True), (3, 1024, 1024, False)])
def test_which_road_a_product_takes(n, n_out, k, few):
    """The road of one token or two says so and is counted apart, stored, added, left to the next kernel and gated; K 8 further on and one token more
    are counted as products on tcgen05."""
    from types import SimpleNamespace
    from xyntetik_runner_b200 import kernels
    from xyntetik_runner_b200.parts import linear
    rt = SimpleNamespace(act_dtype=torch.bfloat16)
    w = torch.randn(n_out, k, device=DEV).to(torch.bfloat16)
    one, both = linear.Linear(w).prepare(rt), linear.Linear(w, halves=2).prepare(rt)
    x, stored, added = torch.randn(n, k, device=DEV).to(torch.bfloat16), torch.empty(n, n_out, device=DEV), torch.zeros(n, n_out, device=DEV)
    pair = torch.empty(n, n_out // 2, device=DEV, dtype=torch.bfloat16)
    torch.cuda.synchronize()
    before, kept = dict(linear.counters), kernels.few_products
    one.forward(x, stored)
    one.forward(x, added, accumulate=True)
    both.forward_gated(x, pair)
    pending = one.forward(x, added, accumulate=True, defer=True)
    if few:
        assert pending is not None and pending.splits == 1
    if pending is not None:
        pending.finish()
    gone = {name: linear.counters[name] - before[name] for name in before}
    assert (gone["few"], gone["tcgen05"]) == ((4, 0) if few else (0, 4)) and kernels.few_products - kept == gone["few"]
    assert (added - 2 * stored).abs().max() <= 1e-4 * stored.abs().max()
    assert kernels.gemm_tc(x, one.packed, stored, packed_rows=n_out) == 1 or not few


def test_an_engines_single_tokens_take_it(tmp_path):
    import tiny
    from xyntetik_runner_b200.engine.runner import Runner
    from xyntetik_runner_b200.parts import linear
    tiny.make_folder(str(tmp_path), "B", "bfloat16")
    before = dict(linear.counters)
    Runner(str(tmp_path), dtype="bfloat16", ctx=64, parallel=2, page_size=8).generate(list(range(3, 12)), n=4, temp=0.0, ignore_eos=True)
    assert linear.counters["few"] > before["few"] + 4 and linear.counters["tcgen05"] > before["tcgen05"] + 4


@pytest.mark.parametrize("n,E,top,width,inner,act,limit", [(1, 16, 2, 1024, 1408, 1, 0.0), (2, 64, 6, 264, 72, 3, 7.0), (2, 12, 2, 1024, 1400, 2, 0.0)])
def test_gated_experts_of_a_few_tokens(n, E, top, width, inner, act, limit):
    """Gated experts' first product in bfloat16 as their layer asks for it: the rows that live against plain products, all others untouched."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n * 3 + E)
    used = sorted(set(torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(n)]).reshape(-1).tolist()))
    tiles, bn = len(used) + 2, 16
    group = torch.tensor(used + [-1, -1], dtype=torch.int32, device=DEV)
    x = torch.randn(tiles * bn, width, generator=g).to(torch.bfloat16)
    w = (torch.randn(E, 2 * inner, width, generator=g) * width ** -0.5).to(torch.bfloat16)
    out = torch.full((tiles * bn, inner), 7.0, device=DEV, dtype=torch.bfloat16)
    packed = kernels.pack_weight_groups(w.to(DEV), 2)
    torch.cuda.synchronize()
    kernels.gemm_tc_grouped(x.to(DEV), packed, out, group, bn, inner, kernels.EPI_GATED, act, limit, live_rows=n, live_tiles=n * top)
    got = out.cpu().double().view(tiles, bn, inner)
    for t, e in enumerate(used):
        gate, up = (x.view(tiles, bn, width)[t, :n].double() @ w[e, i * inner:(i + 1) * inner].double().T for i in range(2))
        if act == 3:
            gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
            want = gate * torch.sigmoid(1.702 * gate) * (up + 1)
        else:
            want = (torch.nn.functional.silu(gate) if act == 1 else torch.nn.functional.gelu(gate, approximate="tanh")) * up
        # one rounding to bfloat16; float32 sums and the hardware's approximate functions 2e-5 of both factors' size
        assert ((got[t, :n] - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * (gate.abs() + 1) * (up.abs() + 2)).all()
    assert (got[:, n:] == 7).all() and (got[len(used):] == 7).all()
