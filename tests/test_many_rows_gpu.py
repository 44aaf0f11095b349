"""The kernels and dispatch branches that take steps of many tokens, at the edges of their tiles."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


# ---- float32 products ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("n,n_out,k,wdt", [(1, 33, 7, torch.float32), (8, 100, 260, torch.bfloat16), (9, 65, 64, torch.bfloat16), (40, 3001, 36, torch.float32),
                                           (300, 2001, 40, torch.bfloat16), (301, 8001, 33, torch.float32), (700, 13001, 36, torch.float32)])
def test_float32_product_in_every_tile(n, n_out, k, wdt):
    """Few tokens, few tiles, many of every size; K off and on the copies' border.  A float32 sum of k products
    is off by at most k 2^-24 times the sum of their sizes; and a row is the same whatever stands beside it."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + k)
    x, w = torch.randn(n, k, generator=g), torch.randn(n_out, k, generator=g).to(wdt)
    out = torch.empty(n, n_out, device=DEV)
    kernels.gemm_simt(x.to(DEV), w.to(DEV), out)
    bound = (x.double().abs() @ w.double().abs().T) * (k + 2) * 2.0 ** -24
    assert ((out.cpu().double() - x.double() @ w.double().T).abs() <= bound).all()
    for t in {0, n // 2, n - 1}:
        one = torch.empty(1, n_out, device=DEV)
        kernels.gemm_simt(x[t:t + 1].to(DEV), w.to(DEV), one)
        assert torch.equal(one[0], out[t])


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


# ---- dense products on CTA pairs ----------------------------------------------------------------------------------------
@pytest.mark.parametrize("n,n_out,k", [(300, 1024, 1024), (401, 3071, 2048), (300, 5632, 1024), (400, 5632, 1024), (512, 5632, 1024), (640, 5632, 1024),
                                       (1025, 4098, 520), (129, 70, 72)])
def test_dense_products_in_every_width(n, n_out, k):
    """Products whose sizes choose tiles of 64, 96, .. 256 tokens, cut and uncut, rows that pair up for a store and rows that do not: a
    sum of k products in float32, and a bfloat16 store's rounding."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + n_out)
    x, w = torch.randn(n, k, generator=g).bfloat16(), (torch.randn(n_out, k, generator=g) * k ** -0.5).bfloat16()
    bias, old = torch.randn(n_out, generator=g), torch.randn(n, n_out, generator=g)
    want = x.double() @ w.double().T + bias.double()
    bound = ((x.double().abs() @ w.double().abs().T) + bias.double().abs()) * (k + 4) * 2.0 ** -24
    xd, wd = x.to(DEV), kernels.pack_weight(w.to(DEV))
    out, wide = torch.full((n + 1, n_out), 7.0, dtype=torch.bfloat16, device=DEV), old.to(DEV)
    kernels.gemm_tc(xd, wd, out[:n], bias.to(DEV), kernels.EPI_STORE, packed_rows=n_out)
    kernels.gemm_tc(xd, wd, wide, bias.to(DEV), kernels.EPI_ADD, packed_rows=n_out)
    assert ((out[:n].cpu().double() - want).abs() <= bound + 2.0 ** -8 * want.abs()).all() and (out[n] == 7.0).all()
    assert ((wide.cpu().double() - want - old.double()).abs() <= bound + 2.0 ** -23 * (want.abs() + old.abs())).all()


# ---- grouped products on CTA pairs -----------------------------------------------------------------------------------
@pytest.mark.parametrize("counts,width,inner,gated", [([1, 0, 32, 33, 256, 257, 15], 72, 200, True), ([300, 513], 128, 136, False), ([0, 0, 5], 64, 64, True),
                                                      ([700], 136, 264, False)])
def test_grouped_products_on_pairs(counts, width, inner, gated):
    """Experts that nobody chose, that got one row, a whole tile, a row more; row tiles in odd number; the plan's table, and both
    products against float64 over the rounded operands: a bfloat16 result of a float32 sum is off by 2^-8 of itself and K 2^-24 of
    the sum of the products' sizes."""
    from xyntetik_runner_b200 import kernels
    if not kernels.pairs_available():
        pytest.skip("no pairs of CTAs on this device")
    g = torch.Generator().manual_seed(sum(counts))
    E, pairs = len(counts), sum(counts)
    ids = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)])[torch.randperm(pairs, generator=g)].int().view(pairs, 1).to(DEV)
    h = torch.randn(pairs, width, generator=g).bfloat16()
    first = (torch.randn(E, (2 if gated else 1) * inner, width, generator=g) * width ** -0.5).bfloat16()
    second = (torch.randn(E, width, inner, generator=g) * inner ** -0.5).bfloat16()
    max_tiles, rows = kernels.moe_tiles_room(pairs, E)
    row_src, pair_row = torch.empty(rows, dtype=torch.int32, device=DEV), torch.empty(pairs, dtype=torch.int32, device=DEV)
    tiles = torch.full((1 + 3 * max_tiles,), -7, dtype=torch.int32, device=DEV)
    kernels.moe_plan_tiles(ids, row_src, pair_row, tiles, E)
    table = tiles[1:1 + 3 * int(tiles[0])].view(-1, 3).cpu().tolist()
    seen = {}
    for e, at, n in table:
        assert 1 <= n <= kernels.PAIR_TILE and at >= 0 and at + n <= rows
        for r in range(at, at + n):
            assert r not in seen
            seen[r] = e
    assert sorted(seen) == sorted(pair_row.tolist()) and len(table) == sum(-(-c // kernels.PAIR_TILE) for c in counts)
    assert all(seen[r] == int(e) for r, e in zip(pair_row.tolist(), ids[:, 0].tolist()))
    assert row_src[pair_row.long()].tolist() == list(range(pairs)) and int((row_src >= 0).sum()) == pairs
    xs = torch.full((rows, width), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.moe_gather(h.to(DEV), xs, row_src, None, 1)
    y = torch.full((rows, inner), float("nan"), dtype=torch.bfloat16, device=DEV)
    act = kernels.ACT_SILU if gated else kernels.ACT_RELU2
    kernels.gemm_tc_grouped_pairs(xs, kernels.pack_weight_groups(first.to(DEV), 2 if gated else 1), y, tiles, max_tiles, inner,
                                  kernels.EPI_GATED if gated else kernels.EPI_STORE, act)
    zz = torch.full((rows, width), float("nan"), device=DEV)
    kernels.gemm_tc_grouped_pairs(y, kernels.pack_weight_groups(second.to(DEV)), zz, tiles, max_tiles, width)
    kernels.tc_check_status(torch.device(DEV))
    got_y, got = y[pair_row.long()].cpu().double(), zz[pair_row.long()].cpu().double()
    for e in range(E):
        mine = (ids[:, 0] == e).cpu()
        w = first[e].double()
        a = h[mine].double()
        z = a @ w.T
        want = torch.nn.functional.silu(z[:, :inner]) * z[:, inner:] if gated else torch.relu(z) ** 2
        # (the sums' own error, width 2^-24 of sums of a few units, is far below the rounding; the hardware's exponential is good to 2^-21)
        assert ((got_y[mine] - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()
        b, v = got_y[mine], second[e].double()
        assert ((got[mine] - b @ v.T).abs() <= (inner + 2) * 2.0 ** -24 * (b.abs() @ v.abs().T) + 1e-12).all()


# ---- attention over expanded keys ------------------------------------------------------------------------------------
@pytest.mark.parametrize("H,D,R,V,page,window,gate", [(3, 128, 64, 128, 64, 0, "each"), (2, 64, 32, 64, 16, 100, "head"), (2, 64, 8, 128, 64, 0, ""),
                                                      (1, 128, 40, 64, 8, 300, "head")])
def test_attention_over_expanded_keys(H, D, R, V, page, window, gate):
    """Portions that start a request, continue one, are too short (another kernel's), and see keys behind a window, with one key that
    stands out; the rows' gather, then the attention, against float64 over the same operands."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(D + R)
    C = 24
    specs = [(0, 130), (700, 5), (515, 33), (128, 128)]
    mp = -(-max(p + n for p, n in specs) // page)
    pages = mp * len(specs)
    cache = torch.zeros(pages, page, C + R).bfloat16()
    bt = torch.randperm(pages, generator=g).view(len(specs), mp).int()
    rows = [torch.randn(p + n, C + R, generator=g).bfloat16() for p, n in specs]
    for s, r in enumerate(rows):
        for j in range(len(r)):
            cache[bt[s, j // page], j % page] = r[j]
        if window:                                                   # pages behind the window of the portion's first token are gone
            for i in range(max(0, specs[s][0] - window + 1) // page):
                bt[s, i] = -1
    n = sum(m for _, m in specs)
    starts = [sum(m for _, m in specs[:s]) for s in range(len(specs))]
    wk, wv = torch.randn(H * D, C, generator=g) * C ** -0.5, torch.randn(H * V, C, generator=g) * C ** -0.5
    q = torch.randn(n, H * (D + R) + 8, generator=g).bfloat16()
    gates = torch.randn(n, H * V if gate == "each" else H, generator=g).bfloat16()
    first = [int(kernels.flat_first_key(np.int64(p), window)) for p, _ in specs]
    keys = sum(p + m - f for (p, m), f in zip(specs, first) if m >= 32)
    flat = torch.full((keys, C + R), 9.0, dtype=torch.bfloat16, device=DEV)
    seg_len, pos0 = _i32([m for _, m in specs]), _i32([p for p, _ in specs])
    cache_d, bt_d = cache.to(DEV), bt.to(DEV)
    kernels.flat_rows(cache_d.data_ptr(), page * (C + R), flat, seg_len, pos0, bt_d, len(specs), mp, page, window, 32)
    want_rows = []
    for s, (p, m) in enumerate(specs):
        if m >= 32:
            r = rows[s].clone()
            if window:
                r[:max(0, p - window + 1) // page * page] = 0
            want_rows.append(r[first[s]:])
    want_rows = torch.cat(want_rows)
    assert torch.equal(flat.cpu(), want_rows)
    kv = torch.cat([want_rows[:, :C].float() @ wk.T, want_rows[:, :C].float() @ wv.T], dim=1).bfloat16()
    scale = (D + R) ** -0.5
    # head 0 of the third portion's last token looks for that request's key 500 or what the window leaves of it
    far = 540
    at = sum(len(rows[s]) - first[s] for s in (0,)) + far - first[2]
    q[starts[2] + 32, :D] = (kv[at, :D].float() * 6).bfloat16()
    out = torch.full((n, H * V), 5.0, dtype=torch.bfloat16, device=DEV)
    tiles = sum(-(-m // 128) for _, m in specs if m >= 32)
    kernels.attention_tc_flat(q.to(DEV), kv.to(DEV), flat[:, C:], out, _i32(starts), seg_len, pos0, len(specs), H, D, R, V, window, scale, 32, tiles,
                              gate=gates.to(DEV) if gate else None, gate_each=gate == "each")
    kernels.tc_check_status(torch.device(DEV))
    got = out.cpu().double()
    assert (got[starts[1]:starts[1] + 5] == 5.0).all()
    at = 0
    for s, (p, m) in enumerate(specs):
        if m < 32:
            continue
        k = kv[at:at + p + m - first[s]].double()
        tail = want_rows[at:at + p + m - first[s], C:].double()
        at += len(k)
        pos, key = torch.arange(p, p + m)[:, None], torch.arange(first[s], p + m)[None, :]
        see = (key <= pos) & ((pos - key < window) if window else torch.ones_like(key <= pos))
        for h in range(H):
            qh = q[starts[s]:starts[s] + m, h * (D + R):(h + 1) * (D + R)].double()
            sc = (qh[:, :D] @ k[:, h * D:(h + 1) * D].T + qh[:, D:] @ tail.T) * scale
            o = torch.softmax(sc.masked_fill(~see, float("-inf")), dim=-1) @ k[:, H * D + h * V:H * D + (h + 1) * V]
            if gate:
                z = gates[starts[s]:starts[s] + m].double()
                o = o * torch.sigmoid(z[:, h * V:(h + 1) * V] if gate == "each" else z[:, h:h + 1])
            # probabilities are rounded to bfloat16 (2^-9 of each, weights that sum to one) and the result once more
            top = k[:, H * D + h * V:H * D + (h + 1) * V].abs().max()
            assert ((got[starts[s]:starts[s] + m, h * V:(h + 1) * V] - o).abs() <= 2.0 ** -8 * o.abs() + 2.0 ** -8 * top).all(), (s, h)


# ---- the gated linear recurrence of long portions --------------------------------------------------------------------
@pytest.mark.parametrize("R,B,taps,lens,dtype", [(48, 2, 4, [70, 1, 33], torch.bfloat16), (33, 3, 1, [65], torch.bfloat16),
                                                 (256, 1, 3, [31, 320], torch.float32), (1280, 5, 4, [300, 257], torch.bfloat16)])
def test_gated_recurrence_of_long_portions(R, B, taps, lens, dtype):
    """Portions of fewer tokens than segments, of a token more, of many; the products in each of their tiles; two launches, the second
    from the state the first left.  Decays near one over 300 steps: the float32 walk's error grows with the steps it sums over."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(R)
    Bs = R // B
    f = lambda *s: torch.randn(*s, generator=g)
    conv, cb, wa, wi, ba, bi, lam = f(R, taps), f(R), f(B, Bs, Bs) / Bs ** 0.5, f(B, Bs, Bs) / Bs ** 0.5, f(R), f(R), -4.0 + f(R)
    rows = [f(n, 2 * R) for n in lens]

    def plain(x):
        x = x.double()
        u = cb.double().expand(len(x), R).clone()
        for j in range(taps):
            u[j:] += conv[:, taps - 1 - j].double() * x[:len(x) - j, R:]
        ub = u.view(len(x), B, Bs)
        r = torch.sigmoid(torch.einsum("boi,tbi->tbo", wa.double(), ub).reshape(len(x), R) + ba)
        i = torch.sigmoid(torch.einsum("boi,tbi->tbo", wi.double(), ub).reshape(len(x), R) + bi)
        log_a = -8.0 * r * torch.nn.functional.softplus(lam.double())
        inp = torch.sqrt(-torch.expm1(2 * log_a)) * i * u
        S, out = torch.zeros(R, dtype=torch.float64), []
        for t in range(len(x)):
            S = torch.exp(log_a[t]) * S + inp[t]
            out.append(S)
        return torch.stack(out) * torch.nn.functional.gelu(x[:, :R], approximate="tanh"), S

    state = torch.zeros(len(lens) + 1, kernels.rglru_state_floats(R, taps), device=DEV)
    slots = list(range(len(lens), 0, -1))
    cut = [max(1, n // 3) for n in lens]
    got = [[] for _ in lens]
    for part in range(2):
        xs = [r[:c] if part == 0 else r[c:] for r, c in zip(rows, cut)]
        use = [s for s, x in enumerate(xs) if len(x)]
        x = torch.cat([xs[s] for s in use]).to(DEV)
        ln = [len(xs[s]) for s in use]
        st = [sum(ln[:i]) for i in range(len(ln))]
        n = len(x)
        a, b, u = (torch.empty(n, R, device=DEV) for _ in range(3))
        out = torch.empty(n, R, dtype=dtype, device=DEV)
        kernels.rglru(x, conv.to(DEV), cb.to(DEV), None, None, wa.to(DEV), wi.to(DEV), ba.to(DEV), bi.to(DEV), lam.to(DEV), state,
                      _i32([i for i, m in enumerate(ln) for _ in range(m)]), _i32(st), _i32(ln), _i32([slots[s] for s in use]), a, b, u, out, len(ln), R, B,
                      taps, 8.0)
        for i, s in enumerate(use):
            got[s].append(out[st[i]:st[i] + ln[i]].cpu().double())
    assert state[0].abs().sum() == 0
    for s, r in enumerate(rows):
        want, end = plain(r)
        assert torch.allclose(torch.cat(got[s]), want, rtol=5e-5 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0), atol=1e-5)
        assert torch.allclose(state[slots[s], :R].cpu().double(), end, rtol=5e-5, atol=1e-5)
        tail = torch.zeros(taps - 1, R)
        keep = min(taps - 1, len(r))
        if keep:
            tail[taps - 1 - keep:] = r[len(r) - keep:, R:]
        assert torch.equal(state[slots[s], R:].cpu().view(taps - 1, R), tail)


# ---- recurrences in chunks -------------------------------------------------------------------------------------------
def _walk(q, k, v, decay, S):
    """S <- decay S + k v^T, o = S^T q in float64; q, k [T, H, D], v [T, H, V], decay [T, H, D]."""
    out = []
    for t in range(len(q)):
        S = decay[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
        out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    return torch.stack(out), S


def _close(got, want, walk):
    """No further from float64 than a few units of float32 of the largest value, and no further than three times the walk is."""
    far, near = (got.double() - want).abs().max(), (walk.double() - want).abs().max()
    assert far <= max(3.0 * near, 4e-6 * want.abs().max()), (far, near, want.abs().max())


CHUNKED = [("head", 2, 64, 64), ("head", 1, 128, 128), ("key", 2, 64, 128), ("key", 1, 128, 64), ("key deep", 1, 64, 64)]


@pytest.mark.parametrize("kind,H,D,V", CHUNKED)
def test_recurrences_in_chunks(kind, H, D, V):
    """Portions of a token, of a chunk, of a chunk and a token, of several, from states that hold something, against float64 and
    beside the walk on the same inputs: read-outs, new states, other slots.  "deep": decays that clear the memory within a chunk next
    to decays near one, where exponentials of sums would overflow or lose their digits."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(H * D + V + len(kind))
    f = lambda *s: torch.randn(*s, generator=g)
    lens, slots = [130, 1, 64, 65], [3, 0, 4, 1]
    n, S = sum(lens), len(lens)
    starts = [sum(lens[:i]) for i in range(S)]
    state0 = f(6, H * V * D)
    q, k, v = f(n, H, D), f(n, H, D) * D ** -0.5, f(n, H, V)
    if kind == "head":
        dec = torch.tensor([1.0 - 2.0 ** -(2 + 6 * h) for h in range(H)])
        proj = torch.cat([q.reshape(n, -1), k.reshape(n, -1), v.reshape(n, -1)], 1).to(DEV)
        decay = dec.double()[None, :, None].expand(n, H, D)

        def run(state, scratch):
            o = torch.empty(n, H * V, device=DEV)
            kernels.decay_attention(proj, (0, H * D, 2 * H * D), dec.to(DEV), state, _i32(starts), _i32(lens), _i32(slots), o, S, H, D, V, silu=False,
                                    read_scale=0.5, scratch=scratch)
            return o
        floats = kernels.chunked_floats(n, S, H, D, V, "head")
    else:
        R, tau = 8, 12.0
        inner, w_t, bias = f(n, R), f(R, H * D), 2.0 + f(H * D)
        if kind.endswith("deep"):
            inner[::13] *= 200.0
        proj = torch.cat([q.reshape(n, -1), k.reshape(n, -1), v.reshape(n, -1), inner], 1).to(DEV)
        z = inner.double() @ w_t.double() + bias
        decay = torch.exp(torch.nn.functional.logsigmoid(z) / tau).view(n, H, D)

        def run(state, scratch):
            o = torch.empty(n, H * V, device=DEV)
            kernels.key_decay_attention(proj, (0, H * D, 2 * H * D, 2 * H * D + H * V), R, w_t.to(DEV), bias.to(DEV), tau, torch.empty(n, H * D, device=DEV),
                                        state, _i32(starts), _i32(lens), _i32(slots), o, S, H, D, V, read_scale=0.5, scratch=scratch)
            return o
        floats = kernels.chunked_floats(n, S, H, D, V, "key")
    q = q * 0.5
    assert floats > 0
    walk_state, state = state0.to(DEV).clone(), state0.to(DEV).clone()
    by_walk = run(walk_state, None).cpu()
    got = run(state, torch.full((floats,), float("nan"), device=DEV)).cpu()
    assert torch.equal(state[2].cpu(), state0[2]) and torch.equal(state[5].cpu(), state0[5])
    for i, (m, slot) in enumerate(zip(lens, slots)):
        at = slice(starts[i], starts[i] + m)
        before = state0[slot].double().view(H, V, D).transpose(1, 2)
        want, end = _walk(q[at].double(), k[at].double(), v[at].double(), decay[at].double(), before)
        _close(got[at], want.reshape(m, -1), by_walk[at])
        _close(state[slot].cpu(), end.transpose(1, 2).reshape(-1), walk_state[slot].cpu())


@pytest.mark.parametrize("H,D,V,dtype", [(2, 64, 128, torch.float32), (1, 128, 64, torch.bfloat16), (3, 128, 256, torch.bfloat16)])
def test_matrix_memory_with_gates_in_chunks(H, D, V, dtype):
    """The same for the cell with exponential input gates: gates far apart, a maximum that moves, a forget gate near zero."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(H * D + V)
    f = lambda *s: torch.randn(*s, generator=g)
    lens, slots, cap = [300, 1, 64], [2, 0, 3], 15.0
    n, S = sum(lens), len(lens)
    starts = [sum(lens[:i]) for i in range(S)]
    proj = f(n, 2 * H * D + 2 * H * V).to(dtype)
    gates = torch.cat([4.0 * f(n, H), 3.0 + 2.0 * f(n, H)], dim=1)
    gates[::41, H:] = -40.0
    size = D * V + D + 1
    state0 = f(4, H, size)
    state0[..., -1] = state0[..., -1].abs()
    norm_w = torch.ones(H * V)

    def run(state, scratch):
        o, y = torch.empty(n, H * V, device=DEV), torch.empty(n, H * V, dtype=dtype, device=DEV)
        kernels.mlstm(proj.to(DEV), (0, H * D, 2 * H * D, 2 * H * D + H * V), gates.to(DEV), state, torch.empty(n, 3 * H, device=DEV), o, norm_w.to(DEV), y,
                      _i32(starts), _i32(lens), _i32(slots), S, H, D, V, cap, 1e-6, scratch=scratch)
        return o.cpu()
    walk_state, state = state0.reshape(4, -1).to(DEV).clone(), state0.reshape(4, -1).to(DEV).clone()
    by_walk = run(walk_state, None)
    got = run(state, torch.full((kernels.chunked_floats(n, S, H, D, V, "mlstm"),), float("nan"), device=DEV))
    assert torch.equal(state[1].cpu(), state0[1].reshape(-1))
    p = proj.double()
    q, k, v = p[:, :H * D].view(n, H, D) * D ** -0.5, p[:, H * D:2 * H * D].view(n, H, D), p[:, 2 * H * D:2 * H * D + H * V].view(n, H, V)
    li = cap * torch.tanh(gates[:, :H].double() / cap)
    lf = torch.nn.functional.logsigmoid(cap * torch.tanh(gates[:, H:].double() / cap))
    for i, (m, slot) in enumerate(zip(lens, slots)):
        st = state0[slot].double()
        Sm, nm, mx = st[:, :D * V].reshape(H, D, V), st[:, D * V:D * V + D], st[:, -1]
        Sa, na = Sm.abs(), nm.abs()                      # the same sums over sizes: what a rounding of a term can be a share of
        out, bound = [], []
        for t in range(starts[i], starts[i] + m):
            new = torch.maximum(lf[t] + mx, li[t])
            a, s = torch.exp(lf[t] + mx - new), torch.exp(li[t] - new)
            Sm = a[:, None, None] * Sm + s[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
            nm = a[:, None] * nm + s[:, None] * k[t]
            mx = new
            Sa = a[:, None, None] * Sa + s[:, None, None] * k[t].abs()[:, :, None] * v[t].abs()[:, None, :]
            na = a[:, None] * na + s[:, None] * k[t].abs()
            den = torch.maximum((nm * q[t]).sum(-1).abs(), torch.exp(-mx)) + 1e-6
            o = torch.einsum("hdv,hd->hv", Sm, q[t]) / den[:, None]
            size = torch.einsum("hdv,hd->hv", Sa, q[t].abs()) + o.abs() * (na * q[t].abs()).sum(-1)[:, None]
            out.append(o.reshape(-1))
            bound.append((size / den[:, None]).reshape(-1))
        at = slice(starts[i], starts[i] + m)
        # numerator and denominator: a term passes at most 64 additions of its chunk's memory, 6 of the scan, 16 + 8 of a score, 32 + 6
        # of the last product, and a dozen products and exponentials; the denominator may cancel, so the terms' sizes count
        assert ((got[at].double() - torch.stack(out)).abs() <= 144 * 2.0 ** -24 * torch.stack(bound)).all()
        end = torch.cat([Sm.reshape(H, -1), nm, mx[:, None]], dim=1).reshape(-1)
        _close(state[slot].cpu(), end, walk_state[slot].cpu())


# ---- recurrences a token a step ---------------------------------------------------------------------------------------
@pytest.mark.parametrize("kind,H,D,V", [("head", 3, 64, 40), ("head", 2, 128, 128), ("head", 1, 100, 4), ("key", 2, 36, 24), ("key", 1, 128, 72), ("ssd", 2, 64, 64),
                                        ("ssd", 4, 100, 20)])
def test_single_tokens_follow_the_walk_bit_for_bit(kind, H, D, V):
    """Two requests' tokens in steps of one token each against the same tokens in one step: read-outs, states and tails."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(H * D + V)
    f = lambda *s: torch.randn(*s, generator=g).to(DEV)
    S, T, taps, slots = 2, 7, 4, [2, 0]
    G, R = H // 2 if kind == "ssd" else H, 8
    CH = H * V + 2 * G * D
    width = CH + H if kind == "ssd" else 2 * H * D + H * V + (R if kind == "key" else 0)
    rows = f(S, T, width)
    dec, w_t, bias = torch.rand(H, generator=g).to(DEV), f(R, H * D), f(H * D)
    conv, cb, dtb, neg_a, skip = f(CH, taps), f(CH), f(H), -torch.rand(H, generator=g).to(DEV), f(H)
    state0 = f(4, kernels.ssd_state_floats(H, G, D, V, taps) if kind == "ssd" else H * D * V)

    def step(x, counts, state):
        n = x.shape[0]
        starts, o = [0, counts[0]], torch.empty(n, H * V, device=DEV)
        where = (state, _i32(starts), _i32(counts), _i32(slots))
        if kind == "head":
            kernels.decay_attention(x.clone(), (0, H * D, 2 * H * D), dec, *where, o, S, H, D, V, read_scale=0.5)
        elif kind == "key":
            kernels.key_decay_attention(x, (0, H * D, 2 * H * D, 2 * H * D + H * V), R, w_t, bias, 3.0, torch.empty(n, H * D, device=DEV), *where, o, S, H, D, V)
        else:
            kernels.ssd(x, 0, CH, conv, cb, dtb, neg_a, skip, state, _i32([0] * counts[0] + [1] * counts[1]), *where[1:], torch.empty(n, CH, device=DEV),
                        torch.empty(n, 2 * H, device=DEV), o, S, H, G, D, V, taps)
        return o.view(S, -1, H * V)
    whole, single = state0.clone(), state0.clone()
    want = step(rows.reshape(S * T, width), [T, T], whole)
    got = torch.cat([step(rows[:, t].contiguous(), [1, 1], single) for t in range(T)], dim=1)
    assert torch.equal(got, want) and torch.equal(single, whole) and torch.equal(whole[1], state0[1]) and not torch.equal(whole[0], state0[0])


# ---- streams of many rows ----------------------------------------------------------------------------------------------
@pytest.mark.parametrize("n,width,dtype", [(33, 2048, torch.bfloat16), (40, 4096, torch.float32), (35, 2052, torch.bfloat16), (34, 70, torch.bfloat16),
                                           (33, 36, torch.float32)])
def test_streams_of_many_rows(n, width, dtype):
    """Rows that take 16 bytes an access and rows that do not, the widest that stay in registers: the norm that is added, the average over
    depth, the scaled sum; what is cleared is zero.  A norm's sum of `width` squares and three more roundings; an average's k + 1 terms."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + width)
    f = lambda *s: torch.randn(*s, generator=g)
    eps32 = 2.0 ** -24
    half = 2.0 ** -8 if dtype == torch.bfloat16 else eps32
    d0, x0, gain = f(n, width), f(n, width), torch.tensor([0.7])
    d, x, cast = d0.to(DEV), x0.to(DEV), torch.empty(n, width, dtype=dtype, device=DEV)
    kernels.norm_add(d, x, gain.to(DEV), 1e-5, cast=cast, clear=True)
    add = d0.double() / torch.sqrt(d0.double().pow(2).mean(1, keepdim=True) + 1e-5) * 0.7
    want = x0.double() + add
    tol = eps32 * (want.abs() + (width + 4) * add.abs())
    assert ((x.cpu().double() - want).abs() <= tol).all() and ((cast.cpu().double() - want).abs() <= tol + half * want.abs()).all() and not d.any()
    k = 10
    first, hist, w = f(n, width), f(k, n, width), f(k + 1)
    x, past = x0.to(DEV), hist.to(DEV)
    kernels.depth_average(x, first.to(DEV), past, w.to(DEV), k, cast=cast)
    terms = torch.cat([first[None], hist[:k - 1], x0[None]]).double() * w.double()[:, None, None]
    want, tol = terms.sum(0), (k + 1) * eps32 * terms.abs().sum(0)
    assert ((x.cpu().double() - want).abs() <= tol).all() and ((cast.cpu().double() - want).abs() <= tol + half * want.abs()).all()
    assert torch.equal(past.cpu(), torch.cat([hist[:k - 1], x0[None]]))
    for clear in (False, True):
        d, x = d0.to(DEV), x0.to(DEV)
        kernels.scaled_add(x, d, 0.3, clear=clear)
        assert torch.allclose(x.cpu(), x0 + 0.3 * d0, rtol=1e-6, atol=1e-6) and torch.equal(d.cpu(), torch.zeros_like(d0) if clear else d0)


# ---- choice, plan and gather of few tokens in one launch -------------------------------------------------------------
@pytest.mark.parametrize("n,E,identity,top,mode,splits,align", [(1, 16, 0, 2, 0, 1, 16), (8, 64, 0, 6, 0, 8, 16), (32, 16, 0, 2, 1, 3, 16), (40, 12, 4, 2, 2, 2, 16),
                                                                (64, 3, 0, 3, 0, 9, 32), (85, 40, 0, 3, 1, 1, 16)])
def test_route_few_against_its_parts(n, E, identity, top, mode, splits, align):
    """The same choice and weights as the kernels it stands for; a plan that gives every pair a row in a tile of its expert and no two
    the same; the rows themselves; tiles without rows marked; columns behind the router's outputs carried along."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + E)
    outputs, W, extra = E + identity, 64, 0 if mode == 2 else 1
    ldz = outputs + extra
    parts = torch.randn(splits, n, ldz, generator=g).to(DEV)
    h = torch.randn(n, W, generator=g).bfloat16().to(DEV)
    corr = None if mode == 0 else (0.3 * torch.randn(outputs, generator=g)).to(DEV)
    total = parts[0].clone()
    for s in range(1, splits):
        total += parts[s]
    zs = total.clone() if splits == 1 else torch.full((n, ldz), float("nan"), device=DEV)
    pairs = n * top
    mt = kernels.moe_max_tiles(pairs, E, align)
    wts, pair_row = torch.empty(n, top, device=DEV), torch.empty(pairs, dtype=torch.int32, device=DEV)
    tile_group = torch.full((mt,), 77, dtype=torch.int32, device=DEV)
    xs = torch.full((mt * align, W), 3.0, dtype=torch.bfloat16, device=DEV)
    groups = (4, 2) if mode == 2 else (1, 1)
    kernels.route_few(zs if splits == 1 else parts, splits, zs, outputs, E, top, wts, pair_row, tile_group, align, h, xs, mode, corr, *groups, 1.7)
    assert torch.equal(zs, total)
    ids, want = torch.empty(n, top, dtype=torch.int32, device=DEV), torch.empty(n, top, device=DEV)
    if mode == 2:
        kernels.route_groups(zs, ids, want, top, corr, *groups, 1.7)
    else:
        kernels.route_topk(zs[:, :outputs], ids, want, top, sigmoid_scores=mode == 1, correction=corr)
    assert torch.equal(wts, want)
    ids, rows, tiles = ids.reshape(-1).tolist(), pair_row.tolist(), tile_group.tolist()
    real = [r for r in rows if r >= 0]
    assert len(set(real)) == len(real)
    for p, (e, r) in enumerate(zip(ids, rows)):
        assert (r < 0) == (e >= E)
        if r >= 0:
            assert tiles[r // align] == e and torch.equal(xs[r], h[p // top])
    used = sum(-(-ids.count(e) // align) for e in range(E))
    assert all(0 <= t < E for t in tiles[:used]) and all(t == -1 for t in tiles[used:])


@pytest.mark.parametrize("kind,H,D,V", [("head", 2, 64, 64), ("key", 1, 128, 64), ("mlstm", 2, 64, 128)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_chunks_do_not_look_ahead(kind, H, D, V, bad):
    """A value that is no number, in the middle of a chunk: the read-outs of the tokens before it, of other columns and of other
    portions are bit for bit what they are without it, and those from it on are what the walk makes of them: no numbers."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(D + V)
    f = lambda *s: torch.randn(*s, generator=g)
    lens, token, column = [90, 70], 64 + 11, 5
    n, S = sum(lens), 2
    starts, slots = [0, 90], [1, 0]
    state0 = f(2, H, D * V + D + 1 if kind == "mlstm" else D * V)
    state0[..., -1] = 0.5
    proj0, gates = f(n, 2 * H * D + 2 * H * V + 8) * 0.3, torch.cat([f(n, H), 3.0 + f(n, H)], dim=1)
    dec, w_t, bias = torch.rand(H, generator=g) * 0.1 + 0.9, f(8, H * D), 2.0 + f(H * D)

    def run(planted, chunked):
        proj = proj0.clone()
        if planted:
            proj[token, 2 * H * D + column] = bad
        proj, state, o = proj.to(DEV), state0.reshape(2, -1).to(DEV).clone(), torch.empty(n, H * V, device=DEV)
        seg = (_i32(starts), _i32(lens), _i32(slots))
        scratch = torch.full((kernels.chunked_floats(n, S, H, D, V, kind),), float("nan"), device=DEV) if chunked else None
        if kind == "head":
            kernels.decay_attention(proj, (0, H * D, 2 * H * D), dec.to(DEV), state, *seg, o, S, H, D, V, silu=False, scratch=scratch)
        elif kind == "key":
            kernels.key_decay_attention(proj, (0, H * D, 2 * H * D, 2 * H * D + 2 * H * V), 8, w_t.to(DEV), bias.to(DEV), 12.0,
                                        torch.empty(n, H * D, device=DEV), state, *seg, o, S, H, D, V, scratch=scratch)
        else:
            kernels.mlstm(proj, (0, H * D, 2 * H * D, 2 * H * D + H * V), gates.to(DEV), state, torch.empty(n, 3 * H, device=DEV), o,
                          torch.ones(H * V, device=DEV), torch.empty(n, H * V, device=DEV), *seg, S, H, D, V, 15.0, 1e-6, scratch=scratch)
        return o.cpu()
    clean, got, walk = run(False, True), run(True, True), run(True, False)
    assert torch.isfinite(clean).all()
    touched = torch.zeros(n, H * V, dtype=torch.bool)
    touched[token:lens[0], column] = True
    assert torch.equal(got[~touched], clean[~touched])
    assert not torch.isfinite(got[touched]).any() and not torch.isfinite(walk[touched]).any() and torch.isfinite(walk[~touched]).all()


@pytest.mark.parametrize("token", [0, 70, 299])
@pytest.mark.parametrize("which", ["forget", "input"])
def test_gates_that_are_no_numbers_in_chunks(token, which):
    """A gate of one head that is no number: the same read-outs, states and running maxima are numbers as in the walk, and what comes
    before it, the other head and the other portion keep their bits."""
    from xyntetik_runner_b200 import kernels
    H, D, V = 2, 64, 64
    g = torch.Generator().manual_seed(token)
    f = lambda *s: torch.randn(*s, generator=g)
    lens, starts, slots = [300, 40], [0, 300], [0, 1]
    n, size = sum(lens), D * V + D + 1
    proj, gates0, state0 = f(n, 2 * H * D + 2 * H * V), torch.cat([f(n, H), 3.0 + f(n, H)], dim=1), f(2, H, size)
    state0[..., -1] = 0.5

    def run(planted, chunked):
        gates = gates0.clone()
        if planted:
            gates[token, (H if which == "forget" else 0) + 1] = float("nan")
        state, o = state0.reshape(2, -1).to(DEV).clone(), torch.empty(n, H * V, device=DEV)
        scratch = torch.empty(kernels.chunked_floats(n, 2, H, D, V, "mlstm"), device=DEV) if chunked else None
        kernels.mlstm(proj.to(DEV), (0, H * D, 2 * H * D, 2 * H * D + H * V), gates.to(DEV), state, torch.empty(n, 3 * H, device=DEV), o,
                      torch.ones(H * V, device=DEV), torch.empty(n, H * V, device=DEV), _i32(starts), _i32(lens), _i32(slots), 2, H, D, V, 15.0, 1e-6,
                      scratch=scratch)
        return o.cpu(), state.cpu()
    (clean, clean_state), (got, state), (walk, walk_state) = run(False, True), run(True, True), run(True, False)
    assert torch.equal(torch.isnan(got), torch.isnan(walk)) and torch.equal(torch.isnan(state), torch.isnan(walk_state))
    assert torch.isnan(got[token:300, V:]).all() and torch.isfinite(clean).all()
    for same in (got[:token] == clean[:token], got[:, :V] == clean[:, :V], got[300:] == clean[300:], state[1] == clean_state[1], state[0, :size] == clean_state[0, :size]):
        assert same.all()


@pytest.mark.parametrize("what", ["keys", "decays"])
def test_scores_of_chunks_out_of_the_short_cuts_range(what):
    """Decays per channel that reach exp(-59) over a chunk: with keys of 1e14 (and queries as small) exp(-c) k leaves float32's range where the
    walk does not; and a decay that is no number leaves the tokens before it what they are, however far their decays have gone."""
    from xyntetik_runner_b200 import kernels
    H, D, V, n, token = 1, 64, 64, 150, 110
    g = torch.Generator().manual_seed(9)
    f = lambda *s: torch.randn(*s, generator=g)
    scale = 1e14 if what == "keys" else 1.0
    q, k, v = f(n, H * D) / scale, f(n, H * D) * D ** -0.5 * scale, f(n, H * V)
    inner, w_t = torch.zeros(n, 8), torch.zeros(8, H * D)
    w_t[0] = 1.0
    if what == "decays":
        inner[token:, 0] = float("nan")
    z = -11.06 if what == "keys" else -36.0
    proj = torch.cat([q, k, v, inner], 1).to(DEV)
    state0 = f(1, H * D * V) * scale

    def run(chunked):
        state, o = state0.to(DEV).clone(), torch.empty(n, H * V, device=DEV)
        kernels.key_decay_attention(proj, (0, H * D, 2 * H * D, 2 * H * D + H * V), 8, w_t.to(DEV), torch.full((H * D,), z).to(DEV), 12.0,
                                    torch.empty(n, H * D, device=DEV), state, _i32([0]), _i32([n]), _i32([0]), o, 1, H, D, V,
                                    scratch=torch.empty(kernels.chunked_floats(n, 1, H, D, V, "key"), device=DEV) if chunked else None)
        return o.cpu()
    walk, got = run(False), run(True)
    upto = n if what == "keys" else token
    decay = torch.exp(torch.nn.functional.logsigmoid(torch.tensor(z, dtype=torch.float64)) / 12.0).expand(upto, H, D)
    want, _ = _walk(q[:upto].double().view(-1, H, D), k[:upto].double().view(-1, H, D), v[:upto].double().view(-1, H, V), decay,
                    state0.double().view(H, V, D).transpose(1, 2))
    _close(got[:upto], want.reshape(upto, -1), walk[:upto])
    assert torch.equal(torch.isnan(got), torch.isnan(walk))


@pytest.mark.parametrize("each", [False, True])
def test_gates_of_expanded_attention_keep_float32(each):
    """Output gates far on either side: sigmoid(z) in float32 down to its smallest values; the results differ from float64 by their
    rounding to bfloat16, the probabilities' and 2^-16 of a gate that float32 holds without its leading bit."""
    from xyntetik_runner_b200 import kernels
    H, D, R, V, n = 2, 64, 8, 64, 40
    g = torch.Generator().manual_seed(1)
    f = lambda *s: torch.randn(*s, generator=g).bfloat16()
    q, kv, tail = f(n, H * (D + R)), f(n, H * (D + V)), f(n, R)
    kv[:, H * D:] = (1000.0 + 100.0 * kv[:, H * D:].float()).bfloat16()
    z = torch.tensor([-88.0, -87.5, -86.0, -60.0, -5.0, 0.0, 4.0, 60.0, 88.0, 100.0]).repeat(n, H * V // 10 + 1)[:, :H * V if each else H].bfloat16()
    z = torch.stack([row.roll(t) for t, row in enumerate(z)]).contiguous() if each else z.flatten().roll(3).view(n, H).contiguous()
    if not each:
        z[:, 0] = torch.tensor([-88.0, -87.5, -60.0, 0.0, 88.0]).repeat(n // 5).bfloat16()
    out = torch.empty(n, H * V, dtype=torch.bfloat16, device=DEV)
    kernels.attention_tc_flat(q.to(DEV), kv.to(DEV), tail.to(DEV), out, _i32([0]), _i32([n]), _i32([0]), 1, H, D, R, V, 0, 0.05, 32, 1, gate=z.to(DEV),
                              gate_each=each)
    kernels.tc_check_status(torch.device(DEV))
    see = torch.arange(n)[:, None] >= torch.arange(n)[None, :]
    for h in range(H):
        qh, kh, vh = (t.double() for t in (q[:, h * (D + R):(h + 1) * (D + R)], kv[:, h * D:(h + 1) * D], kv[:, H * D + h * V:H * D + (h + 1) * V]))
        o = torch.softmax(((qh[:, :D] @ kh.T + qh[:, D:] @ tail.double().T) * 0.05).masked_fill(~see, float("-inf")), dim=-1) @ vh
        o = o * torch.sigmoid(z.double()[:, h * V:(h + 1) * V] if each else z.double()[:, h:h + 1])
        assert ((out[:, h * V:(h + 1) * V].double().cpu() - o).abs() <= (2.0 ** -8 + 2.0 ** -8) * o.abs()).all()


@pytest.mark.parametrize("n,n_out,k,wdt,skip,extra", [(9, 70, 34, torch.float32, 0, 2), (70, 600, 37, torch.float32, 1, 1), (300, 2001, 66, torch.bfloat16, 0, 0),
                                                      (300, 2001, 68, torch.bfloat16, 0, 3), (70, 600, 64, torch.bfloat16, 2, 0), (65, 4800, 35, torch.float32, 0, 0),
                                                      (300, 2001, 40, torch.bfloat16, 1, 0), (1, 33, 3, torch.bfloat16, 3, 5), (300, 2001, 16, torch.float32, 0, 0),
                                                      (300, 2001, 4, torch.bfloat16, 0, 4)])
def test_float32_product_off_the_copies_borders(n, n_out, k, wdt, skip, extra):
    """Operands whose addresses, rows' distances or K do not allow 16-byte copies, and K of a few values, with few tiles and with many: the
    same bits as the same numbers on 16-byte borders with zeros behind them, stored, added, as bfloat16 behind a factor and a bias."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(n + k + skip)
    x, w = torch.randn(n, k, generator=g), torch.randn(n_out, k, generator=g).to(wdt)
    xs = torch.full((n, k + extra), float("nan"), device=DEV)
    xs[:, :k] = x.to(DEV)
    flat = torch.full((n_out * k + 16,), float("nan"), dtype=wdt, device=DEV)
    flat[skip:skip + n_out * k] = w.to(DEV).reshape(-1)
    pad = -(-k // 8) * 8 + 8
    off = (xs[:, :k], flat[skip:skip + n_out * k].view(n_out, k))
    even = [torch.nn.functional.pad(t.to(DEV), (0, pad - k)).contiguous() for t in (x, w)]
    base, bias = torch.randn(n, n_out, generator=g).to(DEV), torch.randn(n_out, generator=g).to(DEV)
    for kind in ("store", "add", "bf16"):
        got, want = ((base.clone() if kind == "add" else torch.empty(n, n_out, dtype=torch.bfloat16 if kind == "bf16" else torch.float32, device=DEV)) for _ in range(2))
        for (a, b), out in ((off, got), (even, want)):
            kernels.gemm_simt(a, b, out, bias if kind == "bf16" else None, kind == "add", 0.5 if kind == "bf16" else 1.0)
        assert torch.equal(got, want), kind
        if kind == "store":
            bound = (x.double().abs() @ w.double().abs().T) * (k + 2) * 2.0 ** -24
            assert ((got.cpu().double() - x.double() @ w.double().T).abs() <= bound).all()


@pytest.mark.parametrize("kind,H,D,V,lens", [("head", 2, 64, 64, [3, 900, 1, 64]), ("key", 1, 128, 64, [640, 1, 513]), ("key", 2, 64, 128, [1030]),
                                             ("mlstm", 2, 64, 64, [1, 777, 65]), ("mlstm", 1, 128, 64, [1100])])
def test_portions_of_many_chunks(kind, H, D, V, lens):
    """Portions of nine to eighteen chunks, as steps bring them (the memories follow from one another eight chunks at a time), beside short
    ones, in two launches, the second from the first's states: against float64 and beside the walk."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(sum(lens) + D)
    f = lambda *s: torch.randn(*s, generator=g)
    S, n = len(lens), sum(lens)
    starts, slots = [sum(lens[:i]) for i in range(S)], list(range(S, 0, -1))
    size = D * V + (D + 1 if kind == "mlstm" else 0)
    state0 = f(S + 1, H, size)
    if kind == "mlstm":
        state0[..., -1] = 0.5
    dec = torch.tensor([1.0 - 2.0 ** -(4 + 4 * h) for h in range(H)])
    w_t, bias = f(8, H * D), 3.0 + f(H * D)
    rows = []
    for _ in range(2):
        q, k, v = f(n, H * D), f(n, H * D) * (1.0 if kind == "mlstm" else D ** -0.5), f(n, H * V)
        rows.append((torch.cat([q, k, v, f(n, H * V), f(n, 8)], 1), torch.cat([f(n, H), 4.0 + f(n, H)], 1)))

    def run(chunked):
        state, outs = state0.reshape(S + 1, -1).to(DEV).clone(), []
        seg = (_i32(starts), _i32(lens), _i32(slots))
        scratch = torch.full((kernels.chunked_floats(n, S, H, D, V, kind),), float("nan"), device=DEV) if chunked else None
        for proj, gates in rows:
            proj, o = proj.to(DEV), torch.empty(n, H * V, device=DEV)
            if kind == "head":
                kernels.decay_attention(proj, (0, H * D, 2 * H * D), dec.to(DEV), state, *seg, o, S, H, D, V, silu=False, scratch=scratch)
            elif kind == "key":
                kernels.key_decay_attention(proj, (0, H * D, 2 * H * D, 2 * H * D + 2 * H * V), 8, w_t.to(DEV), bias.to(DEV), 12.0,
                                            torch.empty(n, H * D, device=DEV), state, *seg, o, S, H, D, V, scratch=scratch)
            else:
                kernels.mlstm(proj, (0, H * D, 2 * H * D, 2 * H * D + H * V), gates.to(DEV), state, torch.empty(n, 3 * H, device=DEV), o,
                              torch.ones(H * V, device=DEV), torch.empty(n, H * V, device=DEV), *seg, S, H, D, V, 15.0, 1e-6, scratch=scratch)
            outs.append(o.cpu())
        return outs, state.cpu()
    walk, walk_state = run(False)
    got, state = run(True)
    assert torch.equal(state[0], state0[0].reshape(-1))
    for i, (m, slot) in enumerate(zip(lens, slots)):
        at = slice(starts[i], starts[i] + m)
        st = state0[slot].double()
        if kind == "mlstm":
            Sm, nm, mx = st[:, :D * V].reshape(H, D, V), st[:, D * V:D * V + D], st[:, -1]
        else:
            Sm = st.view(H, V, D).transpose(1, 2)
        for part, (proj, gates) in enumerate(rows):
            p = proj[at].double()
            q, k, v = p[:, :H * D].view(m, H, D), p[:, H * D:2 * H * D].view(m, H, D), p[:, 2 * H * D:2 * H * D + H * V].view(m, H, V)
            if kind == "mlstm":
                q = q * D ** -0.5
                li = 15.0 * torch.tanh(gates[at, :H].double() / 15.0)
                lf = torch.nn.functional.logsigmoid(15.0 * torch.tanh(gates[at, H:].double() / 15.0))
                want = []
                for t in range(m):
                    new = torch.maximum(lf[t] + mx, li[t])
                    a, s = torch.exp(lf[t] + mx - new), torch.exp(li[t] - new)
                    Sm = a[:, None, None] * Sm + s[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
                    nm, mx = a[:, None] * nm + s[:, None] * k[t], new
                    want.append(torch.einsum("hdv,hd->hv", Sm, q[t]))            # the numerators: a denominator may cancel
                    den = torch.maximum((nm * q[t]).sum(-1).abs(), torch.exp(-mx)) + 1e-6
                    got[part][starts[i] + t] *= den.float().repeat_interleave(V)
                    walk[part][starts[i] + t] *= den.float().repeat_interleave(V)
                want = torch.stack(want)
            else:
                if kind == "head":
                    decay = dec.double()[None, :, None].expand(m, H, D)
                else:
                    decay = torch.exp(torch.nn.functional.logsigmoid(p[:, -8:] @ w_t.double() + bias) / 12.0).view(m, H, D)
                want, Sm = _walk(q, k, v, decay, Sm)
            _close(got[part][at], want.reshape(m, -1), walk[part][at])
        end = torch.cat([Sm.reshape(H, -1), nm, mx[:, None]], 1).reshape(-1) if kind == "mlstm" else Sm.transpose(1, 2).reshape(-1)
        _close(state[slot], end, walk_state[slot])


def test_gated_recurrence_in_segments_beside_short_portions():
    """The route of long portions, taken for portions of a token, of fewer tokens than segments and of many in one launch: the same as each
    portion alone, and the walk's results in float32."""
    from xyntetik_runner_b200 import kernels
    R, B, taps, lens = 48, 2, 4, [400, 1, 20, 33]
    g = torch.Generator().manual_seed(2)
    f = lambda *s: torch.randn(*s, generator=g).to(DEV)
    Bs, n, S = R // B, sum(lens), len(lens)
    args = (f(R, taps), f(R), None, None, f(B, Bs, Bs) / Bs ** 0.5, f(B, Bs, Bs) / Bs ** 0.5, f(R), f(R), -4.0 + f(R))
    proj0, state0 = f(n, 2 * R), f(S, kernels.rglru_state_floats(R, taps))
    starts = [sum(lens[:i]) for i in range(S)]

    def run(which, dtype):
        rows = torch.cat([proj0[starts[s]:starts[s] + lens[s]] for s in which]).clone()
        ln = [lens[s] for s in which]
        m, state = len(rows), state0.clone()
        a, b, u, out = torch.empty(m, R, device=DEV), torch.empty(m, R, device=DEV), torch.empty(m, R, device=DEV), torch.empty(m, R, dtype=dtype, device=DEV)
        kernels.rglru(rows, *args, state, _i32([i for i, x in enumerate(ln) for _ in range(x)]), _i32([sum(ln[:i]) for i in range(len(ln))]), _i32(ln),
                      _i32(which), a, b, u, out, len(ln), R, B, taps, 8.0)
        return out, state
    got, state = run([0, 1, 2, 3], torch.bfloat16)
    want, want_state = run([0, 1, 2, 3], torch.float32)
    # (a state is a sum of at most 400 terms in another order; a read-out is rounded to bfloat16 behind it)
    assert torch.allclose(got.float(), want, rtol=2.0 ** -8, atol=1e-5) and torch.allclose(state, want_state, rtol=5e-5, atol=1e-5)
    alone, alone_state = run([0], torch.bfloat16)
    assert torch.allclose(got[:400].float(), alone.float(), rtol=2.0 ** -8, atol=1e-5) and torch.allclose(state[0], alone_state[0], rtol=5e-5, atol=1e-5)


@pytest.mark.parametrize("n,n_out", [(33, 33), (33, 1000), (100, 129), (64, 257), (300, 97), (300, 257), (700, 1)])
def test_products_whose_rows_part_a_warp(n, n_out):
    """Rows of W that end inside a warp's 32 while tokens go on for more chunks of sixteen than one: lanes without a row leave a chunk early, and the
    next read of tensor memory is for the whole warp again.  Stored, added, gated."""
    from xyntetik_runner_b200 import kernels
    k = 328
    g = torch.Generator().manual_seed(n + n_out)
    x = torch.randn(n, k, generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * n_out, k, generator=g) * k ** -0.5).to(torch.bfloat16)
    gate, up = (x.double() @ w[i * n_out:(i + 1) * n_out].double().T for i in range(2))
    # float32 sums of k exact products: (k + 2) 2^-24 of the products' sizes
    bound = x.double().abs() @ w[:n_out].double().abs().T * (k + 2) * 2.0 ** -24
    xd, one, both = x.to(DEV), kernels.pack_weight(w[:n_out].to(DEV)), kernels.pack_weight(w.to(DEV), 2)
    torch.cuda.synchronize()
    out = torch.empty(n, n_out, device=DEV)
    kernels.gemm_tc(xd, one, out, packed_rows=n_out)
    assert ((out.cpu().double() - gate).abs() <= bound).all()
    kernels.gemm_tc(xd, one, out, None, kernels.EPI_ADD, packed_rows=n_out)
    assert ((out.cpu().double() - 2 * gate).abs() <= 2 * bound + gate.abs() * 2.0 ** -22).all()
    pair = torch.empty(n, n_out, dtype=torch.bfloat16, device=DEV)
    kernels.gemm_tc(xd, both, pair, None, kernels.EPI_GATED, packed_rows=n_out)
    ref = torch.nn.functional.silu(gate) * up
    assert ((pair.double().cpu() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-5 * (gate.abs() + 1) * (up.abs() + 1)).all()
    assert int(kernels.workspace(torch.device(DEV)).status.item()) == 0


@pytest.mark.parametrize("lens", [[2048], [2049, 3], [1700, 2500]])
def test_portions_whose_gates_a_thread_holds_and_does_not(lens):
    """mLSTM's running maxima: a thread's run of eight tokens, the most that it keeps both logarithms of, and of nine and ten; against float64."""
    test_portions_of_many_chunks("mlstm", 1, 64, 64, lens)


@pytest.mark.parametrize("tiles,align", [(127, 16), (192, 16), (517, 16), (47, 64), (3073, 1), (12291, 1)])
@pytest.mark.parametrize("dtype,width", [(torch.bfloat16, 40), (torch.bfloat16, 33), (torch.float32, 300), (torch.bfloat16, 2056)])
def test_gather_of_planned_tiles(tiles, align, dtype, width):
    """Rows below and above the 3,072 (wide ones 12,288) from which four go to a block, in tiles that the plan uses, uses in part and leaves alone: a row's token, zeros in
    padding, unused tiles as they were."""
    from xyntetik_runner_b200 import kernels
    g = torch.Generator().manual_seed(tiles + width)
    rows, top, n = tiles * align, 3, 97
    group = torch.where(torch.rand(tiles, generator=g) < 0.7, torch.randint(0, 9, (tiles,), generator=g), torch.tensor(-1)).int()
    src = torch.where(torch.rand(rows, generator=g) < 0.8, torch.randint(0, n * top, (rows,), generator=g), torch.tensor(-1)).int()
    h = torch.randn(n, width, generator=g).to(dtype)
    out = torch.full((rows, width), 7.0, dtype=dtype, device=DEV)
    kernels.moe_gather(h.to(DEV), out, src.to(DEV), group.to(DEV), top, align)
    want = torch.where((src >= 0)[:, None], h[src.clamp(min=0).long() // top], torch.tensor(0.0, dtype=dtype))
    want[(group < 0).repeat_interleave(align)] = 7.0
    assert torch.equal(out.cpu(), want)
