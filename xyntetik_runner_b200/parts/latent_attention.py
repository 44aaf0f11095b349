"""Latent attention: keys and values of all heads are expanded from one small latent vector per token.

With h the mixer's input, H heads, per head D plain and R rotated query/key elements, value size V, latent size C:
    q = W_q h                   heads laid out as [D plain | R rotated]
    [c' | r'] = W_dkv h         c = RMSNorm(c') * w (the latent), r = rotate(r') (one rotated key part for all heads)
    k_h = [W_uk,h c | r],  v_h = W_uv,h c
    s_ij = (q_plain . W_uk,h c_j + rotate(q_rot) . r_j) * scale,  j <= i;  a = softmax(s);  o_h = sum_j a_ij v_hj
    y = W_o concat_h(sigmoid(W_g h)_h * o_h)
Only [c | r] is cached: one row of C + R values per token (one plane, one "kv head"), whatever H is.  Two orders of the
same sums.  Few tokens over many keys (a decode step): no key is expanded, the query is taken into the latent space,
attention runs over the cached rows with C + R columns a score and C a value, and the result is expanded by W_uv
afterwards (csrc/latent_attention.cu).  Portions of many tokens: the keys and values of all heads are expanded once, by one
dense product over the portion's cached rows, and attention runs with D + R and V columns on tcgen05 (csrc/attention_tc.cu,
``_flat_plan`` says when).  The rotation uses the first `rotary_dim` of the R elements
in the pairing the position encoding names (half-split or adjacent).

Options, all off by default:
    q_rank Q:    the queries pass a latent of their own, q = W_uq (RMSNorm(W_dq h) * w_dq);
    window w:    position i sees the positions j with 0 <= i - j < w;
    gate_each:   the gate has H V elements and multiplies the heads' outputs element by element (else one per head);
    own_rows False: the layer has no W_dkv and reads the rows that another layer caches (the schedule entry's
                 `cache_from`); `retain` is then the longest window among the readers of a layer's rows.
"""
from __future__ import annotations

from typing import Optional

import numpy as np
import torch

from .. import kernels
from ..weights.loader import TensorSpec
from .base import KVNeed, Mixer, PositionEncoding, register_mixer
from . import linear_tc
from .linear import Linear


# the tensor-core kernel for the sizes it takes (a module attribute, so that a test can compare the two kernels)
USE_MMA = True
USE_FLAT = True
counters = {"mma": 0, "simt": 0, "flat": 0}

# Portions of at least so many tokens may have their keys expanded, as far as a step's gathered and expanded rows take no more than
# so many bytes (9 KB a key at 16 heads of 128 + 128 over rows of 576: 32,768 keys).  They stay allocated beside the cached rows, and
# the other order needs none of them.
FLAT_MIN, FLAT_BYTES = 32, 1 << 29


def _rows_for(keys: int) -> int:
    """Rows of the buffers that hold `keys` expanded keys: a power of two (a buffer that grows invalidates the step graphs)."""
    return 1 << (keys - 1).bit_length()


class LatentAttention(Mixer):
    graph_safe = True

    def __init__(self, width: int, heads: int, dim: int, rot_dim: int, vdim: int, kv_rank: int, scale: float,
                 position: PositionEncoding, eps: float, prefix: str, gated: bool = True,
                 q: str = "q", dkv: str = "dkv", dkv_norm: str = "dkv.norm", uk: str = "uk", uv: str = "uv", g: str = "g", o: str = "o",
                 q_rank: Optional[int] = None, dq: str = "dq", dq_norm: str = "dq.norm", uq: str = "uq",
                 window: Optional[int] = None, retain: Optional[int] = ..., gate_each: bool = False, own_rows: bool = True):
        if kv_rank > 1024:
            raise ValueError(f"{prefix}: latent size {kv_rank}: the attention kernel takes up to 1024")
        self.width, self.H, self.D, self.R, self.V, self.C = width, heads, dim, rot_dim, vdim, kv_rank
        self.scale, self.position, self.eps, self.prefix, self.gated = float(scale), position, float(eps), prefix, gated
        self.Q, self.window, self.gate_each, self.own_rows = q_rank, window, bool(gate_each), bool(own_rows)
        # how long the cached rows are kept: this layer's window unless a reader of its rows looks further back
        self.retain = window if retain is ... else retain
        self.names = {k: prefix + v for k, v in dict(q=q, dkv=dkv, norm=dkv_norm, uk=uk, uv=uv, g=g, o=o, dq=dq, dq_norm=dq_norm,
                                                     uq=uq).items()}
        self.proj = self.out = self.w_uk = self.w_uv = self.norm_w = self.freq = self.up_q = self.q_norm_w = None
        self.w_uk_packed = self.w_uv_packed = None
        self.rot_dims = 0
        self.adjacent = False

    def kv_need(self):
        return KVNeed(1, self.C + self.R, self.retain, planes=1)

    def gate_width(self) -> int:
        return 0 if not self.gated else (self.H * self.V if self.gate_each else self.H)

    def tensors(self):
        n, H, D, R, V, C, W = self.names, self.H, self.D, self.R, self.V, self.C, self.width
        t = {n["uk"]: TensorSpec((H * D, C)), n["uv"]: TensorSpec((H * V, C)), n["o"]: TensorSpec((W, H * V))}
        if self.Q is None:
            t[n["q"]] = TensorSpec((H * (D + R), W))
        else:
            t.update({n["dq"]: TensorSpec((self.Q, W)), n["dq_norm"]: TensorSpec((self.Q,), "vector", "ones_jitter"),
                      n["uq"]: TensorSpec((H * (D + R), self.Q))})
        if self.own_rows:
            t.update({n["dkv"]: TensorSpec((C + R, W)), n["norm"]: TensorSpec((C,), "vector", "ones_jitter")})
        if self.gated:
            t[n["g"]] = TensorSpec((self.gate_width(), W))
        return t

    def bind(self, tensors, rt):
        n = self.names
        ws = [tensors.pop(n["q"] if self.Q is None else n["dq"])] + ([tensors.pop(n["dkv"])] if self.own_rows else []) \
            + ([tensors.pop(n["g"])] if self.gated else [])
        if len({w.dtype for w in ws}) > 1:
            ws = [w.to(torch.float32) for w in ws]
        # one product for the queries (or their latent), the down projection and the gates
        self.proj = Linear(torch.cat(ws, dim=0)).prepare(rt)
        del ws
        if self.Q is not None:
            self.up_q = Linear(tensors.pop(n["uq"])).prepare(rt)
            self.q_norm_w = tensors[n["dq_norm"]].to(torch.float32).contiguous()
        self.out = Linear(tensors[n["o"]]).prepare(rt)
        self.w_uk, self.w_uv = tensors[n["uk"]].contiguous(), tensors[n["uv"]].contiguous()
        # for the tensor-core products per head: W_uk,h^T ([C, D]: the query goes into the latent space) and W_uv,h ([V, C])
        self.w_uk_packed = self.w_uv_packed = None
        if (linear_tc.ENABLED and rt.act_dtype == torch.bfloat16 and self.w_uk.dtype == torch.bfloat16 and self.w_uv.dtype == torch.bfloat16
                and self.w_uk.is_cuda and self.D % 8 == 0 and self.D >= 8 and self.C % 8 == 0):
            self.w_uk_packed = kernels.pack_weight_groups(self.w_uk.view(self.H, self.D, self.C).transpose(1, 2).contiguous())
            self.w_uv_packed = kernels.pack_weight_groups(self.w_uv.view(self.H, self.V, self.C))
        self._heads_of_tiles = {}
        self.expand = None
        if (self.w_uk_packed is not None and (self.C + self.R) % 8 == 0
                and kernels.attention_tc_flat_supported(rt.act_dtype, self.D, self.R, self.V)):
            self.expand = Linear(torch.cat([self.w_uk, self.w_uv], dim=0)).prepare(rt)
        self.norm_w = tensors[n["norm"]].to(torch.float32).contiguous() if self.own_rows else None
        self.position.prepare(rt)
        rot = self.position.rotary()
        if rot is not None and rot.rotary_dim:
            if rot.mscale != 1.0 or rot.rotary_dim > self.R:
                raise ValueError(f"{self.prefix}: this mixer rotates the first rotary_dim <= rot_dim elements, cosines and sines unscaled")
            self.rot_dims = rot.rotary_dim
            self.adjacent = rot.pairing == "adjacent"
            # angles are position * frequency in float64; the frequencies come from the position encoding
            f64 = getattr(self.position, "inv_freq64_host", None)
            f64 = rot.inv_freq.double().cpu().numpy() if f64 is None else f64
            self.freq = torch.from_numpy(np.ascontiguousarray(f64, dtype=np.float64)).to(rt.device)

    def _tile_heads(self, tiles_per_head: int, device) -> torch.Tensor:
        """int32 [H * tiles_per_head]: the head whose matrix a tile of rows meets in the grouped per-head products."""
        t = self._heads_of_tiles.get(tiles_per_head)
        if t is None:
            t = torch.arange(self.H, dtype=torch.int32, device=device).repeat_interleave(tiles_per_head).contiguous()
            self._heads_of_tiles[tiles_per_head] = t
        return t

    def weight_bytes(self):
        return (self.proj.nbytes() + self.out.nbytes() + self.w_uk.numel() * self.w_uk.element_size()
                + self.w_uv.numel() * self.w_uv.element_size() + (self.up_q.nbytes() if self.up_q is not None else 0))

    def _flat_plan(self, ctx, n: int):
        """(keys to expand, 128-token tiles, token ranges left to the other order) where expanding keys pays, else None.  Both sides' times
        in microseconds, from one B200.  Over the latent rows: 50 TFLOP/s on 2 C + R columns a key and head (heads counted in sixteens), and
        0.1 a token for what stands around it (at 16 heads over 512).  Expanded: a product at 900 TFLOP/s, then a CTA per 128 tokens and head walks its keys 128 at
        a time, 1.33 each, 2.6 where some of its 128 tokens do not exist; the longest walk or all of them over 148 SMs, whichever is more.  Tokens that
        are left to the other order cost its launches again for every run of neighbours, and splits over the step's longest reach.  Measured, a layer, latent rows / expanded,
        16 heads of 128 + 64 over a latent of 512: 2,048 tokens 1,365 / 137; behind 2,000 keys 48 tokens 135 / 98, beside 16 single tokens 124 /
        152, 96 and 16 249 / 162; behind 8,000 keys 32 and 16 221 / 335, 96 and 16 501 / 343; 8 heads of 64 + 32 over 256, behind 8,000
        keys: 32 tokens 155 / 203, 64 262 / 207, 32 and 16 198 / 277."""
        H, D, R, V, C, window = self.H, self.D, self.R, self.V, self.C, self.window or 0
        if int(ctx.host["seg_len"].max()) < FLAT_MIN:
            return None
        # (plain numbers: a step's host time is not hidden, and an array operation a portion costs more than its portion)
        keys = tokens = tiles = longest = 0
        pairs = walk = walks = 0.0
        others = []
        for start, m, at in zip(ctx.host["seg_start"].tolist(), ctx.host["seg_len"].tolist(), ctx.host["seg_pos0"].tolist()):
            longest = max(longest, at + m)
            if m < FLAT_MIN:
                others.append((start, start + m))
                continue
            reach, mean, own = at + m - int(kernels.flat_first_key(at, window)), at + (m + 1) / 2.0, -(-m // 128)
            keys, tokens, tiles = keys + reach, tokens + m, tiles + own
            pairs += (min(mean, window) if window else mean) * m
            one = reach / 128.0 * (2.6 if m % 128 else 1.33)
            walk, walks = max(walk, one), walks + one * own
        if _rows_for(keys) * (H * (D + V) + C + R) * 2 > FLAT_BYTES:
            return None
        # the tokens of the other portions, neighbours together: a launch each
        rest = []
        for first, end in sorted(others):
            if rest and rest[-1][1] == first:
                rest[-1][1] = end
            else:
                rest.append([first, end])
        absorbed = pairs * -(-H // 16) * 16 * 2 * (2 * C + R) / 50e6 + 0.1 * tokens * H * C / 8192
        flat = 5.0 + keys * 2.0 * C * H * (D + V) / 900e6 + max(walk, walks * H / 148.0)
        flat += len(rest) * (45.0 + 0.005 * (min(longest, window) if window else longest))
        return None if flat >= absorbed or len(rest) > 4 else (keys, tiles, rest)

    def _absorbed(self, ctx, qt, positions, tok_seg, bt, cache_ptr, page_stride, o, gate, gate_col, window):
        """Attention over the latent rows of the tokens whose queries are qt's rows, into o's."""
        n, H, D, R, V, C = qt.shape[0], self.H, self.D, self.R, self.V, self.C
        reach = min(ctx.max_kv_len, window) if window else ctx.max_kv_len
        chunk, splits = ctx.once(("latent_splits", n, H, window), lambda: kernels.latent_attention_splits(n, H, reach))
        po = pm = None
        if splits > 1:
            mt = -(-H // 16)
            po = ctx.buf("latent_part_o", (n * mt * splits * 16 * C,), torch.float32)
            pm = ctx.buf("latent_part_ml", (n * mt * splits * 32,), torch.float32)
        args = (cache_ptr, page_stride, positions, tok_seg, bt, H, C, R, ctx.max_pages, ctx.page_size, self.scale, chunk, splits)
        if self.w_uk_packed is not None:
            # the two per-head products on tcgen05: rows of one head together (n_pad a head), one grouped product each
            bn = 16 if n <= 16 else (32 if n <= 32 else (64 if n <= 64 else 128))
            n_pad = -(-n // bn) * bn
            groups = self._tile_heads(n_pad // bn, o.device)
            qh = ctx.buf("latent_qh", (H * n_pad, D), torch.bfloat16)
            kernels.heads_gather(qt, 0, D + R, qh, n, n_pad, H, D)
            ql = ctx.buf("latent_q", (H * n_pad, C), torch.bfloat16)
            kernels.gemm_tc_grouped(qh, self.w_uk_packed, ql, groups, bn, C)
            ol = ctx.buf("latent_o", (H * n_pad, C), torch.bfloat16)
            kernels.latent_attention_mma(ql, qt, D, D + R, ol, po, pm, *args, n_pad=n_pad, window=window)
            oh = ctx.buf("latent_oh", (H * n_pad, V), torch.float32)
            kernels.gemm_tc_grouped(ol, self.w_uv_packed, oh, groups, bn, V)
            kernels.heads_scatter_gate(oh, o, gate, gate_col, n, n_pad, H, V, gate_each=self.gate_each)
        else:
            # the plain query parts, taken through W_uk^T into the latent space (bfloat16: an operand of the tensor cores)
            ql = ctx.buf("latent_q", (n, H * C), torch.bfloat16)
            kernels.head_matmul(qt, 0, D + R, self.w_uk, False, ql, n, H, D, C)
            ol = ctx.buf("latent_o", (n, H * C), torch.float32)
            kernels.latent_attention_mma(ql, qt, D, D + R, ol, po, pm, *args, window=window)
            kernels.head_matmul(ol, 0, C, self.w_uv, True, o, n, H, C, V, gate=gate, gate_col=gate_col, gate_each=self.gate_each)
        counters["mma"] += 1

    def forward(self, ctx, h, x, lay):
        n, H, D, R, V, C = h.shape[0], self.H, self.D, self.R, self.V, self.C
        if lay.writes_cache != self.own_rows:
            raise ValueError(f"{self.prefix}: a layer with rows of its own writes its cache entry, one without reads another's")
        q_cols = H * (D + R)
        first = q_cols if self.Q is None else self.Q
        down_col = first
        gate_col = first + (C + R if self.own_rows else 0)
        total = gate_col + self.gate_width()
        ld = -(-total // 8) * 8                      # rows start on 16-byte boundaries
        proj = ctx.buf("latent_proj", (n, ld), ctx.act_dtype)[:, :total]
        self.proj.forward(h, proj)
        if self.Q is None:
            qt = proj[:, :q_cols]
        else:
            # the queries' latent is normed in float32 and taken up to the heads' queries
            cq = ctx.buf("latent_cq", (n, self.Q), ctx.act_dtype)
            kernels.rmsnorm_act(proj[:, :self.Q], self.q_norm_w, cq, self.eps)
            qt = ctx.buf("latent_queries", (n, -(-q_cols // 8) * 8), ctx.act_dtype)[:, :q_cols]
            self.up_q.forward(cq, qt)
        cache_ptr, page_stride, _ = ctx.cache_layer(lay)
        bt = ctx.block_tables[lay.group]
        kernels.latent_prep(qt, proj[:, down_col:down_col + C + R] if self.own_rows else None, ctx.positions, ctx.tok_seg, bt, self.freq,
                            self.norm_w, cache_ptr if lay.writes_cache else None, page_stride, H, D, R, C, self.rot_dims,
                            ctx.max_pages, ctx.page_size, self.eps, adjacent=self.adjacent)
        o = ctx.buf("attn_out", (n, H * V), ctx.act_dtype)
        gate = proj if self.gated else None
        window = self.window or 0
        if USE_MMA and D > 0 and kernels.latent_attention_mma_supported(ctx.act_dtype, D, R, C):
            flat = ctx.once(("latent_flat", H, D, R, V, C, window), lambda: self._flat_plan(ctx, n)) if USE_FLAT and self.expand is not None else None
            if flat:
                keys, tiles, rest = flat
                room = _rows_for(keys)
                rows = ctx.buf("latent_rows", (room, C + R), torch.bfloat16)[:keys]
                kernels.flat_rows(cache_ptr, page_stride, rows, ctx.seg_len, ctx.seg_pos0, bt, ctx.n_seg, ctx.max_pages, ctx.page_size, window, FLAT_MIN)
                kv = ctx.buf("latent_kv", (room, H * (D + V)), torch.bfloat16)[:keys]
                self.expand.forward(rows[:, :C], kv)
                kernels.attention_tc_flat(qt, kv, rows[:, C:], o, ctx.seg_start, ctx.seg_len, ctx.seg_pos0, ctx.n_seg, H, D, R, V, window, self.scale,
                                          FLAT_MIN, tiles, gate=None if gate is None else gate[:, gate_col:], gate_each=self.gate_each)
                counters["flat"] += 1
                for at, end in rest:
                    self._absorbed(ctx, qt[at:end], ctx.positions[at:end], ctx.tok_seg[at:end], bt, cache_ptr, page_stride, o[at:end],
                                   None if gate is None else gate[at:end], gate_col, window)
            else:
                self._absorbed(ctx, qt, ctx.positions, ctx.tok_seg, bt, cache_ptr, page_stride, o, gate, gate_col, window)
        else:
            ql = ctx.buf("latent_q", (n, H * C), torch.float32)
            if D > 0:
                kernels.head_matmul(qt, 0, D + R, self.w_uk, False, ql, n, H, D, C)
            else:
                ql.zero_()                       # no plain query part: the scores come from the rotated parts alone
            ol = ctx.buf("latent_o", (n, H * C), torch.float32)
            kernels.latent_attention(ql, qt, D, D + R, ol, cache_ptr, page_stride, ctx.positions, ctx.tok_seg, bt, H, C, R,
                                     ctx.max_pages, ctx.page_size, self.scale, window=window)
            kernels.head_matmul(ol, 0, C, self.w_uv, True, o, n, H, C, V, gate=gate, gate_col=gate_col, gate_each=self.gate_each)
            counters["simt"] += 1
        ctx.set_pending(x, self.out.forward(o, x, accumulate=True, defer=True))


register_mixer("latent_attention", LatentAttention)
