"""Attention whose keys and values are expanded from a small cached latent.

Per token the cache keeps one row: a normalised latent c (`kv_rank` elements), from which every
head's unrotated key part (U_k c) and value (U_v c) follow, and one rotated key part (`rot_dim`
elements) that all heads share.  Queries go through a latent of their own (`q_rank`), are laid
out per head as [`dim` unrotated | `rot_dim` rotated], and the score of head h for key j is
(q_plain . U_k,h c_j + q_rot . k_rot,j) * scale.  The key map is folded into the query
(q' = [U_k,h^T q_plain | q_rot]) and the value map applied after the weighted sum, so attention
runs on the cached rows themselves: one shared row of kv_rank + rot_dim key elements whose first
kv_rank elements are the values, for all heads.  An output gate sigmoid(W_g x)_h scales head h
before the output projection.  `window` > 0: a query at p sees keys p - window + 1 .. p.  `rot_dim` 0: no rotated part (the
score is the plain part's alone).  `sink`: exp(sink_h), a learned number per head, joins the denominator of head h's
softmax; it has no value.  `wide_weights`: in 16-bit modes the softmax weights keep float32 precision also where the
weighted sum runs on the tensor cores.

A mixer built with `own_latent=False` has no down-projection for keys and values: it runs as a
schedule entry with `cache_of`, reads the rows another run cached, and expands them with its own
U_k, U_v (and may look back over a window of its own).

The reference has no such mixer (its attention caches whole keys and values:
crates/model/src/llama.rs:185-257).
"""
from __future__ import annotations

import torch

from ..ops import lib as ops
from . import attention_plan
from .base import CacheNeed, Mixer, PagedKVNeed, ParamSpec
from .linear import RESIDUAL, STORE, STORE_F32, linear, linear_deferred


# Steps of single tokens cut every token's keys among CTAs while they bring fewer rows than this per SM.
SPLIT_BELOW = 4
MAX_SPLITS = 1024       # what the merge kernel folds per (token, head)

# Prompt portions write their requests' keys and values out (a product of the cached rows with U_k and U_v) and attend to
# those on the tcgen05 kernel: (128 + 64 + 128) products a (query, key) pair and head instead of the (kv_rank + 64 + kv_rank) on
# the cached rows, for 2 * 256 * kv_rank a key and head.  That pays where a key meets EXPAND_MIN_QUERIES queries of the step or
# more on average (B200, a prompt step of four layers of 16 heads, rank 512, us, cached rows -> written out: 256 tokens 975 -> 984, 400
# 1001 -> 993, 700 1331 -> 1019, 1500 2691 -> 1373, 2048 3903 -> 1684: below it is the launches that count).  The tcgen05 kernel is so
# much the quicker that kv_rank has no say: a layer's time on the GPU, 16 heads, 400 tokens, rank 64 / 128 / 256 / 512: 85 -> 64, 92 ->
# 64, 95 -> 66, 119 -> 68; 1,024 tokens after 4,096: 574 -> 172, 648 -> 173, 962 -> 177, 1346 -> 181; 4 heads, 400 tokens, rank 64 75 -> 57;
# 128 heads 216 -> 159; a window of 128 keys 71 -> 63.  What limits it is scratch: EXPAND_MAX_KEYS keys (306 MB with 16 heads of rank
# 512) and EXPAND_MAX_BYTES (16,101 keys with 128 of them).
EXPAND_MIN_QUERIES, EXPAND_MAX_KEYS, EXPAND_MAX_BYTES = 192, 32768, 1 << 30


def rows_plan(q_len, pos0, window):
    """(start, first): request r's keys from first[r] on lie at rows start[r] .. start[r + 1] - 1.  `first` is a multiple of the
    kernel's 64-key stages that no query of the step sees past."""
    import numpy as np
    q_len, pos0 = np.asarray(q_len, dtype=np.int64), np.asarray(pos0, dtype=np.int64)
    first = np.maximum(0, pos0 - window + 1) // 64 * 64 if window > 0 else np.zeros_like(pos0)
    start = np.concatenate([[0], np.cumsum(pos0 + q_len - first)])
    return start, first


def _sink_init(shape, g, device, std):
    return torch.randn(shape, generator=g, device=device, dtype=torch.float32)


class LatentAttention(Mixer):
    graph_safe = True

    def __init__(self, width, heads, dim, rot_dim, vdim, kv_rank, q_rank, eps, scale, dtype, rotary=None, window=0,
                 own_latent=True, sink=False, wide_weights=False):
        """rotary: a `RotaryEmbedding` over the rot_dim part (its rope_dim leading elements turn, in either pairing),
        or None for no rotation."""
        self.width, self.H, self.Dn, self.Rr, self.Dv = width, int(heads), int(dim), int(rot_dim), int(vdim)
        self.R, self.Rq = int(kv_rank), int(q_rank)
        self.eps, self.scale, self.dtype = float(eps), float(scale), dtype
        self.rotary, self.window, self.own_latent = rotary, int(window), bool(own_latent)
        self.has_sink, self.wide_weights = bool(sink), bool(wide_weights)
        if rotary is not None and rotary.rope_dim > self.Rr:
            raise ValueError("the rotary table must cover at most rot_dim elements")
        self.Dk = self.R + self.Rr
        for name in ("dq_weight", "dq_norm_weight", "uq_weight", "dkv_weight", "dkv_norm_weight", "uk_weight", "uv_weight",
                     "g_weight", "o_weight", "sink"):
            setattr(self, "w_" + name, None)
        self.w_in = self.w_uk_t = self.w_uv_h = None

    def param_specs(self):
        E, H = self.width, self.H
        out = {"dq.weight": ParamSpec((self.Rq, E)), "dq_norm.weight": ParamSpec((self.Rq,), kind="vector", init="ones_normal"),
               "uq.weight": ParamSpec((H * (self.Dn + self.Rr), self.Rq)),
               "uk.weight": ParamSpec((H * self.Dn, self.R)), "uv.weight": ParamSpec((H * self.Dv, self.R)),
               "g.weight": ParamSpec((H, E)), "o.weight": ParamSpec((E, H * self.Dv))}
        if self.has_sink:
            out["sink"] = ParamSpec((H,), kind="vector", init=_sink_init)
        if self.own_latent:
            out["dkv.weight"] = ParamSpec((self.R + self.Rr, E))
            out["dkv_norm.weight"] = ParamSpec((self.R,), kind="vector", init="ones_normal")
        return out

    def finalize(self):
        # one product for everything that reads the mixer's input: query latent | key/value latent | gate logits
        rows = [self.w_dq_weight] + ([self.w_dkv_weight] if self.own_latent else []) + [self.w_g_weight]
        self.w_in = torch.cat(rows, dim=0).contiguous()
        self.w_dq_weight = self.w_dkv_weight = self.w_g_weight = None
        # per head: U_k,h^T as [kv_rank, dim] (a linear map from the head's plain query part) and U_v,h as [vdim, kv_rank]
        self.w_uk_t = self.w_uk_weight.view(self.H, self.Dn, self.R).transpose(1, 2).contiguous()
        self.w_uv_h = self.w_uv_weight.view(self.H, self.Dv, self.R)     # (a view: contiguous [H, vdim, kv_rank])
        self.w_ukv = None
        if ops.attention_rows_supported(self.dtype, self.Dn, self.Rr, self.Dv, self.R):
            self.w_ukv = torch.cat([self.w_uk_weight, self.w_uv_weight], dim=0).contiguous()     # every head's key rows, then every head's value rows
            self.w_uv_h = self.w_ukv[self.H * self.Dn:].view(self.H, self.Dv, self.R)
            self.w_uv_weight = None
        self.w_uk_weight = None

    def cache_need(self):
        return CacheNeed(paged=PagedKVNeed(1, self.Dk, self.window, parts=1))

    def forward(self, x, ctx, cache, residual, accumulate=True, defer=False):
        T, H, Dn, Rr, Dv, R, Rq, Dk = ctx.n_tokens, self.H, self.Dn, self.Rr, self.Dv, self.R, self.Rq, self.Dk
        cap = ctx.token_capacity
        writes = self.own_latent
        if writes != cache.writes:
            raise ValueError("a latent mixer without a key/value projection runs as a reader of another run's cache "
                             "(and one with it as a writer)")
        # a few tokens: the product stays in partials and the next kernel sums them while it reads
        part = linear_deferred(x, self.w_in, ctx, T) if ctx.defer_residuals else None
        proj = None
        if part is None:
            proj = ctx.buf("lat_proj", (cap, self.w_in.shape[0]), torch.float32)
            linear(x, self.w_in, proj, STORE_F32, ctx, M=T)
        cq = ctx.buf("lat_cq", (cap, Rq), self.dtype)
        gate = ctx.buf("lat_gate", (cap, H), torch.float32)
        table = ctx.block_tables[cache.group]
        off_gate = Rq + (Dk if writes else 0)
        ops.latent_prep(proj, T, 0, Rq, self.w_dq_norm_weight, Rq if writes else -1, R, Rr,
                        self.w_dkv_norm_weight if writes else None, off_gate, H, ctx, table, self.rotary, cache.plane,
                        cache.page_stride, cache.page_size, cq, gate, self.eps, partials=part)
        q = ctx.buf("lat_q", (cap, H * (Dn + Rr)), self.dtype)
        linear(cq, self.w_uq_weight, q, STORE, ctx, M=T)
        plan = self._expand_plan(ctx)
        if plan is not None:
            ov = ctx.buf("lat_ov", (cap, H * Dv), self.dtype)
            self._expanded(q, ov, gate, plan, ctx, cache, table)
            return self._project(ov, ctx, residual, accumulate, defer)
        qf = ctx.buf("lat_qf", (cap, H * Dk), self.dtype)
        few = T <= ops.head_linear_max_tokens()      # every head's product in one launch: a few tokens on the CUDA cores ...
        if few or ops.head_linear_mma_supported(q, Dn + Rr, self.w_uk_t, qf, Dk):     # ... many on the tensor cores
            ops.head_linear(q, Dn + Rr, self.w_uk_t, qf, Dk, T)
        else:
            for h in range(H):
                linear(q[:, h * (Dn + Rr):h * (Dn + Rr) + Dn], self.w_uk_t[h], qf[:, h * Dk:h * Dk + R], STORE, ctx, M=T)
        ops.latent_q_rope(q, qf, T, ctx.positions, self.rotary, H, Dn, Rr, R, ctx.err)
        o = ctx.buf("lat_o", (cap, H * R), self.dtype)
        single = ctx.max_q_len == 1
        part, slots = None, 0
        if single and T * -(-H // 8) < SPLIT_BELOW * attention_plan.sm_count():
            # few single tokens: their key ranges are cut among CTAs.  The number of slots depends on the
            # batch's sizes alone while a CUDA graph is captured or replayed (the longest context the table holds).
            split = ops.attention_latent_split()
            longest = table.shape[1] * cache.page_size if ctx.fixed_shapes else ctx.max_kv_len
            if self.window > 0:
                longest = min(longest, self.window + split)
            slots = longest // split + 2
            if slots <= MAX_SPLITS:
                part = ctx.buf("lat_part", (T * H * slots * (R + 2),), torch.float32)
            else:
                slots = 0
        ops.attention_latent(qf, o, gate, T, ctx, table, cache.plane, cache.page_stride, cache.page_size, H, Dk, R,
                             self.scale, self.window, single_tokens=single, part=part, split_slots=slots, sink=self.w_sink, wide_weights=self.wide_weights)
        ov = ctx.buf("lat_ov", (cap, H * Dv), self.dtype)
        if few or ops.head_linear_mma_supported(o, R, self.w_uv_h, ov, Dv):
            ops.head_linear(o, R, self.w_uv_h, ov, Dv, T)
        else:
            for h in range(H):
                linear(o[:, h * R:(h + 1) * R], self.w_uv_h[h], ov[:, h * Dv:(h + 1) * Dv], STORE, ctx, M=T)
        return self._project(ov, ctx, residual, accumulate, defer)

    def _project(self, ov, ctx, residual, accumulate, defer):
        if defer and not accumulate:
            part = linear_deferred(ov, self.w_o_weight, ctx, ctx.n_tokens)
            if part is not None:
                return part
        linear(ov, self.w_o_weight, residual, RESIDUAL if accumulate else STORE_F32, ctx, M=ctx.n_tokens)
        return None

    def _row_elements(self):
        """Scratch of one key that is written out."""
        return self.Dk + self.H * (self.Dn + self.Dv)

    def _expand_plan(self, ctx):
        """Where this step's keys and values are written out: (keys, keys at most, start, first, key_row, work, items), the same for every
        layer with this window and size; None where attention runs on the cached rows."""
        if self.w_ukv is None or ctx.max_q_len < EXPAND_MIN_QUERIES or ctx.fixed_shapes:
            return None
        max_keys = min(EXPAND_MAX_KEYS, EXPAND_MAX_BYTES // (2 * self._row_elements()))
        key = ("latent rows", self.window, max_keys)
        if key in ctx.step_cache:
            return ctx.step_cache[key]
        import numpy as np
        start, first = rows_plan(ctx.h_q_len, ctx.h_pos0, self.window)
        n_keys = int(start[-1])
        seen = sum(n * min(p + (n + 1) // 2, self.window if self.window > 0 else p + n) for p, n in zip(ctx.h_pos0, ctx.h_q_len))
        plan = None
        if n_keys <= max_keys and seen >= EXPAND_MIN_QUERIES * n_keys:
            R = len(ctx.h_q_len)
            items = attention_plan.whole_items(ctx.h_q_len, ctx.h_pos0, self.window, 256)
            host = np.concatenate([start, first, start[:-1] - first, items.reshape(-1)]).astype(np.int32)
            ring, dev = ctx.plan_store.buffers(key, host.size, captured=False)
            ring.next().numpy()[:host.size] = host
            dev[:host.size].copy_(ring.bufs[ring.i][:host.size], non_blocking=True)
            ring.sent()
            ctx.h2d_bytes += host.size * 4
            plan = (n_keys, max_keys, dev[:R + 1], dev[R + 1:2 * R + 1], dev[2 * R + 1:3 * R + 1], dev[3 * R + 1:host.size], items.shape[0])
        ctx.step_cache[key] = plan
        return plan

    def _expanded(self, q, ov, gate, plan, ctx, cache, table):
        n_keys, max_keys, start, first, key_row, work, n_work = plan
        T, H, R = ctx.n_tokens, self.H, self.R
        # (the keys grow with every portion of a prompt, and no captured step comes here)
        rows = ctx.scratch.get("lat_rows", (n_keys, self.Dk), self.dtype, limit=max_keys * self.Dk, captured=False)
        kv = ctx.scratch.get("lat_kv", (n_keys, H * (self.Dn + self.Dv)), self.dtype, limit=max_keys * H * (self.Dn + self.Dv), captured=False)
        ops.latent_gather(cache.plane, cache.page_stride, cache.page_size, table, start, first, ctx.pos0, self.window, n_keys, self.Dk, rows, ctx.err)
        linear(rows[:, :R], self.w_ukv, kv, STORE, ctx, M=n_keys)
        ops.latent_q_rope_own(q, T, ctx.positions, self.rotary, H, self.Dn, self.Rr, ctx.err)
        ops.attention_rows(q, kv, rows, R, n_keys, ov, key_row, ctx.q_start, ctx.pos0, work, n_work, H, self.scale, self.window, ctx.err,
                           gate=gate, sink=self.w_sink, wide_weights=self.wide_weights)
