"""Latent attention, in two forms of its projections.

With a query latent and no rotated part:

    [c_q | c_kv] = W_down h          one GEMM; both halves are RMS-normed, c_kv is what the cache holds
    q = W_uq c_q                     per head: k = W_uk c_kv, v = W_uv c_kv, score = (q . k) * scale
    out = W_o concat(heads)

With direct queries, a rotated part, a window and an output gate (the last three optional):

    [q | g | c_kv | k_r] = W_in h    one GEMM; c_kv is RMS-normed, k_r and the last part q_r of every query head are rotated
    score = (q_n . W_uk c_kv + q_r . k_r) * scale        over the window's keys; k_r is one for all heads
    out = W_o (concat(heads) * sigmoid(g))

Only c_kv (and k_r) are cached (``MLAAttentionCore``), and a layer may own no latent at all and read an earlier layer's
(``kv_sharing_target``) with its own W_uk and W_uv.

Two forms of the same attention serve a step.  *Absorbed* (decode): q is taken into the latent space by W_uk, every head
attends over the latent rows themselves, W_uv maps the result back — nothing but the latents is read.  *Expanded*
(prompt portions): keys and values of the portion's whole context are written out by two GEMMs and a multi-head kernel
runs over them — a score costs ``dim`` multiplications instead of the latent width.  A mixed step is split between the
two by the length of each request's portion, once per step (``LatentPlan``), whatever the batch looks like otherwise.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Optional

import numpy as np
import torch
import torch.nn as nn

from vllm_b200 import ops
from vllm_b200.config import get_current_vllm_config_or_none
from vllm_b200.forward_context import AttentionMetadata, get_forward_context
from vllm_b200.layers.attention import MLAAttentionCore
from vllm_b200.layers.common import RMSNorm
from vllm_b200.layers.linear import (ColumnParallelLinear, MergedColumnParallelLinear, MergedMixedLinear, MergedReplicatedLinear,
                                      RowParallelLinear)
from vllm_b200.parallel.state import get_dcp_group, get_tp_group
from vllm_b200.parallel.utils import divide

# portions of at most this many tokens attend in the latent space, one row per token: re-reading the context that often is
# still cheaper than writing its keys and values out
ABSORB_MAX_TOKENS = 16
# bytes of expanded keys and values held at a time (a longer context is done a few heads at a time), and of the latent rows that they come
# from (more contexts are done a few requests at a time)
EXPAND_BYTES = 1 << 30


@dataclass
class Contexts:
    """Contexts of some requests of a step, expanded together: one entry per request."""
    block_table: torch.Tensor
    q_start: torch.Tensor
    q_len: torch.Tensor
    seq_len: torch.Tensor      # keys of each request that some row of its portion sees
    kv_first: Optional[torch.Tensor]    # position of the first of them (None: all start at 0)
    cu_kv: torch.Tensor        # [n + 1] key rows before each request
    num_kv: int
    max_q: int
    max_kv: int


@dataclass
class LatentPlan:
    """Device-side index arrays of one step (int32 / int64), shared by all its layers of one window."""
    rows: Optional[torch.Tensor] = None        # absorbed: token rows (None: every token of the step)
    row_block_table: Optional[torch.Tensor] = None
    row_seq_lens: Optional[torch.Tensor] = None
    num_rows: int = 0
    max_row_len: int = 0
    contexts: tuple[Contexts, ...] = ()        # expanded

    @classmethod
    def of(cls, md: AttentionMetadata, device: torch.device, window: int, apart: int, most: int) -> "LatentPlan":
        plans = md.latent_plan = md.latent_plan if md.latent_plan is not None else {}
        key = window, apart, most
        if key not in plans:
            plans[key] = cls.build(md, device, *key)
        return plans[key]

    @classmethod
    def build(cls, md: AttentionMetadata, device: torch.device, window: int = 0, apart: int = 1, most: int = 1 << 62) -> "LatentPlan":
        """``apart``: key rows of a request start at multiples of it.  ``most``: key rows of requests that are expanded together (one request
        may have more)."""
        if md.host_lens is not None:
            cu, sl = md.host_lens
        else:
            cu, sl = md.query_start_loc.cpu().numpy(), md.seq_lens.cpu().numpy()
        cu, sl = np.asarray(cu, dtype=np.int64), np.asarray(sl, dtype=np.int64)
        ql = cu[1:] - cu[:-1]
        sl = sl[:len(ql)]
        short = np.nonzero((ql > 0) & (ql <= ABSORB_MAX_TOKENS))[0]
        long = np.nonzero(ql > ABSORB_MAX_TOKENS)[0]
        n_rows, n = int(ql[short].sum()), len(long)
        # token row, request and number of visible keys of every absorbed row
        req = np.repeat(short, ql[short])
        first = np.repeat(np.cumsum(ql[short]) - ql[short], ql[short])
        off = np.arange(n_rows) - first
        vis = sl[req] - ql[req] + off + 1
        kv_first = np.maximum(sl[long] - ql[long] + 1 - window, 0) if window else np.zeros(n, dtype=np.int64)
        kl = sl[long] - kv_first
        rows_kv = -(-kl // apart) * apart
        parts = [cu[req] + off, req, vis]
        groups = grouped(rows_kv, most)
        for i, j in groups:
            parts += [long[i:j], cu[long[i:j]], ql[long[i:j]], kl[i:j], kv_first[i:j], np.concatenate([[0], np.cumsum(rows_kv[i:j])])]
        packed = torch.from_numpy(np.concatenate(parts).astype(np.int32)).to(device, non_blocking=True)
        rows, req_t, vis_t, *rest = packed.split([len(p) for p in parts])
        plan = cls(num_rows=n_rows)
        if n_rows:
            plan.rows = rows.long() if n else None
            plan.row_block_table = md.block_table.index_select(0, req_t)
            plan.row_seq_lens = vis_t
            plan.max_row_len = int(vis.max())
        contexts = []
        for g, (i, j) in enumerate(groups):
            long_t, q_start, q_len, seq_len, first_t, cu_t = rest[6 * g:6 * g + 6]
            contexts.append(Contexts(md.block_table.index_select(0, long_t), q_start, q_len, seq_len, first_t if kv_first[i:j].any() else None, cu_t,
                                     int(rows_kv[i:j].sum()), int(ql[long[i:j]].max()), int(rows_kv[i:j].max())))
        plan.contexts = tuple(contexts)
        return plan


def grouped(sizes, most: int) -> list[tuple[int, int]]:
    """Ranges of neighbours whose sizes add up to at most ``most``, or that are one."""
    out, i, total = [], 0, 0
    for j, n in enumerate(int(n) for n in sizes):
        if j > i and total + n > most:
            out.append((i, j))
            i, total = j, 0
        total += n
    return out + [(i, len(sizes))] if len(sizes) else out


def step_limits():
    """The scheduler configuration of the model that is being built, if there is one."""
    vc = get_current_vllm_config_or_none()
    return None if vc is None else vc.scheduler_config


class LatentForms:
    """The two forms over a layer's attributes ``attn`` (its ``MLAAttentionCore``), ``heads``, ``dim``, ``rot``, ``v_dim``, ``kv_rank``, ``scale``,
    ``window``, ``limits`` (``step_limits()``), and ``_up()``, ``_expand(c, h0, h1)``."""
    # keys of a request start on a boundary of the prompt kernel's key tiles, zeros fill the gap: no tile holds two requests' values
    kv_apart = 1
    # softmax weights keep 16 more bits in steps that are not decode steps alone
    wide_weights = False

    def _attend(self, q: torch.Tensor, md: AttentionMetadata, cache: torch.Tensor) -> torch.Tensor:
        T = q.shape[0]
        out = torch.empty(T, self.heads, self.v_dim, dtype=q.dtype, device=q.device)
        window = self.window or None
        if md.decode_only or not ops.latent_expand_ok(q, self.dim, self.rot, self.v_dim, self.kv_rank):
            return self._absorbed(q, out, lambda q_abs, q_pe: ops.mla_attention(q_abs, q_pe, cache, md, self.scale, self.kv_rank, window))
        plan = LatentPlan.of(md, q.device, self.window, self.kv_apart, self._most_rows(q.element_size()))
        if plan.num_rows:
            def attend(q_abs, q_pe):
                return ops.mla_attention_rows(q_abs, q_pe, cache, plan.row_block_table, plan.row_seq_lens, plan.max_row_len,
                                              self.scale, window, self.wide_weights)
            if plan.rows is None:
                return self._absorbed(q, out, attend)
            part = torch.empty(plan.num_rows, self.heads, self.v_dim, dtype=q.dtype, device=q.device)
            out.index_copy_(0, plan.rows, self._absorbed(q.index_select(0, plan.rows), part, attend))
        for contexts in plan.contexts:
            self._expanded(q, out, contexts, cache, self.shares_rows and len(plan.contexts) == 1)
        return out

    def _absorbed(self, q: torch.Tensor, out: torch.Tensor, attend) -> torch.Tensor:
        w_uk, w_uv = self._up()
        q_abs = torch.bmm(q[..., :self.dim].transpose(0, 1), w_uk).transpose(0, 1)   # [T, h, R], head-major in memory
        o_lat = attend(q_abs, q[..., self.dim:] if self.rot else None)
        torch.bmm(o_lat.transpose(0, 1), w_uv.transpose(1, 2), out=out.transpose(0, 1))
        return out

    def _expanded(self, q: torch.Tensor, out: torch.Tensor, c: Contexts, cache: torch.Tensor, share: bool) -> None:
        # layers that share a cache (and see as much of it) share the gathered rows too
        gathered = get_forward_context().extra.setdefault("latent_rows", {}) if share else {}
        key = self.attn.cache_name, self.window
        rows = gathered.get(key)
        if rows is None:
            rows = gathered[key] = ops.gather_latents(cache, c.block_table, c.cu_kv, c.num_kv, c.max_kv, c.kv_first,
                                                      c.seq_len if self.kv_apart > 1 else None)
        step = self._heads_at_a_time(c.num_kv, q.element_size())
        for h0 in range(0, self.heads, step):
            h1 = min(self.heads, h0 + step)
            k, v = self._expand(rows[:, :self.kv_rank], h0, h1)
            ops.mla_prefill(q, k, v, out, c.q_start, c.q_len, c.seq_len, c.cu_kv, h0, c.max_q, self.scale,
                            rows[:, self.kv_rank:] if self.rot else None, self.window, self.wide_weights)

    def _most_rows(self, itemsize: int) -> int:
        return EXPAND_BYTES // ((self.kv_rank + self.rot) * itemsize)

    def _heads_at_a_time(self, num_kv: int, itemsize: int) -> int:
        return max(1, min(self.heads, EXPAND_BYTES // max(num_kv * (self.dim + self.v_dim) * itemsize, 1)))

    def expanded_bytes(self, requests: int, tokens: int, length: int, itemsize: int) -> int:
        """The most that a step of so many requests and tokens holds of latent rows, keys and values, its contexts ``length`` tokens long at
        most."""
        one = min(length, self.window + tokens) if self.window else length
        one = -(-one // self.kv_apart) * self.kv_apart
        rows = min(min(requests, tokens // (ABSORB_MAX_TOKENS + 1)) * one, max(self._most_rows(itemsize), one))
        per_head = rows * (self.dim + self.v_dim) * itemsize
        return rows * (self.kv_rank + self.rot) * itemsize + max(per_head, min(EXPAND_BYTES, self.heads * per_head))

    def _hold_expanded(self, q: torch.Tensor) -> None:
        """Memory-profiling run: holds for a moment what a step may take."""
        sc = self.limits
        if sc is not None and ops.latent_expand_ok(q, self.dim, self.rot, self.v_dim, self.kv_rank):
            torch.empty(self.expanded_bytes(sc.max_num_seqs, sc.max_num_batched_tokens, sc.max_model_len, q.element_size()), dtype=torch.uint8,
                        device=q.device)


class LatentAttention(LatentForms, nn.Module):
    shares_rows = True

    def __init__(self, hidden_size: int, num_heads: int, dim: int, v_dim: int, q_rank: int, kv_rank: int, scale: float, eps: float,
                 dtype=None, quant_config=None, prefix: str = "", kv_sharing_target: Optional[str] = None, rope: Optional[nn.Module] = None,
                 window: int = 0, cache_window: int = 0, gated: bool = False) -> None:
        """``q_rank`` 0: direct queries, with the parts that ``rope`` (its width is that of the rotated part), ``window`` and ``gated`` name;
        ``cache_window``: how long pages stay (``MLAAttentionCore``)."""
        super().__init__()
        if get_dcp_group().world_size > 1:
            raise NotImplementedError("decode context parallelism with this form of latent attention")
        if q_rank and (rope is not None or window or gated):
            raise NotImplementedError("a query latent beside a rotated part, a window or a gate")
        self.heads = divide(num_heads, get_tp_group().world_size)
        self.dim, self.v_dim, self.q_rank, self.kv_rank = dim, v_dim, q_rank, kv_rank
        self.rope, self.rot, self.window = rope, 0 if rope is None else rope.rotary_dim, window
        self.scale, self.eps, self.limits = float(scale), eps, step_limits()
        self.owns_latent = kv_sharing_target is None
        self.kv_norm = RMSNorm(kv_rank, eps, dtype) if self.owns_latent else None
        if q_rank:
            self.down = MergedReplicatedLinear(hidden_size, [q_rank, kv_rank] if self.owns_latent else [q_rank], False, dtype,
                                               quant_config, f"{prefix}.down")
            self.q_norm = RMSNorm(q_rank, eps, dtype)
            self.uq = ColumnParallelLinear(q_rank, num_heads * dim, False, dtype=dtype, quant_config=quant_config,
                                           prefix=f"{prefix}.uq")
        else:
            parts = [(num_heads * (dim + self.rot), True, "q")] + ([(num_heads * v_dim, True, "g")] if gated else []) + (
                [(kv_rank + self.rot, False, "kv")] if self.owns_latent else [])
            self.part = {name: i for i, (_, _, name) in enumerate(parts)}
            self.in_proj = MergedMixedLinear(hidden_size, [p[0] for p in parts], [p[1] for p in parts], False, dtype, quant_config,
                                             f"{prefix}.in_proj", align=8)
        # kept unquantised: consumed as batched absorbed matrices too, not only as a GEMM weight
        self.ukv = MergedColumnParallelLinear(kv_rank, [num_heads * dim, num_heads * v_dim], False, dtype, None, f"{prefix}.ukv")
        self.o = RowParallelLinear(num_heads * v_dim, hidden_size, False, dtype=dtype, quant_config=quant_config,
                                   prefix=f"{prefix}.o")
        self.attn = MLAAttentionCore(self.heads, kv_rank, self.rot, self.scale, prefix=f"{prefix}.attn",
                                     kv_sharing_target=kv_sharing_target, sliding_window=window or None,
                                     cache_window=cache_window or None)

    def _up(self) -> tuple[torch.Tensor, torch.Tensor]:
        """(W_uk [h, dim, R], W_uv [h, v_dim, R]): views of the stacked weight."""
        w, n = self.ukv.weight, self.heads * self.dim
        return w[:n].view(self.heads, self.dim, self.kv_rank), w[n:].view(self.heads, self.v_dim, self.kv_rank)

    def _expand(self, c: torch.Tensor, h0: int, h1: int) -> tuple[torch.Tensor, torch.Tensor]:
        """Keys and values of heads h0 .. h1 - 1 of the latent rows c."""
        w_uk, w_uv = self._up()
        return (ops.linear(c, w_uk[h0:h1].reshape(-1, self.kv_rank)).view(c.shape[0], h1 - h0, self.dim),
                ops.linear(c, w_uv[h0:h1].reshape(-1, self.kv_rank)).view(c.shape[0], h1 - h0, self.v_dim))

    def forward(self, h: torch.Tensor, positions: Optional[torch.Tensor] = None) -> torch.Tensor:
        T = h.shape[0]
        md, cache = self.attn.bound_cache()
        gate = None
        if self.q_rank:
            lat = self.down(h)
            if self.owns_latent:
                c_q, c_kv = ops.latent_norm_cache(lat, self.q_rank, self.q_norm.weight, self.kv_rank, self.kv_norm.weight, self.eps,
                                                  cache, None if md is None else md.slot_mapping)
            else:
                c_q, c_kv = ops.latent_norm_cache(lat, self.q_rank, self.q_norm.weight, 0, None, self.eps)
            q = self.uq(c_q).view(T, self.heads, self.dim)
        else:
            proj = self.in_proj(h)
            parts = self.in_proj.parts(proj)
            own = self.owns_latent
            if self.rot or own:
                ops.latent_rope_cache(proj, 0, self.heads, self.dim, self.rot, self.in_proj.offsets[self.part["kv"]] if own else 0,
                                      self.kv_rank if own else 0, self.kv_norm.weight if own else None, self.eps, positions,
                                      None if self.rope is None else self.rope.cos_sin_cache,
                                      self.rope is not None and self.rope.is_neox_style, cache if own else None,
                                      md.slot_mapping if own and md is not None else None)
            q = parts[0].view(T, self.heads, self.dim + self.rot)
            gate = parts[self.part["g"]] if "g" in self.part else None
            c_kv = parts[self.part["kv"]][:, :self.kv_rank] if own else None
        if md is None:
            self._hold_expanded(q)
            return self.o(q.new_zeros(T, self.heads * self.v_dim))
        o = self._attend(q, md, cache).view(T, self.heads * self.v_dim)
        return self.o(o if gate is None else ops.sigmoid_mul_(o, gate))
