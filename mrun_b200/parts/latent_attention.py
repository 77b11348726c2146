"""Latent attention over a paged cache of one latent row per token.

The cache row of a token is ``[c | r | 0...]``: its key/value latent c (``kv_rank`` features,
RMS-normed), the rotated key part r that all heads share (``rot_dim`` features) and zeros up to a
width the attention kernels take.  Keys and values of the heads are never made: with
K_h = U_h c and V_h = W_h c (the two up-projections), a head's score is

    q_plain . (U_h c) + q_rot . r  =  (U_h^T q_plain) . c + q_rot . r,

so the query row ``[U_h^T q_plain | q_rot | 0...]`` meets the cache row as one key of a single
key/value head, and the head's output is W_h (sum_j p_j c_j): the same cache row is the value,
and W_h runs on the weighted latent.  The framework's paged attention kernels therefore serve
this mixer unchanged (``heads`` query heads over one kv head whose K and V are the same pages);
prefill, decode and mixed steps take the paths they take for grouped-query attention.  Rows wider
than those kernels' 256 features (a latent of 512, say) go to a tensor-core kernel of their own
(``csrc/attention_latent.cu``: a block a token and 16 heads, a quarter of the value columns a warp), and
so do steps of single tokens with more than 16 heads (without a window).

A layer without a query latent (``q_rank`` = 0) has one query projection ``q`` straight from the
input; it rides in the same product as the key/value down-projection, and so do the rows of a gate
per head, whose sigmoid multiplies the heads behind W_h.  A layer without positions (``rot_dim`` = 0)
caches the latent alone.  ``window`` reaches the
attention kernels as it does for grouped-query attention.

**Steps with prompt portions** of a layer without a window whose heads' keys (plain and rotated part together:
64, 128 or 192 features) and values (64 or 128) the tcgen05 kernel takes make the keys and values after all
(``_expanded``): the scores of a portion against its own context cost (dim + rot_dim + vdim) a key and head that
way against 2 kv_rank + rot_dim, and rows wider than 128 features have no tcgen05 kernel (B200, two portions
of 760 and 1,140 tokens behind 700 and 350, 16 heads of 128 + 64, a latent of 512: the kernel for wide rows takes
688 of the mixer's 788 us; with keys and values made the mixer takes 222).  The contexts' latents are gathered
out of the pages, the rotated part they share goes beside every head's plain key, each segment's keys and
values become one large page of scratch, and the paged kernels run over those.  Only while the contexts
together are not much longer than the step (``EXPAND_ROWS`` times its rows), so that a long context is not
projected up again for every portion of it, and, with a rotated part or a query latent, only where the
scores over the latents cost more (``_worth_making``); other steps, decode steps and the 32-bit path stay with the
latent.

Per step: one product for both down-projections (their weights stacked), one kernel that norms
the two latents, rotates r and writes the cache row, the query up-projection, a per-head product
with U_h^T, one kernel that rotates the queries' rotated parts into the query rows, attention, a
per-head product with W_h, the output projection (left pending for the norm after it).
"""
from __future__ import annotations

import numpy as np
import torch

from ..cache.needs import PagedLatent
from ..config.spec import LatentAttentionSpec, TensorSpec
from ..kernels import ops
from ..kernels.attention import latent_wide_ok, paged_attention, supports_tensor_cores
from .base import POSITIONS, Runtime, register_mixer


EXPAND_ROWS = 4             # rows of scratch a step's row may bring with it where keys and values are made
EXPAND_SEGMENTS = 8         # and the most segments (each is two products of its own)


class _Pages:
    """Scratch keys and values as the attention kernels take a cache: a page a segment."""

    def __init__(self, k, v, table):
        self.k, self.v, self.block_tables, self.max_blocks = k, v, table, 1


@register_mixer("latent_attention")
class LatentAttention:
    accepts_normed_rows = True      # its first product takes ``ops.NormedRows`` as x
    can_defer_output = True         # ``forward(..., defer_output=True)`` may return ``ops.PendingLinear``

    @staticmethod
    def tensor_specs(spec: LatentAttentionSpec, prefix: str):
        s = spec
        if s.q_rank:
            query = [TensorSpec(f"{prefix}.dq", (s.q_rank, s.hidden)),
                     TensorSpec(f"{prefix}.dq.norm", (s.q_rank,), "norm"),
                     TensorSpec(f"{prefix}.uq", (s.heads * (s.dim + s.rot_dim), s.q_rank))]
        else:
            query = [TensorSpec(f"{prefix}.q", (s.heads * (s.dim + s.rot_dim), s.hidden))]
        gate = [TensorSpec(f"{prefix}.g", (s.heads, s.hidden))] if s.head_gate else []
        return query + gate + [
            TensorSpec(f"{prefix}.dkv", (s.kv_rank + s.rot_dim, s.hidden)),
            TensorSpec(f"{prefix}.dkv.norm", (s.kv_rank,), "norm"),
            TensorSpec(f"{prefix}.uk", (s.heads * s.dim, s.kv_rank)),
            TensorSpec(f"{prefix}.uv", (s.heads * s.vdim, s.kv_rank)),
            TensorSpec(f"{prefix}.o", (s.hidden, s.heads * s.vdim)),
        ]

    def __init__(self, spec: LatentAttentionSpec, tensors, runtime: Runtime):
        s = self.spec = spec
        self.runtime = runtime
        if s.window is not None and s.window < 1:
            raise ValueError("a window holds at least one position")
        # the first product: [query latent | key/value latent | shared key part], or, without a
        # query latent, [queries | key/value latent | shared key part]
        parts = [tensors["dq" if s.q_rank else "q"], tensors["dkv"]]
        self.gate_off = sum(p.shape[0] for p in parts)
        if s.head_gate:
            parts.append(tensors["g"])
        if not s.q_rank:        # zero rows at the end: the queries in the product's rows start on 16 bytes
            rows = sum(p.shape[0] for p in parts)
            parts.append(torch.zeros((-rows % 8, s.hidden), dtype=parts[0].dtype, device=parts[0].device))
        self.w_down = runtime.matrix(torch.cat(parts, dim=0))
        self.q_norm = runtime.vector_f32(tensors["dq.norm"]) if s.q_rank else None
        self.kv_norm = runtime.vector_f32(tensors["dkv.norm"])
        self.w_uq = runtime.matrix(tensors["uq"]) if s.q_rank else None
        # U_h^T per head, [heads, kv_rank, dim]: the per-head product takes weights as [out, in]
        self.w_uk_t = runtime.matrix(tensors["uk"].view(s.heads, s.dim, s.kv_rank).transpose(1, 2))
        self.w_uv = runtime.matrix(tensors["uv"].view(s.heads, s.vdim, s.kv_rank))
        self.w_o = runtime.matrix(tensors["o"])
        self.position = POSITIONS.build(s.position, {}, runtime) if s.position is not None else None
        self.rot_dims = self.position.rotary_dim if self.position is not None else 0
        self.pairing = getattr(self.position, "pairing", "half")
        if self.rot_dims > s.rot_dim:
            raise ValueError(f"{self.rot_dims} rotating features do not fit the rotated part of {s.rot_dim}")
        # the cache row's width: a size the tensor-core attention kernels are built for
        self.width = -(-(s.kv_rank + s.rot_dim) // 16) * 16
        # the tiled kernel that very wide groups fall to needs a tile list made on the host; without a
        # window the single tokens of such groups have the kernel for wide rows
        self.graph_safe = not (supports_tensor_cores(runtime.precision.act, self.width, s.heads) and s.heads > 16
                               and (s.window is not None or not latent_wide_ok(runtime.precision.act, self.width, s.kv_rank)))

        # Whether prompt steps may make the heads' keys and values from the latents (``_expanded``): key and value sizes
        # that the tcgen05 kernel takes, and, with a rotated part or a query latent, cache rows that it does not
        # take itself (on rows of 64 and 128 features it runs over the latents at the same cost).
        self.expandable = (runtime.precision.act == torch.bfloat16 and s.window is None and s.vdim in (64, 128)
                           and s.dim + s.rot_dim in (64, 128, 192) and s.dim % 8 == 0 and s.rot_dim % 8 == 0
                           and (self.width > 128 or (s.rot_dim == 0 and not s.q_rank and s.dim in (64, 128))))
        self.costly = bool(s.rot_dim or s.q_rank)

    def _scratch_rows(self, ctx) -> int:
        """Rows of the scratch pages of a step whose keys and values are made, 0 for a step that keeps the latent."""
        if not self.expandable or ctx.max_q_len == 1 or len(ctx.segments) > EXPAND_SEGMENTS:
            return 0
        if self.costly and not self._worth_making(ctx):
            return 0
        rows = 128
        while rows < ctx.max_kv_len:
            rows *= 2
        return rows if rows * len(ctx.segments) <= EXPAND_ROWS * max(128, ctx.num_tokens) else 0

    def _worth_making(self, ctx) -> bool:
        """Whether the step's scores over the latents cost more than keys and values made for them.  On B200, us a layer: the
        kernel for wide rows takes 0.45 for 1,000 (token, key) pairs of 16 heads, the absorbed products 0.03 a token; made keys
        and values cost the host two more products a segment and, once a step, two more uploads.  A layer's pass over a
        planned step, made / latents: one request of 384 tokens 164 / 153, of 768 159 / 217, four of 128 316 / 188, four of
        475 257 / 311.  A new step of a model of four such layers: one request of 512 tokens 1,576 / 1,372, of 768
        1,608 / 1,469, of 1,024 1,631 / 1,910, two of 512 1,796 / 1,518, two of 768 1,847 / 2,242, four of 384
        2,101 / 1,808, four of 500 2,124 / 2,323, eight of 250 2,583 / 1,957."""
        groups = -(-self.spec.heads // 16)
        pairs = sum(seg.q_len * (2 * seg.pos_start + seg.q_len + 1) // 2 for seg in ctx.segments)
        return groups * (0.45e-3 * pairs + 0.03 * ctx.num_tokens) >= 100 + 31 * len(ctx.segments)

    def _expanded(self, q, ctx, cache, group, rows: int) -> torch.Tensor:
        """The heads' outputs over keys and values made from the contexts' latents: [tokens, heads * vdim].  ``q``
        is rotated in place."""
        s, n = self.spec, len(ctx.segments)
        k = q.new_empty((n, s.heads, rows, s.dim + s.rot_dim))
        latents = ops.latent_rows(cache.k, group.block_tables, ctx.seg_slot[:n], ctx.seg_kv_len[:n], rows, s.kv_rank, k, s.rot_dim)
        if self.rot_dims:
            ops.latent_rotate(q, self.position.rotation(ctx), self.rot_dims, self.pairing, s.heads, s.dim, s.rot_dim)
        v = q.new_empty((n, s.heads, rows, s.vdim))
        for i, seg in enumerate(ctx.segments):
            used = -(-(seg.pos_start + seg.q_len) // 128) * 128
            c = latents[i, :used].expand(s.heads, used, s.kv_rank)
            torch.bmm(c, self.w_uk_t, out=k[i, :, :used, :s.dim])
            torch.bmm(c, self.w_uv.transpose(1, 2), out=v[i, :, :used])
        table = ctx.shared.get("segment_pages")
        if table is None:           # state slot -> its segment's page
            pages = np.full(group.block_tables.shape[0], -1, dtype=np.int32)
            pages[[seg.slot for seg in ctx.segments]] = np.arange(n, dtype=np.int32)
            table = ctx.shared["segment_pages"] = ctx.upload(pages).view(-1, 1)
        scratch = _Pages(k, v, table)
        out = q.new_empty((q.shape[0], s.heads * s.vdim))
        return paged_attention(q, q.stride(0), out, scratch, scratch, ctx, s.heads, s.softmax_scale, 0)

    def cache_need(self):
        return PagedLatent(self.width, self.spec.window)

    def activation_elements(self) -> int:
        s = self.spec
        latent = s.q_rank + s.kv_rank + s.rot_dim + s.heads * (s.dim + s.rot_dim + 2 * self.width + s.vdim)
        return latent + (EXPAND_ROWS * (s.kv_rank + s.heads * (s.dim + s.rot_dim + s.vdim)) if self.expandable else 0)

    def forward(self, x, ctx, cache, defer_output: bool = False):
        s, width = self.spec, self.width
        tokens = x.shape[0]
        group = ctx.group(cache.group_key)
        down = ops.linear(x, self.w_down)
        gate = down[:, self.gate_off:self.gate_off + s.heads] if s.head_gate else None
        down = down[:, :self.gate_off]
        rot = self.position.rotation(ctx) if self.position is not None else None
        slots = group.slot_mapping if cache.writable else None
        if s.q_rank:
            cq = down.new_empty((tokens, s.q_rank))
            ops.latent_prepare(down, self.q_norm, self.kv_norm, s.eps, rot, self.rot_dims, self.pairing, slots, cq,
                               cache.k, s.q_rank, s.kv_rank, s.rot_dim)
            q = ops.linear(cq, self.w_uq)
        else:
            nq = s.heads * (s.dim + s.rot_dim)
            q = down[:, :nq]
            ops.latent_prepare(down[:, nq:], None, self.kv_norm, s.eps, rot, self.rot_dims, self.pairing, slots, None,
                               cache.k, 0, s.kv_rank, s.rot_dim)
        rows = self._scratch_rows(ctx)
        if rows and cache.writable:
            value = self._expanded(q, ctx, cache, group, rows)
            if gate is not None:
                ops.head_gate(value, gate, s.heads)
            return ops.linear_or_pending(value, self.w_o) if defer_output else ops.linear(value, self.w_o)
        q_att = down.new_empty((tokens, s.heads, width))
        ops.linears_batched(q.unflatten(1, (s.heads, s.dim + s.rot_dim))[:, :, :s.dim], self.w_uk_t,
                            out=q_att[:, :, :s.kv_rank])
        if width > s.kv_rank:       # a rotated part, or zeros up to the row's width
            ops.latent_query(q, rot, self.rot_dims, self.pairing, q_att, s.heads, s.dim, s.rot_dim, s.kv_rank)
        mixed = down.new_empty((tokens, s.heads * width))
        paged_attention(q_att.view(tokens, s.heads * width), s.heads * width, mixed, cache, group, ctx, s.heads,
                        s.softmax_scale, s.window or 0, value_dim=s.kv_rank)
        value = down.new_empty((tokens, s.heads, s.vdim))
        ops.linears_batched(mixed.view(tokens, s.heads, width)[:, :, :s.kv_rank], self.w_uv, gate=gate, out=value)
        value = value.view(tokens, s.heads * s.vdim)
        if defer_output:
            return ops.linear_or_pending(value, self.w_o)
        return ops.linear(value, self.w_o)
