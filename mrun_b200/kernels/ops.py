"""Typed wrappers over the kernel library: they check dtypes, layouts and devices, and pass raw
pointers with the current CUDA stream.  Every function needs CUDA tensors; none has a CPU path.
"""
from __future__ import annotations

import ctypes
import os
from typing import Optional

import torch

from . import lib as _lib
from .lib import KernelError

F32, BF16 = 0, 1
_c_int, _c_long, _c_float = ctypes.c_int, ctypes.c_long, ctypes.c_float


def dtype_code(dtype: torch.dtype) -> int:
    if dtype == torch.float32:
        return F32
    if dtype == torch.bfloat16:
        return BF16
    raise KernelError(f"dtype {dtype} has no kernel (float32 and bfloat16 do)")


def _queue() -> int:
    """The current stream of the current device.  Asked for by its raw handle: a Stream object took 29 % of an
    uncaptured step's host time (a mixer's decode step of five kernels on B200: 119 us a pass, 96 without)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _address(t: Optional[torch.Tensor]) -> Optional[int]:
    """For :meth:`Library.call` only, which knows the parameters' types: ctypes passes a plain number as a 32-bit int wherever
    they are not declared."""
    return None if t is None else t.data_ptr()


def _stream() -> ctypes.c_void_p:
    """The current stream for a function of any library, its parameters' types declared or not."""
    return ctypes.c_void_p(_queue())


def _ptr(t: Optional[torch.Tensor]) -> ctypes.c_void_p:
    """A tensor's address for a function of any library, its parameters' types declared or not."""
    return ctypes.c_void_p(_address(t))


def _check(t: torch.Tensor, name: str, dtype: Optional[torch.dtype] = None, dense: bool = True) -> None:
    if not t.is_cuda:
        raise KernelError(f"{name} is on {t.device}; the kernels run on CUDA only")
    if dtype is not None and t.dtype != dtype:
        raise KernelError(f"{name} has dtype {t.dtype}, expected {dtype}")
    if dense and not t.is_contiguous():
        raise KernelError(f"{name} is not contiguous")


def embed(table: torch.Tensor, ids: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """out[t] = float(table[ids[t]]); out is float32 [tokens, hidden]."""
    _check(table, "table"); _check(ids, "ids", torch.int32); _check(out, "out", torch.float32)
    vocab, hidden = table.shape
    tokens = ids.numel()
    if out.shape != (tokens, hidden):
        raise KernelError(f"embed: out is {tuple(out.shape)}, expected {(tokens, hidden)}")
    _lib.core().call("mrun_embed", _address(table), dtype_code(table.dtype), _address(ids), _address(out),
                     tokens, hidden, vocab, _queue())
    return out


def add_rmsnorm(resid: torch.Tensor, delta: Optional[torch.Tensor], weight: torch.Tensor, eps: float,
                out: torch.Tensor, rows: Optional[torch.Tensor] = None, scaled=None) -> torch.Tensor:
    """resid (+= delta, += share * extra row by row for ``scaled`` = (extra, share)) then out =
    rmsnorm(resid) * weight; with ``rows`` only those rows are normed and resid is left as it is.
    ``delta`` is 32-bit or of ``out``'s dtype, ``extra`` of ``out``'s, ``share`` float32 [rows of resid]."""
    _check(resid, "resid", torch.float32); _check(weight, "weight", torch.float32); _check(out, "out")
    hidden = resid.shape[-1]
    n_rows = resid.shape[0] if rows is None else rows.numel()
    if delta is not None:
        _check(delta, "delta")
        if delta.shape != resid.shape or delta.dtype not in (torch.float32, out.dtype):
            raise KernelError(f"add_rmsnorm: delta {tuple(delta.shape)} {delta.dtype} vs resid {tuple(resid.shape)}, out {out.dtype}")
    extra = share = None
    if scaled is not None:
        extra, share = scaled
        _check(extra, "extra", out.dtype); _check(share, "share", torch.float32)
        if extra.shape != resid.shape or share.numel() != resid.shape[0]:
            raise KernelError(f"add_rmsnorm: extra {tuple(extra.shape)}, share {tuple(share.shape)} vs resid {tuple(resid.shape)}")
    if rows is not None:
        _check(rows, "rows", torch.int32)
    if weight.numel() != hidden or out.shape != (n_rows, hidden):
        raise KernelError(f"add_rmsnorm: weight {tuple(weight.shape)}, out {tuple(out.shape)}, "
                          f"expected hidden {hidden}, rows {n_rows}")
    _lib.core().call("mrun_add_rmsnorm", _address(resid), _address(delta), dtype_code(delta.dtype if delta is not None else out.dtype),
                     _address(weight), eps, _address(out), dtype_code(out.dtype), _address(rows), n_rows, hidden,
                     _address(extra), _address(share), _queue())
    return out


def add_scaled_rows(y: torch.Tensor, x: torch.Tensor, share: torch.Tensor) -> torch.Tensor:
    """y[t] += share[t] * x[t] in place, the sum in 32-bit; ``x`` of y's dtype, or bfloat16 with a 32-bit y."""
    _check(y, "y"); _check(x, "x"); _check(share, "share", torch.float32)
    if y.dim() != 2 or x.shape != y.shape or share.numel() != y.shape[0]:
        raise KernelError(f"add_scaled_rows: y {tuple(y.shape)}, x {tuple(x.shape)}, share {tuple(share.shape)}")
    _lib.core().call("mrun_add_scaled_rows", _address(y), dtype_code(y.dtype), _address(x), dtype_code(x.dtype), _address(share),
                     y.shape[0], y.shape[1], _queue())
    return y


def add_layernorm(resid: torch.Tensor, delta: Optional[torch.Tensor], weight: torch.Tensor, eps: float,
                  out: torch.Tensor, rows: Optional[torch.Tensor] = None,
                  bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """resid (+= delta) then out = (resid - mean) * rsqrt(variance + eps) * weight (+ bias), the
    variance the mean of the squared deviations; with ``rows`` only those rows are normed and resid is left as
    it is.  ``delta`` is 32-bit or of ``out``'s dtype."""
    _check(resid, "resid", torch.float32); _check(weight, "weight", torch.float32); _check(out, "out")
    hidden = resid.shape[-1]
    n_rows = resid.shape[0] if rows is None else rows.numel()
    if delta is not None:
        _check(delta, "delta")
        if delta.shape != resid.shape or delta.dtype not in (torch.float32, out.dtype):
            raise KernelError(f"add_layernorm: delta {tuple(delta.shape)} {delta.dtype} vs resid {tuple(resid.shape)}, "
                              f"out {out.dtype}")
    if bias is not None:
        _check(bias, "bias", torch.float32)
        if bias.numel() != hidden:
            raise KernelError(f"add_layernorm: bias has {bias.numel()} entries, the width is {hidden}")
    if rows is not None:
        _check(rows, "rows", torch.int32)
    if weight.numel() != hidden or out.shape != (n_rows, hidden):
        raise KernelError(f"add_layernorm: weight {tuple(weight.shape)}, out {tuple(out.shape)}, "
                          f"expected hidden {hidden}, rows {n_rows}")
    _lib.core().call("mrun_add_layernorm", _address(resid), _address(delta), dtype_code(delta.dtype if delta is not None else out.dtype),
                     _address(weight), _address(bias), eps, _address(out), dtype_code(out.dtype), _address(rows), n_rows,
                     hidden, _queue())
    return out


def post_layernorm_add(stream: torch.Tensor, pending, next_weight: Optional[torch.Tensor] = None,
                       next_bias: Optional[torch.Tensor] = None, next_eps: float = 0.0,
                       out: Optional[torch.Tensor] = None, rows: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
    """stream += layer norm of a :class:`PendingPostLayerNorm`'s branch (None: nothing is added), in
    place and in 32-bit; then ``out`` gets the new rows in its dtype or, with ``next_weight``, their
    layer norm (``out`` None: nothing).  With ``rows`` only those rows are computed and the stream
    is left as it is."""
    _check(stream, "stream", torch.float32)
    hidden = stream.shape[1]
    n_rows = stream.shape[0] if rows is None else rows.numel()
    branch = weight = bias = None
    eps = 0.0
    if pending is not None:
        branch, weight, bias, eps = pending.branch, pending.weight, pending.bias, pending.eps
        _check(branch, "branch", torch.float32)
        if branch.shape != stream.shape:
            raise KernelError(f"post_layernorm_add: stream {tuple(stream.shape)}, branch {tuple(branch.shape)}")
    for name, v in (("weight", weight), ("bias", bias), ("next_weight", next_weight), ("next_bias", next_bias)):
        if v is not None:
            _check(v, name, torch.float32)
            if v.numel() != hidden:
                raise KernelError(f"post_layernorm_add: {name} has {v.numel()} entries, the width is {hidden}")
    code = F32
    if out is not None:
        _check(out, "out")
        code = dtype_code(out.dtype)
        if out.shape != (n_rows, hidden):
            raise KernelError(f"post_layernorm_add: out {tuple(out.shape)}, expected {(n_rows, hidden)}")
    if rows is not None:
        _check(rows, "rows", torch.int32)
    _lib.core().call("mrun_post_layernorm_add", _address(stream), _address(branch), _address(weight), _address(bias), eps,
                     _address(next_weight), _address(next_bias), next_eps, _address(out), code, _address(rows),
                     n_rows, hidden, _queue())
    return out


def pair_norm_mean(a: torch.Tensor, b: torch.Tensor, weight_a: torch.Tensor, weight_b: torch.Tensor, eps: float,
                   share: float = 0.5) -> torch.Tensor:
    """float32 ``share * (rmsnorm(a) * weight_a + rmsnorm(b) * weight_b)`` row by row (eps inside the
    root); ``a`` and ``b`` are float32 [rows, hidden]."""
    for name, t in (("a", a), ("b", b), ("weight_a", weight_a), ("weight_b", weight_b)):
        _check(t, name, torch.float32)
    rows, hidden = a.shape
    if b.shape != a.shape or weight_a.numel() != hidden or weight_b.numel() != hidden:
        raise KernelError(f"pair_norm_mean: a {tuple(a.shape)}, b {tuple(b.shape)}, weights {weight_a.numel()} / {weight_b.numel()}")
    out = torch.empty_like(a)
    _lib.core().call("mrun_pair_norm_mean", _address(a), _address(b), _address(weight_a), _address(weight_b), eps,
                     share, _address(out), rows, hidden, _queue())
    return out


def pair_norm_add_layernorm(resid: torch.Tensor, pending, weight: torch.Tensor, eps: float, out: torch.Tensor,
                            rows: Optional[torch.Tensor] = None) -> torch.Tensor:
    """resid += share * (rmsnorm(a) * weight_a + rmsnorm(b) * weight_b) for a :class:`PendingPairNorm`,
    then out = layer norm of resid with ``weight``; with ``rows`` only those rows are worked on and
    resid is left as it is."""
    _check(resid, "resid", torch.float32); _check(weight, "weight", torch.float32); _check(out, "out")
    for name, t in (("a", pending.a), ("b", pending.b), ("weight_a", pending.weight_a), ("weight_b", pending.weight_b)):
        _check(t, name, torch.float32)
    hidden = resid.shape[-1]
    n_rows = resid.shape[0] if rows is None else rows.numel()
    if rows is not None:
        _check(rows, "rows", torch.int32)
    if pending.a.shape != resid.shape or pending.b.shape != resid.shape or weight.numel() != hidden \
            or pending.weight_a.numel() != hidden or pending.weight_b.numel() != hidden or out.shape != (n_rows, hidden):
        raise KernelError(f"pair_norm_add_layernorm: resid {tuple(resid.shape)}, a {tuple(pending.a.shape)}, "
                          f"b {tuple(pending.b.shape)}, out {tuple(out.shape)}")
    _lib.core().call("mrun_pair_norm_add_layernorm", _address(resid), _address(pending.a), _address(pending.b), _address(pending.weight_a),
                     _address(pending.weight_b), pending.eps, pending.share, _address(weight), eps,
                     _address(out), dtype_code(out.dtype), _address(rows), n_rows, hidden, _queue())
    return out


def rotary_table(positions: torch.Tensor, inv_freq: torch.Tensor, out: torch.Tensor,
                 magnitude: float = 1.0) -> torch.Tensor:
    """out[t, j] = magnitude * (cos, sin)(positions[t] * inv_freq[j]); inv_freq is float64."""
    _check(positions, "positions", torch.int32); _check(inv_freq, "inv_freq", torch.float64)
    _check(out, "out", torch.float32)
    tokens, half = positions.numel(), inv_freq.numel()
    if out.shape != (tokens, half, 2):
        raise KernelError(f"rotary_table: out is {tuple(out.shape)}, expected {(tokens, half, 2)}")
    _lib.core().call("mrun_rotary_table", _address(positions), _address(inv_freq), _address(out), tokens,
                     half, magnitude, _queue())
    return out


def qk_norm_rope_cache(qkv: torch.Tensor, heads: int, kv_heads: int, head_dim: int,
                       q_weight: Optional[torch.Tensor], k_weight: Optional[torch.Tensor], eps: float,
                       rot: Optional[torch.Tensor], rotary_dim: int, slots: Optional[torch.Tensor],
                       k_cache: Optional[torch.Tensor], v_cache: Optional[torch.Tensor],
                       page_size: int) -> None:
    """In place on the q part of ``qkv``; k and v go into the pages that ``slots`` names."""
    _check(qkv, "qkv")
    tokens = qkv.shape[0]
    if qkv.shape[1] != (heads + 2 * kv_heads) * head_dim:
        raise KernelError(f"qk_norm_rope_cache: qkv is {tuple(qkv.shape)}, expected width "
                          f"{(heads + 2 * kv_heads) * head_dim}")
    for name, w in (("q_weight", q_weight), ("k_weight", k_weight)):
        if w is not None:
            _check(w, name, torch.float32)
            if w.numel() != head_dim:
                raise KernelError(f"qk_norm_rope_cache: {name} has {w.numel()} elements, head_dim is {head_dim}")
    if rot is not None:
        _check(rot, "rot", torch.float32)
        if rot.shape != (tokens, rotary_dim // 2, 2):
            raise KernelError(f"qk_norm_rope_cache: rot is {tuple(rot.shape)}, expected "
                              f"{(tokens, rotary_dim // 2, 2)}")
    if slots is not None:
        _check(slots, "slots", torch.int32)
        if slots.numel() != tokens:
            raise KernelError("qk_norm_rope_cache: one slot per token is needed")
        for name, c in (("k_cache", k_cache), ("v_cache", v_cache)):
            _check(c, name, qkv.dtype)
            if c.dim() != 4 or c.shape[1:] != (kv_heads, page_size, head_dim):
                raise KernelError(f"qk_norm_rope_cache: {name} is {tuple(c.shape)}, expected "
                                  f"[pages, {kv_heads}, {page_size}, {head_dim}]")
    _lib.core().call("mrun_qk_norm_rope_cache", _address(qkv), dtype_code(qkv.dtype), _address(q_weight),
                     _address(k_weight), eps, _address(rot), rotary_dim if rot is not None else 0,
                     _address(slots), _address(k_cache), _address(v_cache), tokens, heads,
                     kv_heads, head_dim, page_size, _queue())


def proj_norm_rope_cache(x: torch.Tensor, q_off: int, k_off: int, v_off: int, heads: int, kv_heads: int, dim: int,
                         vdim: int, q_weight: Optional[torch.Tensor], k_weight: Optional[torch.Tensor], eps: float,
                         rot: Optional[torch.Tensor], rotary_dim: int, pairing: str, slots: Optional[torch.Tensor],
                         k_cache: Optional[torch.Tensor], v_cache: Optional[torch.Tensor], page_size: int) -> None:
    """RMS norm of q and of k over the whole projection (all heads of a token together, weights of
    that size), rotation of the first ``rotary_dim`` features of every head, k and v into the
    pages ``slots`` names (key pages [pages, kv_heads, page, dim], value pages [.., vdim]).  ``x``:
    rows whose q, k and v heads start at columns ``q_off``, ``k_off``, ``v_off``; q is worked on in
    place.  ``k_off`` < 0: the rows have no keys and values."""
    ld = _strided_rows(x, "x")
    tokens = x.shape[0]
    for name, w, n in (("q_weight", q_weight, heads * dim), ("k_weight", k_weight, kv_heads * dim)):
        if w is not None:
            _check(w, name, torch.float32)
            if w.numel() != n:
                raise KernelError(f"proj_norm_rope_cache: {name} has {w.numel()} elements, the projection has {n}")
    if rot is not None:
        _check(rot, "rot", torch.float32)
        if rot.shape != (tokens, rotary_dim // 2, 2):
            raise KernelError(f"proj_norm_rope_cache: rot is {tuple(rot.shape)}, expected {(tokens, rotary_dim // 2, 2)}")
    if k_off >= 0 and slots is not None:
        _check(slots, "slots", torch.int32)
        for name, c, n in (("k_cache", k_cache, dim), ("v_cache", v_cache, vdim)):
            _check(c, name, x.dtype)
            if c.dim() != 4 or c.shape[1:] != (kv_heads, page_size, n):
                raise KernelError(f"proj_norm_rope_cache: {name} is {tuple(c.shape)}, expected "
                                  f"[pages, {kv_heads}, {page_size}, {n}]")
    width = x.shape[1]
    if q_off + heads * dim > width or (k_off >= 0 and (k_off + kv_heads * dim > width or v_off + kv_heads * vdim > width)):
        raise KernelError("proj_norm_rope_cache: the heads do not fit the rows")
    _lib.core().call("mrun_proj_norm_rope_cache", _address(x), ld, q_off, k_off, v_off,
                     dtype_code(x.dtype), _address(q_weight), _address(k_weight), eps, _address(rot),
                     rotary_dim if rot is not None else 0, PAIRINGS[pairing],
                     _address(slots if k_off >= 0 else None), _address(k_cache), _address(v_cache), tokens, heads,
                     kv_heads, dim, vdim, page_size, _queue())


def head_norm_rope_cache(x: torch.Tensor, q_off: int, k_off: int, v_off: int, heads: int, kv_heads: int, dim: int,
                         vdim: int, q_weight: Optional[torch.Tensor], k_weight: Optional[torch.Tensor], eps: float,
                         rot: Optional[torch.Tensor], rotary_dim: int, pairing: str, slots: Optional[torch.Tensor],
                         k_cache: Optional[torch.Tensor], v_cache: Optional[torch.Tensor], page_size: int,
                         bias: Optional[torch.Tensor] = None, keep: Optional[torch.Tensor] = None, blend=None) -> None:
    """RMS norm of every q and k head over its own ``dim`` features (weights of ``dim`` entries that
    the heads share; None: no norm), rotation of the first ``rotary_dim`` features of every head,
    k and v into the pages ``slots`` names (key pages [pages, kv_heads, page, dim], value pages
    [.., vdim]).  ``x``: rows whose q, k and v heads start at columns ``q_off``, ``k_off``,
    ``v_off``; q is worked on in place.  ``v_off`` < 0: the values are the keys as projected,
    before norm and rotation.  ``bias`` (float32, [q | k | v] features) is added first.  ``keep`` (rows of
    kv_heads * vdim features of x's dtype, may be strided) gets the values; ``blend`` = (rows, share): the
    values then become (1 - share) * v + share * rows."""
    ld = _strided_rows(x, "x")
    tokens = x.shape[0]
    for name, w in (("q_weight", q_weight), ("k_weight", k_weight)):
        if w is not None:
            _check(w, name, torch.float32)
            if w.numel() != dim:
                raise KernelError(f"head_norm_rope_cache: {name} has {w.numel()} elements, a head has {dim}")
    if rot is not None:
        _check(rot, "rot", torch.float32)
        if rot.shape != (tokens, rotary_dim // 2, 2):
            raise KernelError(f"head_norm_rope_cache: rot is {tuple(rot.shape)}, expected {(tokens, rotary_dim // 2, 2)}")
    if slots is not None:
        _check(slots, "slots", torch.int32)
        for name, c, n in (("k_cache", k_cache, dim), ("v_cache", v_cache, vdim)):
            _check(c, name, x.dtype)
            if c.dim() != 4 or c.shape[1:] != (kv_heads, page_size, n):
                raise KernelError(f"head_norm_rope_cache: {name} is {tuple(c.shape)}, expected "
                                  f"[pages, {kv_heads}, {page_size}, {n}]")
    if bias is not None:
        _check(bias, "bias", torch.float32)
        if bias.numel() != (heads + kv_heads) * dim + (kv_heads * vdim if v_off >= 0 else 0):
            raise KernelError(f"head_norm_rope_cache: bias has {bias.numel()} entries")
    first, share = blend if blend is not None else (None, 0.0)
    strides = []
    for name, t in (("keep", keep), ("blend", first)):
        strides.append(_strided_rows(t, name) if t is not None else 0)
        if t is not None and (t.shape != (tokens, kv_heads * vdim) or t.dtype != x.dtype):
            raise KernelError(f"head_norm_rope_cache: {name} is {tuple(t.shape)} {t.dtype}, expected {(tokens, kv_heads * vdim)} {x.dtype}")
    width = x.shape[1]
    if q_off + heads * dim > width or k_off + kv_heads * dim > width or (v_off >= 0 and v_off + kv_heads * vdim > width):
        raise KernelError("head_norm_rope_cache: the heads do not fit the rows")
    _lib.core().call("mrun_head_norm_rope_cache", _address(x), ld, q_off, k_off, v_off,
                     dtype_code(x.dtype), _address(q_weight), _address(k_weight), eps, _address(rot),
                     rotary_dim if rot is not None else 0, PAIRINGS[pairing], _address(slots), _address(k_cache),
                     _address(v_cache), tokens, heads, kv_heads, dim, vdim,
                     page_size, _address(bias), _address(first), strides[1], share, _address(keep),
                     strides[0], _queue())


def check_sink(sink: Optional[torch.Tensor], heads: int) -> None:
    if sink is not None:
        _check(sink, "sink", torch.float32)
        if sink.numel() != heads:
            raise KernelError(f"attention: sink has {sink.numel()} scores for {heads} query heads")


def paged_attention_generic(q: torch.Tensor, q_stride: int, out: torch.Tensor, k_cache: torch.Tensor,
                            v_cache: torch.Tensor, block_tables: torch.Tensor, token_slot: torch.Tensor,
                            positions: torch.Tensor, heads: int, scale: float, window: int = 0, sink: Optional[torch.Tensor] = None,
                            gate: Optional[torch.Tensor] = None, form=None) -> torch.Tensor:
    """Attention of every token over its request's pages, 32-bit arithmetic on CUDA cores.

    ``q`` may be a view into a wider buffer: row t starts ``q_stride`` elements after row t-1.
    ``block_tables`` has one row per state slot; ``token_slot[t]`` names the row of token t.
    The value pages may have another feature size than the key pages.  ``sink`` (float32, a score a
    query head): one more term without a value in the softmax's denominator.  ``gate``: [tokens, heads] in q's dtype
    (rows may be strided), whose sigmoid multiplies each head's output.  ``form``: a score form
    (:class:`mrun_b200.kernels.attention.ScoreForm`), whose output rows may be strided.
    """
    _check(q, "q", dense=False); _check(out, "out", q.dtype, dense=form is None)
    _check(k_cache, "k_cache", q.dtype); _check(v_cache, "v_cache", q.dtype)
    _check(block_tables, "block_tables", torch.int32); _check(token_slot, "token_slot", torch.int32)
    _check(positions, "positions", torch.int32)
    pages, kv_heads, page_size, head_dim = k_cache.shape
    tokens = positions.numel()
    if v_cache.dim() != 4 or v_cache.shape[:3] != k_cache.shape[:3]:
        raise KernelError("paged_attention: k and v caches differ in pages, heads or page size")
    value_dim = v_cache.shape[3]
    if out.shape != (tokens, heads * value_dim) or token_slot.numel() != tokens:
        raise KernelError(f"paged_attention: out {tuple(out.shape)} / token_slot {token_slot.numel()} "
                          f"do not match {tokens} tokens of {heads}x{value_dim}")
    if block_tables.dim() != 2:
        raise KernelError("paged_attention: block_tables must be [slots, max_blocks]")
    check_sink(sink, heads)
    gate_stride = 0
    if gate is not None:
        gate_stride = _strided_rows(gate, "gate")
        if gate.shape != (tokens, heads) or gate.dtype != q.dtype:
            raise KernelError(f"paged_attention: gate is {tuple(gate.shape)} {gate.dtype}, expected {(tokens, heads)} {q.dtype}")
    _lib.core().call("mrun_paged_attention_generic", _address(q), q_stride, _address(out), _address(k_cache),
                     _address(v_cache), dtype_code(q.dtype), _address(block_tables), block_tables.shape[1],
                     _address(token_slot), _address(positions), tokens, heads, kv_heads,
                     head_dim, value_dim, page_size, pages * kv_heads * page_size,
                     scale, window, _address(sink), _address(gate), gate_stride,
                     ctypes.byref(form) if form is not None else _address(None), _queue())
    return out


def paged_attention_f32(q: torch.Tensor, q_stride: int, out: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor,
                        block_tables: torch.Tensor, token_slot: torch.Tensor, positions: torch.Tensor, first: Optional[torch.Tensor],
                        count: Optional[torch.Tensor], tiles: int, tile_tokens: int, heads: int, scale: float,
                        window: int = 0) -> torch.Tensor:
    """32-bit attention over the pages for heads of 64 and 128 features (keys and values alike) in tiles of
    at most ``tile_tokens`` consecutive tokens of a request: tile i holds ``count[i]`` tokens from row
    ``first[i]`` on; None: every token a tile.  Rows that no tile names are left as they are."""
    _check(q, "q", torch.float32, dense=False); _check(out, "out", torch.float32)
    _check(k_cache, "k_cache", torch.float32); _check(v_cache, "v_cache", torch.float32)
    _check(block_tables, "block_tables", torch.int32); _check(token_slot, "token_slot", torch.int32)
    _check(positions, "positions", torch.int32)
    pages, kv_heads, page_size, head_dim = k_cache.shape
    tokens = positions.numel()
    if v_cache.shape != k_cache.shape:
        raise KernelError(f"paged_attention_f32: key pages {tuple(k_cache.shape)}, value pages {tuple(v_cache.shape)}")
    if out.shape != (tokens, heads * head_dim) or token_slot.numel() != tokens:
        raise KernelError(f"paged_attention_f32: out {tuple(out.shape)} / token_slot {token_slot.numel()} "
                          f"do not match {tokens} tokens of {heads}x{head_dim}")
    if block_tables.dim() != 2:
        raise KernelError("paged_attention_f32: block_tables must be [slots, max_blocks]")
    for name, t in (("first", first), ("count", count)):
        if t is not None:
            _check(t, name, torch.int32)
            if t.numel() != tiles:
                raise KernelError(f"paged_attention_f32: {name} has {t.numel()} entries for {tiles} tiles")
    if first is None and tiles != tokens:
        raise KernelError(f"paged_attention_f32: {tiles} tiles of single tokens for {tokens} tokens")
    _lib.core().call("mrun_paged_attention_f32", _address(q), q_stride, _address(out), _address(k_cache), _address(v_cache),
                     _address(block_tables), block_tables.shape[1], _address(token_slot), _address(positions), _address(first), _address(count),
                     tiles, tile_tokens, heads, kv_heads, head_dim, page_size,
                     pages * kv_heads * page_size, scale, window, _queue())
    return out


GATE_FUNCTIONS = {"silu": 1, "gelu_tanh": 2}      # codes of the C ABI (MRUN_GATE_*); 0 = no gated epilogue


def gate_code(activation: str) -> int:
    try:
        return GATE_FUNCTIONS[activation]
    except KeyError:
        raise KernelError(f"no kernel has the gate function {activation!r} "
                          f"(known: {', '.join(sorted(GATE_FUNCTIONS))})") from None


def swiglu(gate_up: torch.Tensor, out: torch.Tensor, interleaved: bool = False, activation: str = "silu") -> torch.Tensor:
    """out = act(gate) * up.  Plain layout: gate_up[:, :I] are the gates, gate_up[:, I:] the ups.
    Interleaved: runs of eight gates followed by the eight ups of the same outputs."""
    _check(gate_up, "gate_up"); _check(out, "out", gate_up.dtype)
    tokens, inter = out.shape
    if gate_up.shape != (tokens, 2 * inter):
        raise KernelError(f"swiglu: gate_up {tuple(gate_up.shape)} vs out {tuple(out.shape)}")
    _lib.core().call("mrun_swiglu", _address(gate_up), _address(out), dtype_code(out.dtype), tokens,
                     inter, 8 if interleaved else 0, gate_code(activation), _queue())
    return out


def add_bias(y: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
    """y[t, n] += bias[n] in place; bias is float32."""
    _check(y, "y"); _check(bias, "bias", torch.float32)
    if y.dim() != 2 or bias.numel() != y.shape[1]:
        raise KernelError(f"add_bias: y {tuple(y.shape)} vs bias {tuple(bias.shape)}")
    _lib.core().call("mrun_add_bias", _address(y), dtype_code(y.dtype), _address(bias), y.shape[0],
                     y.shape[1], _queue())
    return y


SKINNY_ROWS = 16      # the decode GEMM takes up to this many rows


def skinny_ok(x, w: torch.Tensor) -> bool:
    """Whether the decode GEMM takes this product: few rows, bf16, K a multiple of 32."""
    if isinstance(x, NormedRows):
        x = x.xw
    return (x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.shape[0] <= SKINNY_ROWS
            and x.shape[1] % 32 == 0 and x.stride(1) == 1 and x.stride(0) % 8 == 0
            and x.data_ptr() % 16 == 0)


SUMS_UNIT = 2.0 ** -30        # a row's total of squares is a 64-bit integer in these units


class NormedRows:
    """The output of an RMSNorm whose row scale has not been applied yet: ``xw`` holds
    bf16(stream * norm weight) and ``sums`` (int64, a row each) each row's total of squares of the stream
    in units of 2^-30.  The decode GEMM takes it as its x and applies rsqrt(total / width + eps)
    to its own sums (so does the tcgen05 GEMM for 17 to 128 rows); :meth:`finish` makes the plain
    normed rows."""

    def __init__(self, xw: torch.Tensor, sums: torch.Tensor, eps: float):
        self.xw, self.sums, self.eps = xw, sums, float(eps)

    @property
    def shape(self):
        return self.xw.shape

    @property
    def dtype(self):
        return self.xw.dtype

    @property
    def device(self):
        return self.xw.device

    def finish(self) -> torch.Tensor:
        tokens, width = self.xw.shape
        out = torch.empty_like(self.xw)
        _lib.core().call("mrun_norm_finish", _address(self.xw), _address(self.sums), self.eps, _address(out),
                         tokens, width, _queue())
        return out


class RowSums:
    """Zeroed per-row totals for the products of one step: one buffer per device, cleared once at
    the start of a step (:meth:`begin_step`: one memset, which a captured step replays) and handed
    out slice by slice, so that no product clears its own."""

    ROWS = 16 * 1024
    _arenas = {}

    @classmethod
    def begin_step(cls, device: torch.device) -> None:
        arena = cls._arenas.get(device)
        if arena is None:
            arena = cls._arenas[device] = [torch.zeros(cls.ROWS, dtype=torch.int64, device=device), 0]
        arena[0].zero_()                   # always: a captured step must clear what other steps left
        arena[1] = 0

    @classmethod
    def take(cls, device: torch.device, rows: int = 16) -> torch.Tensor:
        """The next ``rows`` zeroed totals of the step (a multiple of 16 is taken), or a fresh
        zeroed tensor outside a step or when the step has used all of its buffer."""
        rows = -(-rows // 16) * 16
        arena = cls._arenas.get(device)
        if arena is None or arena[1] + rows > cls.ROWS:
            return torch.zeros(rows, dtype=torch.int64, device=device)
        arena[1] += rows
        return arena[0][arena[1] - rows:arena[1]]


class PendingLinear:
    """A product ``x @ w.T`` that has not run yet: a part returns it as its output where the norm
    that follows can run it with the residual sum and the norm folded into its epilogue
    (:func:`linear_into_norm`).  :meth:`compute` runs it as an ordinary product.  ``scaled`` = (rows,
    share): rows of the output's shape that join it, row t times share[t] (float32)."""

    def __init__(self, x: torch.Tensor, w: torch.Tensor, scaled=None):
        self.x, self.w, self.scaled = x, w, scaled

    @property
    def shape(self):
        return (self.x.shape[0], self.w.shape[0])

    def compute(self, out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
        y = linear(self.x, self.w, out_dtype=out_dtype)
        return y if self.scaled is None else add_scaled_rows(y, *self.scaled)


class PendingPostNorm:
    """A branch output (float32 rows) that joins the stream as ``scale * rmsnorm(branch) * weight``
    and has not been added yet: the norm that follows adds it and norms the new rows in one
    kernel (:func:`post_norm_add`).  :meth:`compute` makes the addend itself."""

    def __init__(self, branch: torch.Tensor, weight: torch.Tensor, eps: float, scale: float, act: torch.dtype):
        self.branch, self.weight, self.eps, self.scale, self.act = branch, weight, float(eps), float(scale), act

    @property
    def shape(self):
        return self.branch.shape

    def compute(self) -> torch.Tensor:
        addend = torch.zeros_like(self.branch)
        post_norm_add(addend, self.branch, self.weight, self.scale, self.eps, None, 0.0, None)
        return addend.to(self.act)


class PendingPairNorm:
    """Two branch outputs (float32 rows) that join the stream as ``share * (rmsnorm(a) * weight_a +
    rmsnorm(b) * weight_b)`` and have not been combined yet: a layer norm that follows norms both,
    adds them and norms the new rows in one kernel (:func:`pair_norm_add_layernorm`).
    :meth:`compute` makes the addend itself (float32)."""

    def __init__(self, a: torch.Tensor, b: torch.Tensor, weight_a: torch.Tensor, weight_b: torch.Tensor, eps: float,
                 share: float):
        self.a, self.b, self.weight_a, self.weight_b = a, b, weight_a, weight_b
        self.eps, self.share = float(eps), float(share)

    @property
    def shape(self):
        return self.a.shape

    def compute(self) -> torch.Tensor:
        return pair_norm_mean(self.a, self.b, self.weight_a, self.weight_b, self.eps, self.share)


class PendingPostLayerNorm:
    """A branch output (float32 rows) that joins the stream as its layer norm with ``weight`` and
    ``bias`` and has not been added yet (:func:`post_layernorm_add`).  :meth:`compute` makes the
    addend itself (float32)."""

    def __init__(self, branch: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], eps: float):
        self.branch, self.weight, self.bias, self.eps = branch, weight, bias, float(eps)

    @property
    def shape(self):
        return self.branch.shape

    def compute(self) -> torch.Tensor:
        addend = torch.zeros_like(self.branch)
        post_layernorm_add(addend, self)
        return addend


PENDING = (PendingLinear, PendingPostNorm, PendingPairNorm, PendingPostLayerNorm)      # what a block may hand to the norm after it unadded


def _normed(x):
    """(rows, totals pointer, eps) of a product's x, which may be :class:`NormedRows`."""
    if isinstance(x, NormedRows):
        return x.xw, _address(x.sums), x.eps
    return x, _address(None), 0.0


def gemm_skinny(x, w: torch.Tensor, out_dtype: torch.dtype = torch.bfloat16,
                swiglu_rows: bool = False, activation: str = "silu", rows: int = 0) -> torch.Tensor:
    """y = x @ w.T for at most 16 rows, reading w once at HBM speed.  ``swiglu_rows``: w holds gate
    and up rows interleaved in runs of eight and y = act(gate) * up has half as many columns.
    ``x`` may be :class:`NormedRows`.  ``w`` is a weight: the kernel asks for its first rows while
    the decode GEMM launched before it may still be running, so it must not be that launch's
    output (x, the stream and every output are touched only after that kernel has finished).
    ``rows``: the rows of w a block takes (8..16; 0: the count that fills the device most evenly)."""
    x, sums, eps = _normed(x)
    _check(x, "x", torch.bfloat16, dense=False); _check(w, "w", torch.bfloat16)
    m, k = x.shape
    n = w.shape[0]
    if w.shape[1] != k:
        raise KernelError(f"gemm_skinny: x {tuple(x.shape)} vs w {tuple(w.shape)}")
    out = x.new_empty((m, n // 2 if swiglu_rows else n), dtype=out_dtype)
    _lib.core().call("mrun_gemm_skinny", _address(x), _address(w), _address(out), dtype_code(out_dtype),
                     gate_code(activation) if swiglu_rows else 0, m, n, k,
                     x.stride(0) if m > 1 else max(k, x.stride(0)), out.shape[1],
                     sums, eps, _address(None), _address(None), _address(None), _address(None), rows, _address(None), 0, _address(None),
                     _queue())
    return out


def norm_fusable(pending, resid: torch.Tensor, weight: torch.Tensor) -> bool:
    """Whether :func:`linear_into_norm` takes this pending product and residual stream."""
    return (isinstance(pending, PendingLinear) and (skinny_ok(pending.x, pending.w) or tc5_ok(pending.x, pending.w))
            and resid.dtype == torch.float32 and resid.is_contiguous() and resid.shape == pending.shape
            and resid.shape[1] % 32 == 0 and weight.numel() == resid.shape[1])


def linear_into_norm(pending: PendingLinear, resid: torch.Tensor, weight: torch.Tensor, eps: float,
                     rows: int = 0) -> NormedRows:
    """resid += pending.x @ pending.w.T (32-bit, in place) and the RMSNorm of the new rows with
    ``weight``, as :class:`NormedRows`: one kernel (the decode GEMM up to 16 rows, the tcgen05
    GEMM up to 128)."""
    skinny = skinny_ok(pending.x, pending.w)
    x, in_sums, in_eps = _normed(pending.x)
    w = pending.w
    _check(x, "x", torch.bfloat16, dense=False); _check(w, "w", torch.bfloat16)
    _check(resid, "resid", torch.float32); _check(weight, "weight", torch.float32)
    m, k = x.shape
    n = w.shape[0]
    if w.shape[1] != k or resid.shape != (m, n) or weight.numel() != n:
        raise KernelError(f"linear_into_norm: x {tuple(x.shape)}, w {tuple(w.shape)}, resid {tuple(resid.shape)}, "
                          f"weight {tuple(weight.shape)}")
    extra = share = None
    ld_extra = 0
    if pending.scaled is not None:
        extra, share = pending.scaled
        ld_extra = _strided_rows(extra, "extra"); _check(share, "share", torch.float32)
        if extra.shape != (m, n) or extra.dtype != torch.bfloat16 or share.numel() != m:
            raise KernelError(f"linear_into_norm: extra {tuple(extra.shape)} {extra.dtype}, share {tuple(share.shape)}")
        if not skinny:          # the tcgen05 product's epilogue has no such rows
            add_scaled_rows(resid, extra.contiguous(), share)
    xw = x.new_empty((m, n), dtype=torch.bfloat16)
    out_sums = RowSums.take(x.device, m)
    head = (_address(x), _address(w), _address(None), dtype_code(torch.bfloat16), 0, m, n, k,
            x.stride(0) if m > 1 else max(k, x.stride(0)), n, in_sums, in_eps, _address(resid),
            _address(weight), _address(xw), _address(out_sums))
    if skinny:
        _lib.core().call("mrun_gemm_skinny", *head, rows, _address(extra), ld_extra, _address(share), _queue())
    else:
        _lib.core().call("mrun_gemm_tc5", *head, 0, _address(_tc5_status(x.device)), _queue())
    return NormedRows(xw, out_sums, eps)


def gemm_f32_nt(x: torch.Tensor, w: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """y = x @ w.T in 32-bit with a fixed summation order, whatever the number of rows.  x may have a row stride."""
    _check(x, "x", torch.float32, dense=False); _check(w, "w", torch.float32)
    if x.dim() != 2 or w.dim() != 2 or x.shape[1] != w.shape[1] or x.stride(1) != 1:
        raise KernelError(f"gemm_f32_nt: x {tuple(x.shape)} (strides {x.stride()}) vs w {tuple(w.shape)}")
    if f32_tc_ok(w):
        return gemm_f32_tc(x, w, out)
    m, k = x.shape
    n = w.shape[0]
    if out is None:
        out = x.new_empty((m, n), dtype=torch.float32)
    _check(out, "out", torch.float32)
    if out.shape != (m, n):
        raise KernelError(f"gemm_f32_nt: out is {tuple(out.shape)}, expected {(m, n)}")
    _lib.core().call("mrun_gemm_f32_nt", _address(x), _address(w), _address(out), m, n, k,
                     x.stride(0) if m > 1 else k, n, _queue())
    return out


F32_TC_SCRATCH = 128 << 20       # bytes of a product's split rows at most: longer ones go in portions
F32_TC_MIN_K = 2048
F32_TC_MIN_N = 64


def f32_tc_ok(w: torch.Tensor) -> bool:
    """Whether 32-bit products with ``w`` go to the tensor cores.  Decided by w alone, so that a row's bits do not depend on
    the rows beside it.  From K = 2,048 on they are faster from a handful of rows on, and for one or two rows from K = 4,096 on (B200, us
    after a pause, this / the chain of multiply-adds: 17 rows of 2,048 x 2,048 17 / 45, 8 of them 15.4 / 18.4, 1 of them 15.4 / 14.3, 1 row of
    6,144 x 2,816 23.4 / 21.4, of 6,144 x 4,096 29.5 / 29.6, of 2,048 x 4,096 19 / 25; 517 rows of 24,576 x 4,096
    429 / 2,233) and closer to 64 bits (3.4e-7 / 1.1e-6 at K = 4,096); at K = 1,024 a few rows take longer (8.2 / 6.0), and at
    K = 256 both are equally close (2.9e-7)."""
    n, k = w.shape
    return k >= F32_TC_MIN_K and n >= F32_TC_MIN_N and k % 4 == 0 and w.data_ptr() % 16 == 0


def _f32_tc_rows(m: int, k: int) -> int:
    """Rows that a portion of such a product splits at once."""
    return max(1, min(m, F32_TC_SCRATCH // (6 * (-(-k // 8) * 8))))


def product_scratch(w: torch.Tensor, rows: int) -> int:
    """Bytes that the product of up to ``rows`` rows with ``w`` takes beside its operands and its result."""
    if w.dtype != torch.float32 or w.dim() != 2 or not f32_tc_ok(w):
        return 0
    k = w.shape[1]
    return 6 * (-(-k // 8) * 8) * _f32_tc_rows(rows, k)


def gemm_f32_tc(x: torch.Tensor, w: torch.Tensor, out: Optional[torch.Tensor] = None, ranges: int = 0, tile: int = 0,
                cluster: int = 0) -> torch.Tensor:
    """:func:`gemm_f32_nt` on the tensor cores, every operand as the sum of three bfloat16 values (``csrc/gemm_f32_tc.cu``).
    ``ranges`` of k, ``tile`` tokens a block, ``cluster`` blocks a tile; 0: chosen, the ranges by the sizes of ``w`` alone."""
    _check(x, "x", torch.float32, dense=False); _check(w, "w", torch.float32)
    if x.dim() != 2 or w.dim() != 2 or x.shape[1] != w.shape[1] or x.stride(1) != 1:
        raise KernelError(f"gemm_f32_tc: x {tuple(x.shape)} (strides {x.stride()}) vs w {tuple(w.shape)}")
    m, k = x.shape
    n = w.shape[0]
    if out is None:
        out = x.new_empty((m, n), dtype=torch.float32)
    _check(out, "out", torch.float32)
    if out.shape != (m, n):
        raise KernelError(f"gemm_f32_tc: out is {tuple(out.shape)}, expected {(m, n)}")
    pitch = -(-k // 8) * 8
    rows = _f32_tc_rows(m, k)
    parts = x.new_empty(3 * rows * pitch, dtype=torch.bfloat16)
    status = status_word(x.device, "gemm_f32_tc", {1: "the copies of w", 2: "the copies of x", 3: "the conversion of w",
                                                   4: "the MMA issuer", 5: "the sums"})
    for at in range(0, m, rows):
        part, to = x[at:at + rows], out[at:at + rows]
        _lib.core().call("mrun_gemm_f32_tc", _address(part), _address(w), _address(to), _address(parts), part.shape[0], n, k,
                         x.stride(0) if m > 1 else k, n, ranges, tile, cluster, _address(status),
                         _queue())
    return out


TC5_ROWS = 128            # the tcgen05 GEMM takes up to this many rows
# Whether products of 17 to 128 rows go to the tcgen05 GEMM.  Off: measured on B200 at the
# Qwen3-8B shapes it loses to the vendor library at 32, 64 and 128 rows (a kernel that holds tensor
# memory has its multiprocessor to itself, so nothing of its start overlaps the kernel before).
TC5_GEMM = False


def _tc5_status(device: torch.device) -> torch.Tensor:
    return status_word(device, "gemm_tc5", {1: "the TMA producer", 2: "the MMA issuer", 3: "the epilogue",
                                            4: "the exchange inside a cluster"})


def tc5_ok(x, w: torch.Tensor) -> bool:
    """Whether the tcgen05 GEMM takes this product: 17..128 rows, bf16, K a multiple of 64."""
    if isinstance(x, NormedRows):
        x = x.xw
    return (TC5_GEMM and isinstance(x, torch.Tensor) and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16
            and x.dim() == 2 and SKINNY_ROWS < x.shape[0] <= TC5_ROWS
            and x.shape[1] % 64 == 0 and x.stride(1) == 1 and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0
            and w.is_contiguous() and w.data_ptr() % 16 == 0)


_sm_count = {}


def sm_count(device: torch.device) -> int:
    n = _sm_count.get(device)
    if n is None:
        n = _sm_count[device] = torch.cuda.get_device_properties(device).multi_processor_count
    return n


def gemm_tc5(x, w: torch.Tensor, out_dtype: torch.dtype = torch.bfloat16, swiglu_rows: bool = False,
             activation: str = "silu", split: int = 0) -> torch.Tensor:
    """y = x @ w.T for 1..128 rows on the tcgen05 tensor cores (TMA-fed, accumulators in tensor
    memory, k split over thread-block clusters whose blocks exchange partial sums through
    distributed shared memory; ``split`` = 0 lets the library choose the cluster size).
    ``swiglu_rows`` as in :func:`gemm_skinny`; ``x`` may be :class:`NormedRows`; ``w`` is a weight
    (its first tiles are asked for before the kernel before has finished).  A wait inside the
    kernel that runs out sets the status word that :func:`tc5_check` reads."""
    x, sums, eps = _normed(x)
    _check(x, "x", torch.bfloat16, dense=False); _check(w, "w", torch.bfloat16)
    m, k = x.shape
    n = w.shape[0]
    if w.shape[1] != k:
        raise KernelError(f"gemm_tc5: x {tuple(x.shape)} vs w {tuple(w.shape)}")
    out = x.new_empty((m, n // 2 if swiglu_rows else n), dtype=out_dtype)
    _lib.core().call("mrun_gemm_tc5", _address(x), _address(w), _address(out), dtype_code(out_dtype),
                     gate_code(activation) if swiglu_rows else 0, m, n, k,
                     x.stride(0) if m > 1 else max(k, x.stride(0)), out.shape[1],
                     sums, eps, _address(None), _address(None), _address(None), _address(None), split,
                     _address(_tc5_status(x.device)), _queue())
    return out


STATUS_WORDS = 32
_status_blocks = {}      # device -> (int32[STATUS_WORDS] on the device, {kernel name: (its word, {code: role})})


def _status(device: torch.device):
    return _status_blocks.get(device if device.index is not None else torch.device(device.type, torch.cuda.current_device()))


def status_word(device: torch.device, kernel: str, roles: dict) -> torch.Tensor:
    """The word a kernel with bounded waits reports into (zero = fine), one per device and kernel,
    never reallocated, so that captured graphs may keep its address.  :func:`tc5_check` reads it."""
    found = _status(device)
    if found is None:
        found = _status_blocks[device] = (torch.zeros(STATUS_WORDS, dtype=torch.int32, device=device), {})
    block, words = found
    entry = words.get(kernel)
    if entry is None:
        if len(words) == STATUS_WORDS:
            raise KernelError(f"no status word is left for {kernel}")
        entry = words[kernel] = (block[len(words):len(words) + 1], dict(roles))
    return entry[0]


def status_block(device: torch.device) -> Optional[torch.Tensor]:
    """All status words of a device in one tensor, to bring them to the host with a step's result; None before the first one."""
    found = _status(device)
    return None if found is None else found[0]


def tc5_check(device: Optional[torch.device] = None) -> None:
    """Raises if a kernel with bounded waits on the device gave up on one (and clears its status word)."""
    for dev, (block, words) in list(_status_blocks.items()):
        if device is not None and _status(device) is not _status_blocks[dev]:
            continue
        codes = block.tolist()
        for (kernel, (word, roles)), code in zip(list(words.items()), codes):
            if code:
                word.zero_()
                raise KernelError(f"{kernel}: {roles.get(code, 'a role')} waited longer than its budget on {dev}; "
                                  f"the results of that call are invalid")


def linear(x, w: torch.Tensor, out_dtype: Optional[torch.dtype] = None,
           bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """y = x @ w.T (+ bias).  float32: this library's own kernels.  bfloat16 with at most 16
    rows (decode): this library's weight-streaming tensor-core kernel (``x`` may then be
    :class:`NormedRows`).  bfloat16 otherwise (prefill): the vendor GEMM library with 32-bit
    accumulation (the reference calls its array library's matmul for the same products and adds
    an optional bias after it, crates/mrun-engine/src/load.rs:294-306)."""
    if isinstance(x, NormedRows):
        if skinny_ok(x, w) or tc5_ok(x, w):
            y = (gemm_skinny if skinny_ok(x, w) else gemm_tc5)(x, w, out_dtype or torch.bfloat16)
            return y if bias is None else add_bias(y, bias)
        x = x.finish()
    if x.dtype == torch.float32:
        y = gemm_f32_nt(x, w)
    else:
        _check(x, "x", torch.bfloat16, dense=False); _check(w, "w", torch.bfloat16)
        if skinny_ok(x, w):
            y = gemm_skinny(x, w, out_dtype or torch.bfloat16)
        elif tc5_ok(x, w):
            y = gemm_tc5(x, w, out_dtype or torch.bfloat16)
        elif out_dtype is None or out_dtype == torch.bfloat16:
            y = torch.mm(x, w.t())
        else:
            y = torch.mm(x, w.t(), out_dtype=out_dtype)
    return y if bias is None else add_bias(y, bias)


ACTIVATIONS = {"relu2": 1, "tanh": 2}      # codes of the C ABI (MRUN_ACT_*): functions of one argument


def plain_act(x: torch.Tensor, activation: str, out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """act(x) element by element in 32-bit."""
    _check(x, "x")
    out = x.new_empty(x.shape, dtype=out_dtype or x.dtype)
    _lib.core().call("mrun_plain_act", _address(x), dtype_code(x.dtype), _address(out), dtype_code(out.dtype),
                     x.numel(), ACTIVATIONS[activation], _queue())
    return out


def linear_act(x, w: torch.Tensor, activation: str) -> torch.Tensor:
    """act(x @ w.T) in x's dtype; up to 16 bfloat16 rows the activation rides in the decode GEMM's
    epilogue (which sees the sums as they would have been stored).  ``x`` may be :class:`NormedRows`."""
    if skinny_ok(x, w):
        return linear_blended(x, w, activation=activation)
    y = linear(x, w)
    if activation == "relu2":
        return relu2_scaled(y, None, 0, 1)
    return plain_act(y, activation)


def linears_batched(x: torch.Tensor, w: torch.Tensor, activation: Optional[str] = None, gate: Optional[torch.Tensor] = None,
                    out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """y[:, b] = act(x[:, b] @ w[b].T * sigmoid(gate[:, b])): ``x`` [rows, batch, K] and ``out`` [rows, batch, N]
    (may be strided along the first two axes; None: a dense one is made), ``w`` dense [batch, N, K], ``gate``
    [rows, batch] in x's dtype (rows may be strided) or None.  One launch up to 16 bfloat16 rows (this
    library's decode GEMM), else as :func:`linear_per_head` and :func:`head_gate` (without an activation)."""
    rows, batch, k = x.shape
    n = w.shape[1]
    if out is None:
        out = x.new_empty((rows, batch, n))
    if not (x.dtype == torch.bfloat16 and rows <= SKINNY_ROWS and k % 32 == 0 and x.stride(0) % 8 == 0
            and x.stride(1) % 8 == 0 and x.data_ptr() % 16 == 0):
        if activation is not None:
            raise KernelError("linears_batched: an activation comes with the decode GEMM only")
        linear_per_head(x, w, out)
        if gate is not None:
            head_gate(out.view(rows, batch * n), gate, batch)
        return out
    _check(x, "x", torch.bfloat16, dense=False); _check(w, "w", torch.bfloat16); _check(out, "out", torch.bfloat16, dense=False)
    if w.shape != (batch, n, k) or x.stride(2) != 1 or out.shape != (rows, batch, n) or out.stride(2) != 1:
        raise KernelError(f"linears_batched: x {tuple(x.shape)} (strides {x.stride()}) vs w {tuple(w.shape)}, out {tuple(out.shape)}")
    ld_gate = 0
    if gate is not None:
        ld_gate = _strided_rows(gate, "gate")
        if gate.shape != (rows, batch) or gate.dtype != x.dtype:
            raise KernelError(f"linears_batched: gate {tuple(gate.shape)} {gate.dtype}")
    _lib.core().call("mrun_gemm_skinny_batched", _address(x), _address(w), _address(out), dtype_code(out.dtype),
                     ACTIVATIONS[activation] if activation else 0, batch, rows, n, k,
                     x.stride(0) if rows > 1 else max(k, x.stride(0)), out.stride(0) if rows > 1 else max(n, out.stride(0)),
                     x.stride(1) if batch > 1 else 0, out.stride(1) if batch > 1 else n, _address(None), _address(None), 0,
                     0, 0, 0.0, _address(gate), ld_gate, _address(None), 0.0, _queue())
    return out


def linear_blended(x, w: torch.Tensor, bias: Optional[torch.Tensor] = None, blend=None,
                   activation: Optional[str] = None) -> torch.Tensor:
    """act(x @ w.T + bias) for at most 16 bfloat16 rows (:func:`skinny_ok`), the bias (float32 [N]) added to the 32-bit
    sums.  ``blend`` = (rows, share, column): the columns from ``column`` on, as many as ``rows`` has, then
    become (1 - share) * y + share * rows.  ``x`` may be :class:`NormedRows`."""
    x, sums, eps = _normed(x)
    _check(x, "x", torch.bfloat16, dense=False); _check(w, "w", torch.bfloat16)
    m, k = x.shape
    n = w.shape[0]
    if w.shape[1] != k:
        raise KernelError(f"linear_blended: x {tuple(x.shape)} vs w {tuple(w.shape)}")
    if bias is not None:
        _check(bias, "bias", torch.float32)
        if bias.numel() != n:
            raise KernelError(f"linear_blended: bias has {bias.numel()} entries for {n} columns")
    rows, share, column = blend if blend is not None else (None, 0.0, 0)
    ld_rows = columns = 0
    if rows is not None:
        ld_rows, columns = _strided_rows(rows, "blend"), rows.shape[1]
        if rows.shape[0] != m or rows.dtype != torch.bfloat16:
            raise KernelError(f"linear_blended: blend {tuple(rows.shape)} {rows.dtype}")
    out = x.new_empty((m, n), dtype=torch.bfloat16)
    _lib.core().call("mrun_gemm_skinny_batched", _address(x), _address(w), _address(out), dtype_code(out.dtype),
                     ACTIVATIONS[activation] if activation else 0, 1,
                     m, n, k, x.stride(0) if m > 1 else max(k, x.stride(0)), n, 0,
                     n, _address(bias), _address(rows), ld_rows, column, columns, share, _address(None),
                     0, sums, eps, _queue())
    return out


def linear_or_pending(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, scaled=None):
    """The last product of a part whose caller accepts a :class:`PendingLinear`: left pending in
    bfloat16 without a bias (the norm after it then runs it with the residual sum folded in: in
    the decode GEMM's epilogue up to 16 rows, as the vendor GEMM's accumulate-into-C above),
    computed otherwise.  ``scaled`` as for :class:`PendingLinear`."""
    if bias is None and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16:
        return PendingLinear(x, w, scaled)
    y = linear(x, w, bias=bias)
    return y if scaled is None else add_scaled_rows(y, *scaled)


def accumulate_ok(pending, resid: torch.Tensor) -> bool:
    """Whether :func:`linear_add_into` takes this pending product and residual stream."""
    return (isinstance(pending, PendingLinear) and isinstance(pending.x, torch.Tensor) and not tc5_ok(pending.x, pending.w)
            and not skinny_ok(pending.x, pending.w)
            and pending.x.dtype == torch.bfloat16 and pending.w.dtype == torch.bfloat16 and pending.x.dim() == 2
            and resid.dtype == torch.float32 and resid.is_contiguous() and tuple(resid.shape) == tuple(pending.shape))


def linear_add_into(resid: torch.Tensor, pending: PendingLinear) -> torch.Tensor:
    """resid += pending.x @ pending.w.T in place: the vendor GEMM with bfloat16 operands, 32-bit
    accumulation and the 32-bit stream as its C and D, so that the product is never rounded to
    bfloat16, written and read again (prompt portions and decode batches above 16 rows).  Its scaled
    rows are the caller's to add."""
    return torch.addmm(resid, pending.x, pending.w.t(), out_dtype=torch.float32, out=resid)


def sample(logits: torch.Tensor, out: torch.Tensor, temperature: Optional[torch.Tensor] = None,
           top_p: Optional[torch.Tensor] = None, top_k: Optional[torch.Tensor] = None,
           min_p: Optional[torch.Tensor] = None, keys: Optional[torch.Tensor] = None) -> torch.Tensor:
    """One token per row of float32 logits; per-row parameter arrays, None = neutral."""
    _check(logits, "logits", torch.float32); _check(out, "out", torch.int32)
    rows, vocab = logits.shape
    for name, t, dt in (("temperature", temperature, torch.float32), ("top_p", top_p, torch.float32),
                        ("top_k", top_k, torch.int32), ("min_p", min_p, torch.float32),
                        ("keys", keys, torch.int64)):
        if t is not None:
            _check(t, name, dt)
            if t.numel() < rows:
                raise KernelError(f"sample: {name} has {t.numel()} entries for {rows} rows")
    if out.numel() < rows:
        raise KernelError(f"sample: out has {out.numel()} entries for {rows} rows")
    _lib.core().call("mrun_sample", _address(logits), rows, vocab, _address(temperature), _address(top_p),
                     _address(top_k), _address(min_p), _address(keys), _address(out), _queue())
    return out


def top_logprobs(logits: torch.Tensor, n: int):
    """(ids int32 [rows, n], log-probabilities float32 [rows, n]) of the n most likely tokens of
    each row of float32 logits, most likely first, ties by the smaller id."""
    _check(logits, "logits", torch.float32)
    rows, vocab = logits.shape
    n = max(1, min(int(n), vocab))
    ids = logits.new_empty((rows, n), dtype=torch.int32)
    values = logits.new_empty((rows, n), dtype=torch.float32)
    _lib.core().call("mrun_top_logprobs", _address(logits), rows, vocab, n, _address(ids),
                     _address(values), _queue())
    return ids, values


def apply_token_mask(logits: torch.Tensor, rows: torch.Tensor, words: torch.Tensor, mask_vocab: torch.Tensor) -> None:
    """In place: logits[rows[m], i] = -inf wherever bit i of words[m] is clear or i >= mask_vocab[m].
    ``words``: int32 [masks, words a mask] (the bits of unsigned 32-bit words), 32 tokens a word."""
    _check(logits, "logits", torch.float32); _check(rows, "rows", torch.int32)
    _check(words, "words", torch.int32); _check(mask_vocab, "mask_vocab", torch.int32)
    masks = rows.numel()
    if words.dim() != 2 or words.shape[0] != masks or mask_vocab.numel() != masks:
        raise KernelError(f"apply_token_mask: {masks} rows, words {tuple(words.shape)}, {mask_vocab.numel()} vocabularies")
    _lib.core().call("mrun_apply_token_mask", _address(logits), logits.shape[1], _address(rows), _address(words),
                     words.shape[1], _address(mask_vocab), masks, _queue())


def repetition_penalty(logits: torch.Tensor, recent: torch.Tensor, penalty: torch.Tensor) -> None:
    """In place: the logits of the ids in recent[row] (negative = empty) are penalised."""
    _check(logits, "logits", torch.float32); _check(recent, "recent", torch.int32)
    _check(penalty, "penalty", torch.float32)
    rows, vocab = logits.shape
    if recent.dim() != 2 or recent.shape[0] != rows or penalty.numel() < rows:
        raise KernelError(f"repetition_penalty: recent {tuple(recent.shape)}, penalty {penalty.numel()}, rows {rows}")
    _lib.core().call("mrun_repetition_penalty", _address(logits), rows, vocab, _address(recent),
                     recent.shape[1], _address(penalty), _queue())


def scatter_i32(dst: torch.Tensor, index: torch.Tensor, value: torch.Tensor) -> None:
    """dst.view(-1)[index[i]] = value[i] for int32 tensors."""
    _check(dst, "dst", torch.int32); _check(index, "index", torch.int32); _check(value, "value", torch.int32)
    if index.numel() != value.numel():
        raise KernelError("scatter_i32: index and value differ in length")
    _lib.core().call("mrun_scatter_i32", _address(dst), _address(index), _address(value), index.numel(),
                     dst.numel(), _queue())


def select_tokens(ids: torch.Tensor, previous: torch.Tensor, source: torch.Tensor) -> None:
    """ids[r] = previous[source[r]] where source[r] >= 0 (int32 tensors)."""
    _check(ids, "ids", torch.int32); _check(previous, "previous", torch.int32); _check(source, "source", torch.int32)
    if source.numel() != ids.numel():
        raise KernelError("select_tokens: one source per row is needed")
    _lib.core().call("mrun_select_tokens", _address(ids), _address(previous), _address(source), ids.numel(),
                     previous.numel(), _queue())



# ------------------------------------------------------------------ latent attention, sandwich norms, routing

def gemm_f32_nt_batched(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """out[b] = x[b] @ w[b].T in IEEE 32-bit with a fixed summation order.  ``x`` [batch, M, K] and
    ``out`` [batch, M, N] may be strided views (unit stride along the last axis: the heads of a
    row laid side by side); ``w`` is dense [batch, N, K]."""
    _check(x, "x", torch.float32, dense=False); _check(w, "w", torch.float32); _check(out, "out", torch.float32, dense=False)
    batch, m, k = x.shape
    n = w.shape[1]
    if w.shape != (batch, n, k) or out.shape != (batch, m, n) or x.stride(2) != 1 or out.stride(2) != 1:
        raise KernelError(f"gemm_f32_nt_batched: x {tuple(x.shape)} w {tuple(w.shape)} out {tuple(out.shape)}")
    _lib.core().call("mrun_gemm_f32_nt_batched", _address(x), _address(w), _address(out), batch, m, n,
                     k, x.stride(1) if m > 1 else max(k, x.stride(1)),
                     out.stride(1) if m > 1 else max(n, out.stride(1)),
                     x.stride(0), n * k, out.stride(0), _queue())
    return out


def linear_per_head(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """out[:, h] = x[:, h] @ w[h].T for every head h: ``x`` [tokens, heads, K] and ``out``
    [tokens, heads, N] may be views into wider rows, ``w`` is dense [heads, N, K].  float32: this
    library's IEEE kernel; bfloat16: the vendor library's batched product with 32-bit sums."""
    if x.dtype == torch.float32:
        gemm_f32_nt_batched(x.transpose(0, 1), w, out.transpose(0, 1))
    else:
        _check(x, "x", torch.bfloat16, dense=False); _check(w, "w", torch.bfloat16)
        torch.bmm(x.transpose(0, 1), w.transpose(1, 2), out=out.transpose(0, 1))
    return out


PAIRINGS = {"half": 0, "interleaved": 1}     # which features a rotation pairs: (i, i + n/2) or (2i, 2i + 1)


def latent_prepare(down: torch.Tensor, q_weight: Optional[torch.Tensor], kv_weight: torch.Tensor, eps: float,
                   rot: Optional[torch.Tensor], rot_dims: int, pairing: str, slots: Optional[torch.Tensor],
                   cq: Optional[torch.Tensor], cache: Optional[torch.Tensor], q_rank: int, kv_rank: int,
                   rot_dim: int) -> None:
    """Rows of ``down`` = [query latent | key/value latent | shared key part].  ``cq`` gets the
    normed query latent; the token's row of ``cache`` ([pages, 1, page_size, width], named by
    ``slots``) gets [normed key/value latent | shared key part, its first ``rot_dims`` features
    rotated | zeros]."""
    _check(down, "down", dense=False)
    tokens = down.shape[0]
    if down.dim() != 2 or down.stride(1) != 1 or down.shape[1] != q_rank + kv_rank + rot_dim:
        raise KernelError(f"latent_prepare: down is {tuple(down.shape)}, expected width {q_rank + kv_rank + rot_dim}")
    _check(kv_weight, "kv_weight", torch.float32)
    if kv_weight.numel() != kv_rank:
        raise KernelError("latent_prepare: the key/value norm weight does not have kv_rank elements")
    if q_rank:
        _check(q_weight, "q_weight", torch.float32); _check(cq, "cq", down.dtype)
        if q_weight.numel() != q_rank or cq.shape != (tokens, q_rank):
            raise KernelError("latent_prepare: the query latent's weight or output does not have q_rank columns")
    width = kv_rank + rot_dim
    if slots is not None:
        _check(slots, "slots", torch.int32); _check(cache, "cache", down.dtype)
        if slots.numel() != tokens or cache.dim() != 4 or cache.shape[1] != 1 or cache.shape[3] < width:
            raise KernelError(f"latent_prepare: cache is {tuple(cache.shape)}, expected [pages, 1, page_size, >= {width}]")
        width = cache.shape[3]
    if rot_dims:
        _check(rot, "rot", torch.float32)
        if rot.shape != (tokens, rot_dims // 2, 2):
            raise KernelError(f"latent_prepare: rot is {tuple(rot.shape)}, expected {(tokens, rot_dims // 2, 2)}")
    _lib.core().call("mrun_latent_prepare", _address(down), dtype_code(down.dtype), down.stride(0),
                     _address(q_weight), _address(kv_weight), eps, _address(rot), rot_dims,
                     PAIRINGS[pairing], _address(slots), _address(cq), _address(cache if slots is not None else None),
                     tokens, q_rank, kv_rank, rot_dim, width, _queue())


def latent_rows(cache: torch.Tensor, block_tables: torch.Tensor, seg_slot: torch.Tensor, seg_kv_len: torch.Tensor, rows: int,
                kv_rank: int, keys: Optional[torch.Tensor] = None, rot_dim: int = 0) -> torch.Tensor:
    """[segments, rows, kv_rank]: the cached latents (the first ``kv_rank`` features of ``cache``'s rows, [pages,
    1, page_size, width]) of every segment's whole context, zeros from its length up to the next
    multiple of 128 and nothing beyond.  ``rows``: a multiple of 128 that holds every context.  With ``rot_dim``
    the features behind the latent go to the last ``rot_dim`` features of every head's row of ``keys`` (dense
    [segments, heads, rows, dim + rot_dim]) likewise."""
    _check(cache, "cache"); _check(block_tables, "block_tables", torch.int32)
    _check(seg_slot, "seg_slot", torch.int32); _check(seg_kv_len, "seg_kv_len", torch.int32)
    segments = seg_slot.numel()
    if cache.dim() != 4 or cache.shape[1] != 1 or seg_kv_len.numel() != segments or cache.shape[3] < kv_rank + rot_dim:
        raise KernelError(f"latent_rows: cache {tuple(cache.shape)}, {segments} segments, {seg_kv_len.numel()} lengths")
    heads = dim = 0
    if rot_dim:
        _check(keys, "keys", cache.dtype)
        if keys.dim() != 4 or keys.shape[0] != segments or keys.shape[2] != rows or keys.shape[3] < rot_dim:
            raise KernelError(f"latent_rows: keys {tuple(keys.shape)} for {segments} segments of {rows} rows")
        heads, dim = keys.shape[1], keys.shape[3] - rot_dim
    out = cache.new_empty((segments, rows, kv_rank))
    _lib.core().call("mrun_latent_rows", _address(cache), dtype_code(cache.dtype), _address(block_tables), block_tables.shape[1],
                     _address(seg_slot), _address(seg_kv_len), _address(out), segments, rows, cache.shape[2],
                     kv_rank, cache.shape[3], _address(keys if rot_dim else None), heads, dim,
                     rot_dim, _queue())
    return out


def latent_rotate(q: torch.Tensor, rot: torch.Tensor, rot_dims: int, pairing: str, heads: int, dim: int, rot_dim: int) -> None:
    """In place on ``q`` [tokens, heads * (dim + rot_dim)] (rows may be strided): rotates the first ``rot_dims`` features
    behind every head's ``dim`` plain ones."""
    ldq = _strided_rows(q, "q"); _check(rot, "rot", torch.float32)
    tokens = q.shape[0]
    if q.shape[1] != heads * (dim + rot_dim) or rot.shape != (tokens, rot_dims // 2, 2):
        raise KernelError(f"latent_rotate: q {tuple(q.shape)}, rot {tuple(rot.shape)}")
    _lib.core().call("mrun_latent_rotate", _address(q), ldq, dtype_code(q.dtype), _address(rot), rot_dims,
                     PAIRINGS[pairing], tokens, heads, dim, rot_dim, _queue())


def latent_query(q: torch.Tensor, rot: Optional[torch.Tensor], rot_dims: int, pairing: str, q_att: torch.Tensor,
                 heads: int, dim: int, rot_dim: int, kv_rank: int) -> None:
    """``q`` [tokens, heads * (dim + rot_dim)] (rows may be strided); fills ``q_att[t, h, kv_rank:]``
    with the head's rotated part and zeros ([tokens, heads, width])."""
    ldq = _strided_rows(q, "q"); _check(q_att, "q_att", q.dtype)
    tokens = q.shape[0]
    if q.shape != (tokens, heads * (dim + rot_dim)) or q_att.dim() != 3 or q_att.shape[:2] != (tokens, heads) \
            or q_att.shape[2] < kv_rank + rot_dim:
        raise KernelError(f"latent_query: q {tuple(q.shape)}, q_att {tuple(q_att.shape)}")
    if rot_dims:
        _check(rot, "rot", torch.float32)
        if rot.shape != (tokens, rot_dims // 2, 2):
            raise KernelError(f"latent_query: rot is {tuple(rot.shape)}, expected {(tokens, rot_dims // 2, 2)}")
    _lib.core().call("mrun_latent_query", _address(q), ldq, dtype_code(q.dtype), _address(rot), rot_dims,
                     PAIRINGS[pairing], _address(q_att), tokens, heads, dim,
                     rot_dim, kv_rank, q_att.shape[2], _queue())


def post_norm_add(stream: torch.Tensor, branch: torch.Tensor, w_post: torch.Tensor, scale: float, eps_post: float,
                  w_next: Optional[torch.Tensor], eps_next: float, out: Optional[torch.Tensor],
                  rows: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
    """stream += scale * rmsnorm(branch) * w_post (32-bit, in place), then out = rmsnorm(stream) *
    w_next (skipped when ``w_next`` is None).  With ``rows`` only those rows are computed and the
    stream is left as it is.  ``branch`` is float32."""
    _check(stream, "stream", torch.float32); _check(branch, "branch", torch.float32)
    _check(w_post, "w_post", torch.float32)
    hidden = stream.shape[1]
    n_rows = stream.shape[0] if rows is None else rows.numel()
    if branch.shape != stream.shape or w_post.numel() != hidden:
        raise KernelError(f"post_norm_add: stream {tuple(stream.shape)}, branch {tuple(branch.shape)}, weight {w_post.numel()}")
    code = F32
    if w_next is not None:
        _check(w_next, "w_next", torch.float32); _check(out, "out")
        if w_next.numel() != hidden or out.shape != (n_rows, hidden):
            raise KernelError(f"post_norm_add: out {tuple(out.shape)}, expected {(n_rows, hidden)}")
        code = dtype_code(out.dtype)
    if rows is not None:
        _check(rows, "rows", torch.int32)
    _lib.core().call("mrun_post_norm_add", _address(stream), _address(branch), _address(w_post), scale,
                     eps_post, _address(w_next), eps_next, _address(out if w_next is not None else None),
                     code, _address(rows), n_rows, hidden, _queue())
    return out


ROUTER_SCORES = {"softmax": 0, "sigmoid": 1, "logit": 2}


def route_top_k(logits: torch.Tensor, top: int, score: str = "softmax", renormalize: bool = False,
                chosen: Optional[torch.Tensor] = None, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """float32 [tokens, experts]: each token's ``top`` largest scores at their experts' places
    (divided by their sum if ``renormalize``), zero elsewhere.  ``score`` = ``"logit"``: the logits
    themselves are ranked and the chosen experts weigh the softmax over the chosen logits only.
    ``bias`` (float32, one entry an expert) is added to the logits first.  ``logits`` may be the
    first columns of wider rows (a product padded to a vendor-friendly width)."""
    _check(logits, "logits", torch.float32, dense=False)
    if logits.dim() != 2 or logits.stride(1) != 1:
        raise KernelError(f"route_top_k: logits has strides {logits.stride()}, expected rows of unit stride")
    tokens, experts = logits.shape
    if bias is not None:
        _check(bias, "bias", torch.float32)
        if bias.numel() != experts:
            raise KernelError(f"route_top_k: bias has {bias.numel()} entries for {experts} experts")
    weights = logits.new_empty((tokens, experts), dtype=torch.float32)
    if chosen is not None:
        _check(chosen, "chosen", torch.int32)
        if chosen.shape != (tokens, top):
            raise KernelError(f"route_top_k: chosen is {tuple(chosen.shape)}, expected {(tokens, top)}")
    _lib.core().call("mrun_route_top_k", _address(logits), logits.stride(0), _address(bias), _address(weights), _address(chosen),
                     tokens, experts, top, ROUTER_SCORES[score],
                     1 if renormalize else 0, _queue())
    return weights


def relu2_scaled(u: torch.Tensor, weights: Optional[torch.Tensor], experts: int, ff: int) -> torch.Tensor:
    """relu(u)^2 column by column; column c < experts * ff is also multiplied by
    ``weights[t, c // ff]`` (float32 [tokens, experts]); later columns are not."""
    _check(u, "u")
    tokens, columns = u.shape
    if weights is not None:
        _check(weights, "weights", torch.float32)
        if weights.shape != (tokens, experts):
            raise KernelError(f"relu2_scaled: weights {tuple(weights.shape)}, expected {(tokens, experts)}")
    else:
        experts, ff = 0, columns
    act = torch.empty_like(u)
    _lib.core().call("mrun_relu2_scaled", _address(u), _address(act), dtype_code(u.dtype), _address(weights), tokens,
                     columns, experts, max(1, ff), _queue())
    return act


def soft_cap(x: torch.Tensor, cap: float) -> torch.Tensor:
    """x = cap * tanh(x / cap) in place on float32."""
    _check(x, "x", torch.float32)
    _lib.core().call("mrun_soft_cap", _address(x), x.numel(), cap, _queue())
    return x


def scale(x: torch.Tensor, factor: float) -> torch.Tensor:
    """x *= factor in place on float32."""
    _check(x, "x", torch.float32)
    _lib.core().call("mrun_scale_f32", _address(x), x.numel(), factor, _queue())
    return x


# ------------------------------------------------------------------ a routed feed-forward's rows sorted by expert

def moe_sort(chosen: torch.Tensor, weights: torch.Tensor):
    """Sorts the (token, chosen expert) pairs by expert.  ``chosen``: int32 [tokens, top], a negative entry a
    pair without a row (its ``dest`` is -1; rows that no pair takes stand at the end, with source 0);
    ``weights``: float32 [tokens, experts].  Returns ``ends`` (int32 [experts]: where each expert's
    rows end), ``source`` (int32 [pairs]: the token of every row), ``row_weight`` (float32
    [pairs]) and ``dest`` (int32 [tokens, top]: the row of every pair)."""
    _check(chosen, "chosen", torch.int32); _check(weights, "weights", torch.float32)
    tokens, top = chosen.shape
    experts = weights.shape[1]
    if weights.shape[0] != tokens:
        raise KernelError(f"moe_sort: chosen {tuple(chosen.shape)} vs weights {tuple(weights.shape)}")
    dev = chosen.device
    pairs = tokens * top
    zeros = torch.zeros(3 * experts + 2 * pairs, dtype=torch.int32, device=dev)
    books = zeros[:3 * experts].view(3, experts)                              # counts, ends, cursor
    source, row_weight = zeros[3 * experts:3 * experts + pairs], zeros[3 * experts + pairs:].view(torch.float32)
    dest = torch.empty((tokens, top), dtype=torch.int32, device=dev)
    _lib.core().call("mrun_moe_sort", _address(chosen), _address(weights), tokens, experts, top,
                     _address(books[0]), _address(books[1]), _address(books[2]), _address(source), _address(row_weight), _address(dest), _queue())
    return books[1], source, row_weight, dest


def gather_rows(x: torch.Tensor, source: torch.Tensor) -> torch.Tensor:
    """out[r] = x[source[r]]."""
    _check(x, "x"); _check(source, "source", torch.int32)
    out = x.new_empty((source.numel(), x.shape[1]))
    _lib.core().call("mrun_gather_rows", _address(x), dtype_code(x.dtype), _address(source), _address(out), source.numel(),
                     x.shape[1], _queue())
    return out


def relu2_rows(u: torch.Tensor, row_weight: torch.Tensor) -> torch.Tensor:
    """relu(u)^2 times the row's weight."""
    _check(u, "u"); _check(row_weight, "row_weight", torch.float32)
    if row_weight.numel() != u.shape[0]:
        raise KernelError("relu2_rows: one weight per row is needed")
    act = torch.empty_like(u)
    _lib.core().call("mrun_relu2_rows", _address(u), _address(act), dtype_code(u.dtype), _address(row_weight), u.shape[0],
                     u.shape[1], _queue())
    return act


def combine_rows(base: Optional[torch.Tensor], rows: torch.Tensor, dest: torch.Tensor, scaled=None) -> torch.Tensor:
    """float32 out[t] = base[t] (+ share[t] * extra[t] for ``scaled`` = (extra, share)) + sum over k of
    rows[dest[t, k]], added in the order of k; a negative dest has no row."""
    _check(rows, "rows", torch.bfloat16); _check(dest, "dest", torch.int32)
    tokens, top = dest.shape
    width = rows.shape[1]
    if base is not None:
        _check(base, "base")
        if base.shape != (tokens, width) or base.dtype not in (torch.float32, torch.bfloat16):
            raise KernelError(f"combine_rows: base {tuple(base.shape)} {base.dtype}")
    extra = share = None
    if scaled is not None:
        extra, share = scaled
        _check(extra, "extra", rows.dtype); _check(share, "share", torch.float32)
        if extra.shape != (tokens, width) or share.numel() != tokens:
            raise KernelError(f"combine_rows: extra {tuple(extra.shape)}, share {tuple(share.shape)}")
    out = rows.new_empty((tokens, width), dtype=torch.float32)
    _lib.core().call("mrun_combine_rows", _address(base), 1 if base is not None and base.dtype == torch.float32 else 0,
                     _address(rows), dtype_code(rows.dtype), _address(dest), _address(out), tokens, top,
                     width, _address(extra), _address(share), _queue())
    return out


def grouped_linear(x: torch.Tensor, w: torch.Tensor, ends: torch.Tensor) -> torch.Tensor:
    """y[r] = x[r] @ w[g].T for the rows r of group g (rows ends[g-1] .. ends[g]): the vendor
    library's grouped product in bfloat16 with 32-bit sums.  ``w``: [groups, out, in], which may
    be a strided view as long as ``in`` has unit stride."""
    _check(x, "x", torch.bfloat16); _check(w, "w", torch.bfloat16, dense=False); _check(ends, "ends", torch.int32)
    return torch.nn.functional.grouped_mm(x, w.transpose(-2, -1), offs=ends)


# ------------------------------------------------------------------ several residual streams a token

def embed_streams(table: torch.Tensor, ids: torch.Tensor, out: torch.Tensor, copies: int) -> torch.Tensor:
    """out[t, s] = float(table[ids[t]]) for each of the ``copies`` streams; out is float32
    [tokens, copies * hidden]."""
    _check(table, "table"); _check(ids, "ids", torch.int32); _check(out, "out", torch.float32)
    vocab, hidden = table.shape
    tokens = ids.numel()
    if out.shape != (tokens, copies * hidden):
        raise KernelError(f"embed_streams: out is {tuple(out.shape)}, expected {(tokens, copies * hidden)}")
    _lib.core().call("mrun_embed_streams", _address(table), dtype_code(table.dtype), _address(ids), _address(out), tokens,
                     hidden, vocab, copies, _queue())
    return out


def embed_bigram(table: torch.Tensor, pairs: Optional[torch.Tensor], ids: torch.Tensor, positions: torch.Tensor,
                 token_slot: torch.Tensor, state: Optional[torch.Tensor], out: torch.Tensor, copies: int, scale: float,
                 buckets: int, mul_prev: int, mul_cur: int) -> torch.Tensor:
    """out[t, s] = table[ids[t]] * scale + pairs[row(t)] for each of the ``copies`` streams; row(t)
    = (previous token * mul_prev + token * mul_cur) mod buckets, row ``buckets`` at position 0.
    ``state`` (int32 [slots, 1]) holds the last token every request brought and is left up to
    date.  ``pairs`` None: the scaled row alone.  Padding rows (negative position) become zero."""
    _check(table, "table"); _check(ids, "ids", torch.int32); _check(out, "out", torch.float32)
    _check(positions, "positions", torch.int32); _check(token_slot, "token_slot", torch.int32)
    vocab, hidden = table.shape
    tokens = ids.numel()
    if out.shape != (tokens, copies * hidden):
        raise KernelError(f"embed_bigram: out is {tuple(out.shape)}, expected {(tokens, copies * hidden)}")
    rows = None
    if pairs is not None:
        _check(pairs, "pairs", table.dtype); _check(state, "state", torch.int32)
        if pairs.shape != (buckets + 1, hidden):
            raise KernelError(f"embed_bigram: pairs is {tuple(pairs.shape)}, expected {(buckets + 1, hidden)}")
        rows = ids.new_empty(tokens, dtype=torch.int32)
    _lib.core().call("mrun_embed_bigram", _address(table), _address(pairs), dtype_code(table.dtype), _address(ids), _address(positions),
                     _address(token_slot), _address(state), _address(rows), _address(out), tokens, hidden, vocab,
                     copies, scale, buckets, mul_prev, mul_cur, _queue())
    return out


class PendingStreams:
    """A sublayer's output (float32 rows) that has not been written into the token's streams yet,
    with the coefficients of the write: x_t <- sum_s mix[s, t] x_s + out[t] * y (``mix`` and
    ``out`` None: the plain residual sum).  The next read of the streams applies it
    (:func:`streams_step`)."""

    def __init__(self, y: torch.Tensor, mix: Optional[torch.Tensor], out: Optional[torch.Tensor]):
        self.y, self.mix, self.out = y, mix, out


def streams_step(streams: torch.Tensor, pending: Optional[PendingStreams], in_c: Optional[torch.Tensor],
                 norm_weight: Optional[torch.Tensor], eps: float, out_dtype: torch.dtype, count: int,
                 rows: Optional[torch.Tensor] = None, want_sum: bool = False):
    """Applies the pending write to the ``count`` streams of every token (float32 [tokens, count *
    width], in place), forms u = sum_s in_c[s] x_s (``in_c`` None: the plain sum) and returns its
    RMS norm times ``norm_weight`` in ``out_dtype`` (``want_sum``: the 32-bit u itself instead).
    With ``rows`` (int32) only those tokens are read and the streams stay as they are."""
    _check(streams, "streams", torch.float32)
    tokens = streams.shape[0]
    width = streams.shape[1] // count
    n_rows = tokens if rows is None else rows.numel()
    y = mix = out_c = None
    if pending is not None:
        y, mix, out_c = pending.y, pending.mix, pending.out
        _check(y, "y", torch.float32)
        if y.shape != (tokens, width):
            raise KernelError(f"streams_step: the pending output is {tuple(y.shape)}, expected {(tokens, width)}")
        for name, c, n in (("mix", mix, count * count), ("out", out_c, count)):
            if c is not None:
                _check(c, name, torch.float32)
                if c.numel() != n:
                    raise KernelError(f"streams_step: {name} has {c.numel()} entries, expected {n}")
    if in_c is not None:
        _check(in_c, "in", torch.float32)
        if in_c.numel() != count:
            raise KernelError(f"streams_step: in has {in_c.numel()} entries, expected {count}")
    if rows is not None:
        _check(rows, "rows", torch.int32)
    h = u = None
    if want_sum:
        u = streams.new_empty((n_rows, width), dtype=torch.float32)
    else:
        _check(norm_weight, "norm_weight", torch.float32)
        if norm_weight.numel() != width:
            raise KernelError(f"streams_step: the norm weight has {norm_weight.numel()} entries, the width is {width}")
        h = streams.new_empty((n_rows, width), dtype=out_dtype)
    _lib.core().call("mrun_streams_step", _address(streams), _address(y), _address(mix), _address(out_c), _address(in_c),
                     _address(None if want_sum else norm_weight), eps, _address(h),
                     dtype_code(out_dtype if h is not None else torch.float32), _address(u), _address(rows),
                     n_rows, count, width, _queue())
    return u if want_sum else h


# ------------------------------------------------------------------ recurrent mixers

def causal_conv(x: torch.Tensor, weight: torch.Tensor, state: torch.Tensor, ctx, residual: bool, silu: bool,
                bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Causal convolution per channel over each request's tokens (the last tap meets the token
    itself) plus ``bias`` (float32 [channels]), added to x (``residual``) and/or passed through SiLU.  ``x``: [tokens, channels],
    rows may be strided; ``weight``: float32 [channels, taps]; ``state``: [slots, taps - 1,
    channels] in x's dtype, the request's last inputs, read and left up to date (empty with one
    tap, which sees the token itself only)."""
    _check(x, "x", dense=False); _check(weight, "weight", torch.float32); _check(state, "state", x.dtype)
    tokens, channels = x.shape
    taps = weight.shape[1]
    if x.stride(1) != 1 or weight.shape[0] != channels or state.shape[1:] != (taps - 1, channels):
        raise KernelError(f"causal_conv: x {tuple(x.shape)}, weight {tuple(weight.shape)}, state {tuple(state.shape)}")
    if bias is not None:
        _check(bias, "bias", torch.float32)
        if bias.numel() != channels:
            raise KernelError(f"causal_conv: bias has {bias.numel()} entries for {channels} channels")
    out = x.new_empty((tokens, channels))
    _lib.core().call("mrun_causal_conv", _address(x), x.stride(0), _address(weight), _address(bias), _address(state), _address(out),
                     channels, dtype_code(x.dtype), _address(ctx.seg_q_start), _address(ctx.seg_slot),
                     ctx.num_segments, ctx.max_q_len, channels, taps,
                     1 if residual else 0, 1 if silu else 0, _queue())
    return out


def _strided_rows(t: torch.Tensor, name: str) -> int:
    _check(t, name, dense=False)
    if t.dim() != 2 or t.stride(1) != 1:
        raise KernelError(f"{name} must be rows of contiguous features")
    return t.stride(0)


CHUNK = 64                # tokens a chunk of the chunked scans
# The longest segment from which on they are worth their three kernels (B200, 16 heads of 128, decay / gated scan, us:
# 128 tokens 39 / 41 in chunks and 41 / 42 walked, 192 tokens 40 / 42 and 56 / 59, 2,048 tokens 118 / 133 and 521 / 561).
CHUNK_MIN_TOKENS = 128
# The same for the delta scan (192 tokens 59 in chunks, 67 walked; 128 tokens 56 and 48; 2,048 tokens 257 and 642).
DELTA_CHUNK_MIN_TOKENS = 192
_NEVER = 1 << 30


def _chunk_count(ctx) -> int:
    """Chunks of the step's segments, 0 where the step's segments are not known on the host."""
    if len(ctx.segments) != ctx.num_segments:
        return 0
    n = ctx.shared.get("scan_chunks")
    if n is None:
        n = ctx.shared["scan_chunks"] = sum(-(-seg.q_len // CHUNK) for seg in ctx.segments)
    return n


def _chunk_least(ctx, tokens: int, delta: bool, heads: int, dim: int, vdim: int) -> int:
    """Tokens that the step's longest segment has at least where the chunked scans take the step, _NEVER where
    the walk is the faster one whatever its length.

    A walk takes as long as its longest segment while its blocks fit the device, and longer in proportion once heads
    and segments side by side fill it; the chunks take a time in proportion to (chunk, head) pairs and, in a delta
    scan, a step a chunk of the longest segment.  ``side``: rows of chunks times heads over the longest segment, how many
    chains lie side by side.  On B200, us in chunks / walked (the lines below lie where the two meet):

    * heads of 128 x 128: chunks from the thresholds on; at 128 tokens and (chunk, head) pairs for less than half of the
      device the decay and gated scans lose by up to 7 % (4 heads, one segment 40 / 37, sixteen segments 44 / 62);
    * decay and gated, 64 x 64: a walk has a quarter of the work and the chunks' padding counts: 16 segments of 160
      tokens, a sixth of the chunks' rows empty, 64 heads 311 / 288 and 4 heads 38 / 45; of 128 tokens, 64 heads 212 / 237;
    * delta, 64 x 64: 8 segments of 192 tokens, 32 heads 154 / 121, 64 heads 285 / 218, but one segment of 192 and 64
      heads 54 / 69, two of 1,024 375 / 391; 64 x 128: segments of 200, 40 and 300, 64 heads 189 / 171; 128 x 64 loses
      where rows are padded (three segments of 300 and three short ones, 32 heads 178 / 162) and not without
      (8 segments of 192 tokens, 32 heads 256 / 261)."""
    least, longest = DELTA_CHUNK_MIN_TOKENS if delta else CHUNK_MIN_TOKENS, ctx.max_q_len
    n = _chunk_count(ctx) if longest >= least else 0
    if not n:
        return least
    rows = CHUNK * n
    side, padded, small = heads * rows / longest, 10 * rows > 11 * tokens, dim * vdim < 128 * 64
    if dim * vdim >= 128 * 128:
        return least if delta or heads * n >= 64 else 160
    if not delta:
        return _NEVER if small and padded and side > 280 else least
    if dim >= 128 and not padded:
        return least
    return least if side * longest <= (200 if small else 160) * (longest - 111) else _NEVER


def _chunks(ctx, tokens: int, least: int) -> int:
    """Chunks of the step's segments where the chunked scans take the step: a segment of at least
    ``least`` tokens, and short segments, each a chunk of its own, that pad the chunks by no more than a quarter of
    the rows and one chunk (which bounds the scratch; steps beyond it are walked as a whole, although chunks
    would still be the faster form for most: a decay scan of 16 heads of 128 over a segment of 1,024 tokens
    takes 138 us in chunks and 297 walked beside 16 single tokens).  0 otherwise."""
    n = 0 if ctx.max_q_len < least else _chunk_count(ctx)
    return n if 4 * CHUNK * n <= 5 * tokens + 4 * CHUNK else 0


def chunk_scratch_elements(dim: int, vdim: int, delta: bool) -> int:
    """16-bit elements a token and head of the chunked scans' scratch at most, with the padding that :func:`_chunks`
    admits (its one chunk beside that left to the engine's fixed allowance); 0 for sizes that are walked."""
    if dim not in (64, 128) or vdim not in (64, 128):
        return 0
    floats = (dim + CHUNK) * CHUNK + dim * vdim + dim + (CHUNK * (2 * dim + vdim) if delta else 0)      # of a chunk
    return -(-5 * 2 * floats // (4 * CHUNK))


def _chunk_scratch(ctx, delta: bool, q, k, v, ld: int, a, bias, state, out, heads: int, dim: int, vdim: int):
    """(scratch, chunks) of a scan that runs chunk by chunk, or None where it is walked."""
    chunks = _chunks(ctx, q.shape[0], _chunk_least(ctx, q.shape[0], delta, heads, dim, vdim))
    if not chunks:
        return None
    size = _lib.core().function("mrun_chunked_scan_floats")
    size.restype = _c_long
    floats = size(1 if delta else 0, _address(q), _address(k), _address(v), ld, dtype_code(q.dtype), _address(a), _address(bias),
                  _address(state), _address(out), chunks, heads, dim, vdim)
    return (q.new_empty(floats, dtype=torch.float32), chunks) if floats else None


def _chunked_scan(q, k, v, ld: int, decay, silu_inputs: bool, a, bias, tau: float, state, ctx, out, heads: int, dim: int,
                  vdim: int) -> bool:
    """Runs a decay or gated scan chunk by chunk where that form takes it."""
    found = _chunk_scratch(ctx, False, q, k, v, ld, a, bias, state, out, heads, dim, vdim)
    if found is None:
        return False
    _lib.core().call("mrun_chunked_scan", _address(q), _address(k), _address(v), ld, _address(decay), 1 if silu_inputs else 0,
                     _address(a), _address(bias), tau, _address(state), _address(out), _address(found[0]), _address(ctx.seg_q_start),
                     _address(ctx.seg_slot), ctx.num_segments, found[1], heads, dim, vdim, _queue())
    return True


def _chunked_delta_scan(q, k, v, ld: int, a, b, ldb: int, a_log, dt_bias, state, ctx, out, heads: int, kv_heads: int, dim: int,
                        vdim: int) -> bool:
    """Runs a delta scan chunk by chunk where that form takes it."""
    found = _chunk_scratch(ctx, True, q, k, v, ld, a, dt_bias, state, out, heads, dim, vdim)
    if found is None:
        return False
    _lib.core().call("mrun_chunked_delta_scan", _address(q), _address(k), _address(v), ld, heads // kv_heads, _address(a), _address(b),
                     ldb, _address(a_log), _address(dt_bias), _address(state), _address(out), _address(found[0]), _address(ctx.seg_q_start),
                     _address(ctx.seg_slot), ctx.num_segments, found[1], heads, dim, vdim, _queue())
    return True


def decay_scan(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, decay: torch.Tensor, state: torch.Tensor, ctx,
               heads: int, dim: int, vdim: int, silu_inputs: bool) -> torch.Tensor:
    """Per head S_t = decay_h S_(t-1) + k_t v_t^T, o_t = S_t^T q_t over each request's tokens, from
    and into ``state`` (float32 [slots, heads, dim, vdim]).  q, k, v: column slices of one matrix
    of rows.  Returns float32 [tokens, heads * vdim]."""
    ld = _strided_rows(q, "q")
    if _strided_rows(k, "k") != ld or _strided_rows(v, "v") != ld or k.dtype != q.dtype or v.dtype != q.dtype:
        raise KernelError("decay_scan: q, k and v must be slices of one matrix")
    _check(decay, "decay", torch.float32); _check(state, "state", torch.float32)
    tokens = q.shape[0]
    if q.shape[1] != heads * dim or k.shape[1] != heads * dim or v.shape[1] != heads * vdim \
            or state.shape[1:] != (heads, dim, vdim) or decay.numel() != heads:
        raise KernelError("decay_scan: sizes do not match")
    out = q.new_empty((tokens, heads * vdim), dtype=torch.float32)
    if _chunked_scan(q, k, v, ld, decay, silu_inputs, None, None, 1.0, state, ctx, out, heads, dim, vdim):
        return out
    scratch = q.new_empty(tokens * (2 * heads * dim + heads * vdim), dtype=torch.float32)
    _lib.core().call("mrun_decay_scan", _address(q), _address(k), _address(v), ld, dtype_code(q.dtype), _address(decay),
                     _address(state), _address(out), _address(scratch), _address(ctx.seg_q_start), _address(ctx.seg_slot),
                     ctx.num_segments, tokens, heads, dim, vdim,
                     1 if silu_inputs else 0, _queue())
    return out


def delta_scan(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, a: torch.Tensor, b: torch.Tensor,
               a_log: torch.Tensor, dt_bias: torch.Tensor, state: torch.Tensor, ctx, heads: int, kv_heads: int,
               dim: int, vdim: int) -> torch.Tensor:
    """The gated delta rule with a decay per head and key channel over each request's tokens (see
    ``csrc/recurrent.cu``).  q, k ([tokens, kv_heads * dim]) and v ([tokens, heads * vdim]):
    column slices of one matrix; ``a``: float32 [tokens, heads * dim]; ``b``: [tokens, heads],
    rows may be strided.  Returns float32 [tokens, heads * vdim]."""
    ld = _strided_rows(q, "q")
    if _strided_rows(k, "k") != ld or _strided_rows(v, "v") != ld or k.dtype != q.dtype or v.dtype != q.dtype:
        raise KernelError("delta_scan: q, k and v must be slices of one matrix")
    ldb = _strided_rows(b, "b")
    _check(a, "a", torch.float32); _check(a_log, "a_log", torch.float32); _check(dt_bias, "dt_bias", torch.float32)
    _check(state, "state", torch.float32)
    tokens = q.shape[0]
    if q.shape[1] != kv_heads * dim or k.shape[1] != kv_heads * dim or v.shape[1] != heads * vdim \
            or a.shape != (tokens, heads * dim) or b.shape != (tokens, heads) or b.dtype != q.dtype \
            or a_log.numel() != heads or dt_bias.numel() != heads * dim or state.shape[1:] != (heads, dim, vdim):
        raise KernelError("delta_scan: sizes do not match")
    out = q.new_empty((tokens, heads * vdim), dtype=torch.float32)
    if _chunked_delta_scan(q, k, v, ld, a, b, ldb, a_log, dt_bias, state, ctx, out, heads, kv_heads, dim, vdim):
        return out
    scratch = q.new_empty(tokens * (2 * kv_heads * dim + heads * (vdim + dim + 1)), dtype=torch.float32)
    _lib.core().call("mrun_delta_scan", _address(q), _address(k), _address(v), ld, dtype_code(q.dtype),
                     heads // kv_heads, _address(a), _address(b), ldb, _address(a_log), _address(dt_bias), _address(state),
                     _address(out), _address(scratch), _address(ctx.seg_q_start), _address(ctx.seg_slot), ctx.num_segments,
                     tokens, heads, dim, vdim, _queue())
    return out


def gated_scan(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, a: torch.Tensor, bias: torch.Tensor, tau: float,
               state: torch.Tensor, ctx, heads: int, dim: int, vdim: int) -> torch.Tensor:
    """Linear attention with a decay per head and key channel over each request's tokens: g =
    sigmoid(a + bias)^(1 / tau), S <- g * S (rows) + k v^T, o = S^T (q * dim^-1/2), from and into
    ``state`` (float32 [slots, heads, dim, vdim]).  q, k ([tokens, heads * dim]) and v ([tokens,
    heads * vdim]): column slices of one matrix; ``a``: float32 [tokens, heads * dim]; ``bias``:
    float32 [heads * dim].  Returns float32 [tokens, heads * vdim]."""
    ld = _strided_rows(q, "q")
    if _strided_rows(k, "k") != ld or _strided_rows(v, "v") != ld or k.dtype != q.dtype or v.dtype != q.dtype:
        raise KernelError("gated_scan: q, k and v must be slices of one matrix")
    _check(a, "a", torch.float32); _check(bias, "bias", torch.float32); _check(state, "state", torch.float32)
    tokens = q.shape[0]
    if q.shape[1] != heads * dim or k.shape[1] != heads * dim or v.shape[1] != heads * vdim \
            or a.shape != (tokens, heads * dim) or bias.numel() != heads * dim or state.shape[1:] != (heads, dim, vdim):
        raise KernelError("gated_scan: sizes do not match")
    out = q.new_empty((tokens, heads * vdim), dtype=torch.float32)
    if _chunked_scan(q, k, v, ld, None, False, a, bias, tau, state, ctx, out, heads, dim, vdim):
        return out
    scratch = q.new_empty(tokens * heads * (3 * dim + vdim), dtype=torch.float32)
    _lib.core().call("mrun_gated_scan", _address(q), _address(k), _address(v), ld, dtype_code(q.dtype), _address(a), _address(bias),
                     tau, _address(state), _address(out), _address(scratch), _address(ctx.seg_q_start), _address(ctx.seg_slot),
                     ctx.num_segments, tokens, heads, dim, vdim, _queue())
    return out


GATE_SHAPES = {"sigmoid": 0, "silu": 1}        # what a gated norm passes its gate through


def gated_norm(o: torch.Tensor, weight: torch.Tensor, gate: torch.Tensor, eps: float, groups: int,
               out_dtype: torch.dtype, gate_function: str = "sigmoid", out: Optional[torch.Tensor] = None,
               scale: float = 1.0) -> torch.Tensor:
    """Per group of ``o.shape[1] // groups`` features: o / sqrt(mean(o^2) + eps) * weight *
    f(gate), f the sigmoid or SiLU (``gate_function``).  ``o``: float32 [tokens, features]; ``weight``: float32, one entry per feature
    of a row or of a group; ``gate``: [tokens, features] in ``out_dtype``, rows may be strided.
    ``out``: where the result goes, times ``scale`` (rows may be strided)."""
    _check(o, "o", torch.float32); _check(weight, "weight", torch.float32)
    ldg = _strided_rows(gate, "gate")
    tokens, features = o.shape
    n = features // groups
    if gate.shape != o.shape or gate.dtype != out_dtype or weight.numel() not in (n, features) or n * groups != features:
        raise KernelError("gated_norm: sizes do not match")
    if out is None:
        out = o.new_empty((tokens, features), dtype=out_dtype)
    ldo = _strided_rows(out, "out")
    if out.shape != o.shape or out.dtype != out_dtype:
        raise KernelError(f"gated_norm: out is {tuple(out.shape)} {out.dtype}")
    _lib.core().call("mrun_gated_norm", _address(o), _address(weight), weight.numel(), _address(gate), ldg,
                     dtype_code(out_dtype), eps, _address(out), ldo, scale, tokens, groups, n,
                     GATE_SHAPES[gate_function], _queue())
    return out


def skip_gate_norm(o: torch.Tensor, x: torch.Tensor, skip: torch.Tensor, z: torch.Tensor, weight: torch.Tensor, eps: float,
                   groups: int) -> torch.Tensor:
    """y = (o + skip_h * x) * SiLU(z), then per group of ``o.shape[1] // groups`` features y /
    sqrt(mean(y^2) + eps) * weight.  ``o``: float32 [tokens, features]; ``x``, ``z``: [tokens,
    features] of the activation type, rows may be strided; ``skip``: float32, one entry a head;
    ``weight``: float32 [features].  Returns rows of the activation type."""
    _check(o, "o", torch.float32); _check(weight, "weight", torch.float32); _check(skip, "skip", torch.float32)
    ldx, ldz = _strided_rows(x, "x"), _strided_rows(z, "z")
    tokens, features = o.shape
    if x.shape != o.shape or z.shape != o.shape or x.dtype != z.dtype or weight.numel() != features or features % groups \
            or features % skip.numel():
        raise KernelError(f"skip_gate_norm: o {tuple(o.shape)}, x {tuple(x.shape)}, z {tuple(z.shape)}, {groups} groups")
    out = o.new_empty((tokens, features), dtype=x.dtype)
    _lib.core().call("mrun_skip_gate_norm", _address(o), _address(x), ldx, _address(skip), features // skip.numel(),
                     _address(z), ldz, _address(weight), dtype_code(x.dtype), eps, _address(out),
                     tokens, groups, features // groups, _queue())
    return out


def token_blend(x: torch.Tensor, mu: torch.Tensor, state: torch.Tensor, ctx) -> torch.Tensor:
    """[tokens, S, channels]: x_t + (x_(t-1) - x_t) * mu[s] over each request's tokens, the row before
    a portion's first token from ``state`` ([slots, 1, channels] in x's dtype, zeros at the start),
    which is left holding the portion's last row.  ``mu``: float32 [S, channels]."""
    ldx = _strided_rows(x, "x")
    _check(mu, "mu", torch.float32); _check(state, "state", x.dtype)
    tokens, channels = x.shape
    if mu.dim() != 2 or mu.shape[1] != channels or state.shape[1:] != (1, channels):
        raise KernelError(f"token_blend: x {tuple(x.shape)}, mu {tuple(mu.shape)}, state {tuple(state.shape)}")
    out = x.new_empty((tokens, mu.shape[0], channels))
    _lib.core().call("mrun_token_blend", _address(x), ldx, _address(mu), _address(state), _address(out), dtype_code(x.dtype),
                     _address(ctx.seg_q_start), _address(ctx.seg_slot), ctx.num_segments, ctx.max_q_len,
                     channels, mu.shape[0], _queue())
    return out


def bonus_scan(r: torch.Tensor, k: torch.Tensor, v: torch.Tensor, a: torch.Tensor, bias: torch.Tensor, bonus: torch.Tensor,
               state: torch.Tensor, ctx, heads: int, dim: int, vdim: int) -> torch.Tensor:
    """Linear attention with a decay per head and key channel and a bonus for the current token, over
    each request's tokens: g = exp(-exp(a + bias)), o = S^T r + (r . (bonus * k)) v, S <- g * S
    (rows) + k v^T, from and into ``state`` (float32 [slots, heads, dim, vdim]).  r, k ([tokens,
    heads * dim]) and v ([tokens, heads * vdim]): column slices of one matrix; ``a``: float32 [tokens,
    heads * dim]; ``bias`` and ``bonus``: float32 [heads * dim].  Returns float32 [tokens, heads *
    vdim]."""
    ld = _strided_rows(r, "r")
    if _strided_rows(k, "k") != ld or _strided_rows(v, "v") != ld or k.dtype != r.dtype or v.dtype != r.dtype:
        raise KernelError("bonus_scan: r, k and v must be slices of one matrix")
    for name, t in (("a", a), ("bias", bias), ("bonus", bonus), ("state", state)):
        _check(t, name, torch.float32)
    tokens = r.shape[0]
    if r.shape[1] != heads * dim or k.shape[1] != heads * dim or v.shape[1] != heads * vdim \
            or a.shape != (tokens, heads * dim) or bias.numel() != heads * dim or bonus.numel() != heads * dim \
            or state.shape[1:] != (heads, dim, vdim):
        raise KernelError("bonus_scan: sizes do not match")
    out = r.new_empty((tokens, heads * vdim), dtype=torch.float32)
    scratch = None
    if not _lib.core().function("mrun_scan_walks")(0, _address(r), _address(k), _address(v), ld, dtype_code(r.dtype), _address(a),
                                                   _address(bias), _address(bonus), _address(state), dim, vdim):
        scratch = r.new_empty(tokens * heads * (3 * dim + vdim), dtype=torch.float32)
    _lib.core().call("mrun_bonus_scan", _address(r), _address(k), _address(v), ld, dtype_code(r.dtype), _address(a), _address(bias),
                     _address(bonus), _address(state), _address(out), _address(scratch), _address(ctx.seg_q_start), _address(ctx.seg_slot),
                     ctx.num_segments, ctx.max_q_len, tokens, heads, dim, vdim, _queue())
    return out


def ssm_scan(c: torch.Tensor, b: torch.Tensor, x: torch.Tensor, dt: torch.Tensor, dt_bias: torch.Tensor,
             a_log: torch.Tensor, state: torch.Tensor, ctx, heads: int, groups: int, size: int, vdim: int) -> torch.Tensor:
    """A selective state-space recurrence over each request's tokens: step = softplus(dt + dt_bias) and
    decay = exp(-exp(a_log) * step) per head; S <- decay * S + step * b x^T, y = S^T c, from and into
    ``state`` (float32 [slots, heads, size, vdim]).  c, b ([tokens, groups * size]) and x ([tokens,
    heads * vdim]): column slices of one matrix; ``dt``: [tokens, heads] in the same type, rows may be
    strided; ``dt_bias``, ``a_log``: float32 [heads].  Returns float32 [tokens, heads * vdim]."""
    ld, lddt = _strided_rows(c, "c"), _strided_rows(dt, "dt")
    if _strided_rows(b, "b") != ld or _strided_rows(x, "x") != ld or len({t.dtype for t in (c, b, x, dt)}) != 1:
        raise KernelError("ssm_scan: c, b and x must be slices of one matrix, dt of its type")
    for name, t in (("dt_bias", dt_bias), ("a_log", a_log), ("state", state)):
        _check(t, name, torch.float32)
    tokens = c.shape[0]
    if c.shape[1] != groups * size or b.shape[1] != groups * size or x.shape[1] != heads * vdim or heads % groups \
            or dt.shape != (tokens, heads) or dt_bias.numel() != heads or a_log.numel() != heads \
            or state.shape[1:] != (heads, size, vdim):
        raise KernelError("ssm_scan: sizes do not match")
    out = c.new_empty((tokens, heads * vdim), dtype=torch.float32)
    scratch = None
    if not _lib.core().function("mrun_scan_walks")(1, _address(c), _address(b), _address(x), ld, dtype_code(c.dtype), _address(None),
                                                   _address(dt_bias), _address(None), _address(state), size, vdim):
        scratch = c.new_empty(tokens * (2 * groups * size + heads * (vdim + 1)), dtype=torch.float32)
    _lib.core().call("mrun_ssm_scan", _address(c), _address(b), _address(x), ld, dtype_code(c.dtype), heads // groups,
                     _address(dt), lddt, _address(dt_bias), _address(a_log), _address(state), _address(out), _address(scratch),
                     _address(ctx.seg_q_start), _address(ctx.seg_slot), ctx.num_segments, ctx.max_q_len, tokens, heads,
                     size, vdim, _queue())
    return out


def selective_scan(x: torch.Tensor, z: torch.Tensor, dt: torch.Tensor, dt_bias: torch.Tensor, a: torch.Tensor, b: torch.Tensor,
                   c: torch.Tensor, skip: torch.Tensor, state: torch.Tensor, ctx) -> torch.Tensor:
    """A state-space recurrence with a decay per channel and state over each request's tokens: step =
    softplus(dt + dt_bias); S <- exp(step * a) * S + step * x * b; y = (S . c + skip * x) * SiLU(z), from and into
    ``state`` (float32 [slots, inner, states]).  ``x``, ``z``: [tokens, inner]; ``b``, ``c``: [tokens, states] column
    slices of one matrix, in 32-bit or, where every segment is a single token, in x's dtype; ``dt``: float32 [tokens, inner]; rows may be strided; ``a``: float32 [inner,
    states] (negative rates).  Returns dense rows of x's dtype."""
    ldx, ldz, ldb, lddt = _strided_rows(x, "x"), _strided_rows(z, "z"), _strided_rows(b, "b"), _strided_rows(dt, "dt")
    for name, t in (("dt_bias", dt_bias), ("a", a), ("skip", skip), ("state", state)):
        _check(t, name, torch.float32)
    tokens, inner = x.shape
    states = b.shape[1]
    if z.shape != x.shape or dt.shape != x.shape or dt.dtype != torch.float32 or c.shape != b.shape or b.shape[0] != tokens \
            or _strided_rows(c, "c") != ldb or a.shape != (inner, states) or dt_bias.numel() != inner or skip.numel() != inner \
            or state.shape[1:] != (inner, states) or z.dtype != x.dtype or c.dtype != b.dtype \
            or b.dtype != (x.dtype if ctx.max_q_len == 1 else torch.float32):
        raise KernelError("selective_scan: sizes or types do not match")
    out = x.new_empty((tokens, inner))
    _lib.core().call("mrun_selective_scan", _address(x), ldx, _address(z), ldz, _address(b), _address(c), ldb,
                     dtype_code(x.dtype), _address(dt), lddt, _address(dt_bias), _address(a), _address(skip), _address(state), _address(out),
                     inner, _address(ctx.seg_q_start), _address(ctx.seg_slot), ctx.num_segments, ctx.max_q_len,
                     tokens, inner, states, _queue())
    return out


def head_gate(y: torch.Tensor, gate: torch.Tensor, heads: int) -> torch.Tensor:
    """In place: every head of ``y`` ([tokens, heads * n]) times the 32-bit sigmoid of its entry
    of ``gate`` ([tokens, heads] in the dtype of ``y``, rows may be strided)."""
    _check(y, "y")
    ldg = _strided_rows(gate, "gate")
    tokens, features = y.shape
    if gate.shape != (tokens, heads) or gate.dtype != y.dtype or features % heads:
        raise KernelError("head_gate: sizes do not match")
    _lib.core().call("mrun_head_gate", _address(y), _address(gate), ldg, dtype_code(y.dtype), tokens, heads,
                     features // heads, _queue())
    return y


# ------------------------------------------------------------------ differential attention

def diff_rope_cache(qkv: torch.Tensor, rot: Optional[torch.Tensor], rot_dims: int, slots: Optional[torch.Tensor],
                    k_cache: torch.Tensor, v_cache: torch.Tensor, heads: int, kv_heads: int, dim: int, vdim: int,
                    page_size: int) -> None:
    """Rotates the q and k vectors of ``qkv`` ([tokens, 2 heads dim | 2 kv_heads dim | kv_heads
    vdim], maps outermost) in place and stores k and v in the pages ``slots`` names (key pages
    [2, pages, kv_heads, page, dim], value pages [chunks, pages, kv_heads, page, vdim / chunks])."""
    _check(qkv, "qkv"); _check(k_cache, "k_cache", qkv.dtype); _check(v_cache, "v_cache", qkv.dtype)
    tokens = qkv.shape[0]
    chunks, pages = v_cache.shape[0], v_cache.shape[1]
    if k_cache.shape != (2, pages, kv_heads, page_size, dim) or v_cache.shape != (chunks, pages, kv_heads, page_size, vdim // chunks) \
            or qkv.shape[1] != 2 * heads * dim + 2 * kv_heads * dim + kv_heads * vdim:
        raise KernelError("diff_rope_cache: sizes do not match")
    if rot is not None:
        _check(rot, "rot", torch.float32)
        if rot.shape != (tokens, rot_dims // 2, 2):
            raise KernelError(f"diff_rope_cache: rot is {tuple(rot.shape)}")
    if slots is not None:
        _check(slots, "slots", torch.int32)
    _lib.core().call("mrun_diff_rope_cache", _address(qkv), qkv.stride(0), dtype_code(qkv.dtype), _address(rot),
                     rot_dims if rot is not None else 0, _address(slots), _address(k_cache), _address(v_cache), pages,
                     tokens, heads, kv_heads, dim, vdim, vdim // chunks,
                     page_size, _queue())


def diff_attention(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, block_tables: torch.Tensor,
                   token_slot: torch.Tensor, positions: torch.Tensor, heads: int, vdim: int, scale: float,
                   lam: float, eps: float, out_scale: float, window: int = 0) -> torch.Tensor:
    """Both maps of a differential attention, their combination a1 - lam * a2 and the head norm
    (times ``out_scale``) in one kernel on CUDA cores, 32-bit arithmetic.  ``q``: rows [2, heads,
    dim], may be a column slice of a wider matrix."""
    ld = _strided_rows(q, "q")
    _check(k_cache, "k_cache", q.dtype); _check(v_cache, "v_cache", q.dtype)
    _check(block_tables, "block_tables", torch.int32); _check(token_slot, "token_slot", torch.int32)
    _check(positions, "positions", torch.int32)
    maps, pages, kv_heads, page_size, dim = k_cache.shape
    tokens = positions.numel()
    if maps != 2 or q.shape != (tokens, 2 * heads * dim) or v_cache.shape[1:4] != (pages, kv_heads, page_size) \
            or v_cache.shape[0] * v_cache.shape[4] != vdim:
        raise KernelError("diff_attention: sizes do not match")
    out = q.new_empty((tokens, heads * vdim))
    _lib.core().call("mrun_diff_attention", _address(q), ld, _address(out), _address(k_cache), _address(v_cache),
                     dtype_code(q.dtype), _address(block_tables), block_tables.shape[1], _address(token_slot),
                     _address(positions), pages, tokens, heads, kv_heads, dim,
                     vdim, v_cache.shape[4], page_size, scale, lam,
                     eps, out_scale, window, _queue())
    return out


def diff_combine(maps: torch.Tensor, heads: int, vdim: int, lam: float, eps: float, out_scale: float) -> torch.Tensor:
    """``maps``: [2, chunks, tokens, heads * vdim / chunks], the maps' outputs chunk by chunk;
    returns (a1 - lam * a2) / rms over each head's ``vdim`` values * ``out_scale``."""
    _check(maps, "maps")
    two, chunks, tokens, row = maps.shape
    if two != 2 or row * chunks != heads * vdim:
        raise KernelError("diff_combine: sizes do not match")
    out = maps.new_empty((tokens, heads * vdim))
    _lib.core().call("mrun_diff_combine", _address(maps), _address(out), dtype_code(maps.dtype), tokens, heads,
                     vdim, vdim // chunks, lam, eps, out_scale, _queue())
    return out


# ------------------------------------------------------------------ experts chosen by a table

def table_route(token_ids: torch.Tensor, table: torch.Tensor, experts: int, chosen: Optional[torch.Tensor] = None) -> torch.Tensor:
    """float32 [tokens, experts]: 1 / top at the experts that row ``token id`` of ``table`` (int32
    [vocab, top]) names, zero elsewhere; ``chosen`` (int32 [tokens, top]) gets the experts."""
    _check(token_ids, "token_ids", torch.int32); _check(table, "table", torch.int32)
    tokens = token_ids.numel()
    vocab, top = table.shape
    weights = token_ids.new_empty((tokens, experts), dtype=torch.float32)
    if chosen is not None:
        _check(chosen, "chosen", torch.int32)
        if chosen.shape != (tokens, top):
            raise KernelError(f"table_route: chosen is {tuple(chosen.shape)}, expected {(tokens, top)}")
    _lib.core().call("mrun_table_route", _address(token_ids), _address(table), _address(weights), _address(chosen), tokens,
                     vocab, experts, top, _queue())
    return weights


def clamped_glu(u: torch.Tensor, weights: Optional[torch.Tensor], blocks: int, ff: int, limit: float, alpha: float,
                up_offset: float = 1.0, out: Optional[torch.Tensor] = None, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``u``: [rows, blocks * 2 * ff], a block of [gate | up] columns per expert.  Returns [rows,
    blocks * ff]: g * sigmoid(alpha * g) * (clamp(up, +-limit) + up_offset) with g = min(gate,
    limit), times ``weights[row, block]`` (float32 [rows, blocks]) or ``weights[row]`` (float32
    [rows]).  ``limit`` infinite: no clamp (alpha = 1 and up_offset = 0: SiLU(gate) * up).  ``u``,
    ``weights`` and ``out`` may be column slices of wider matrices.  ``bias`` (float32, laid out like a
    row of ``u``) is added to gate and up before the clamp: the projections' biases, never rounded
    into ``u``."""
    ldu = _strided_rows(u, "u")
    rows = u.shape[0]
    if u.shape[1] != blocks * 2 * ff:
        raise KernelError(f"clamped_glu: u is {tuple(u.shape)}, expected width {blocks * 2 * ff}")
    per_block, ldw = 0, 0
    if weights is not None:
        _check(weights, "weights", torch.float32, dense=False)
        if weights.dim() == 2 and weights.shape == (rows, blocks) and weights.stride(1) == 1:
            per_block, ldw = 1, weights.stride(0)
        elif weights.dim() == 1 and weights.numel() == rows:
            ldw = weights.stride(0)
        elif weights.dim() == 2 and weights.shape == (rows, 1):
            ldw = weights.stride(0)
        else:
            raise KernelError(f"clamped_glu: weights {tuple(weights.shape)}")
    if bias is not None:
        _check(bias, "bias", torch.float32)
        if bias.numel() != blocks * 2 * ff:
            raise KernelError(f"clamped_glu: bias has {bias.numel()} entries, a row has {blocks * 2 * ff}")
    if out is None:
        out = u.new_empty((rows, blocks * ff))
    lda = _strided_rows(out, "out")
    if out.shape != (rows, blocks * ff) or out.dtype != u.dtype:
        raise KernelError(f"clamped_glu: out is {tuple(out.shape)} {out.dtype}")
    _lib.core().call("mrun_clamped_glu", _address(u), ldu, _address(out), lda, dtype_code(u.dtype), _address(weights),
                     ldw, per_block, rows, blocks, ff, limit,
                     alpha, up_offset, _address(bias), _queue())
    return out


def route_grouped(logits: torch.Tensor, experts: int, top: int, groups: int, keep: int, group_top: int, scale: float,
                  chosen: Optional[torch.Tensor] = None, score: str = "sigmoid", correction: Optional[torch.Tensor] = None,
                  identity: int = 0, renormalize: bool = True, handed_on=None):
    """The choice of a router over groups of experts.  ``logits``: float32 [tokens, experts + identity] or one
    column more (the gate of a shared expert).  Scores are the logits' sigmoids or their softmax
    (``score``); ``correction`` (float32, one entry an expert) is added where experts are ranked, not where
    they weigh.  The experts form ``groups`` equal groups of neighbours, a group's rank is the sum of its
    ``group_top`` largest ranks, and only experts of the ``keep`` best groups can be chosen.
    Returns (float32 [tokens, experts]: score * ``scale``, divided by the sum of the chosen + 1e-20 with
    ``renormalize``, at the chosen experts and zero elsewhere; float32 [tokens]: the sigmoid of the last
    column, or None; float32 [tokens]: the sum of the weights of the chosen among the last ``identity``
    experts, or None; for ``handed_on`` = :class:`NormedRows`, the rows those experts hand on, it contains
    their norm's factor).  In ``chosen`` an identity expert is -1.  ``logits`` may be the first columns of wider
    rows (a product padded to a vendor-friendly width): its row stride is passed on."""
    _check(logits, "logits", torch.float32, dense=False)
    tokens, columns = logits.shape
    total = experts + identity
    if columns not in (total, total + 1):
        raise KernelError(f"route_grouped: logits is {tuple(logits.shape)}, expected {total} or {total + 1} columns")
    if logits.stride(1) != 1 or logits.stride(0) < columns:
        raise KernelError(f"route_grouped: logits has strides {logits.stride()}, expected rows of unit stride")
    if correction is not None:
        _check(correction, "correction", torch.float32)
        if correction.numel() != total:
            raise KernelError(f"route_grouped: correction has {correction.numel()} entries for {total} experts")
    weights = logits.new_empty((tokens, experts), dtype=torch.float32)
    shared = logits.new_empty(tokens, dtype=torch.float32) if columns > total else None
    unchanged = logits.new_empty(tokens, dtype=torch.float32) if identity else None
    if chosen is not None:
        _check(chosen, "chosen", torch.int32)
        if chosen.shape != (tokens, top):
            raise KernelError(f"route_grouped: chosen is {tuple(chosen.shape)}, expected {(tokens, top)}")
    _lib.core().call("mrun_route_grouped", _address(logits), logits.stride(0), ROUTER_SCORES[score], _address(correction),
                     _address(weights), _address(unchanged), _address(shared), _address(chosen), tokens, experts,
                     identity, top, groups, keep, group_top,
                     1 if renormalize else 0, scale,
                     *((_address(handed_on.sums), handed_on.shape[1], handed_on.eps) if handed_on is not None
                       else (_address(None), 0, 0.0)), _queue())
    return weights, shared, unchanged
