"""Wrappers and kernel choice for latent attention (``csrc/latent_attention.cu``, ``csrc/latent_attention_mma.cu``).

Queries and results are head-major, [H, rows, width], so that the per-head products with the key and value
up-projections are grouped matrix products (one group per head).  ``rows`` is the number of tokens, rounded up to
whole 128-row tiles where the tcgen05 grouped product runs."""
from __future__ import annotations

from ctypes import c_float, c_int, c_longlong
from typing import Optional

import torch

from . import _check, _dt, _i32, _ptr, _stream, gemm_tiled, lib
from .layer_ops import _act_args, _f32

TILE = 128


def prepare(proj: torch.Tensor, q_off: int, kv_off: int, norm_w: torch.Tensor, eps: float, freq: Optional[torch.Tensor],
            pairing: str, amp: float, positions, tok_entry, block_table, cache: torch.Tensor, page_size: int,
            q_plain: torch.Tensor, q_rot: torch.Tensor, n_tokens: int, H: int, D: int, R: int, C: int,
            write_cache: bool = True, q_src: Optional[torch.Tensor] = None, rot_block: bool = False) -> None:
    """From the input product (float32 [T, >= ...]): the normed latent and the rotated key part go to the token's
    page, the plain query parts to q_plain [H, rows, D], the rotated ones to q_rot float32 [H, rows, R].  ``freq``: the
    rotary table in float64 (the angle is formed in 64-bit).  ``q_src`` (float32 [T, >= q_off + H (D + R)]): the
    queries come from this array instead of ``proj`` (a product of their own).  ``rot_block``: q_rot is [H, rows, 64] of the
    cache's type instead, zeros behind the R-th column."""
    if q_src is None:
        q_src = proj
    assert q_src.dtype == torch.float32 and q_src.stride(1) == 1 and q_src.shape[0] == proj.shape[0]
    assert proj.dtype == torch.float32 and proj.stride(1) == 1 and cache.is_contiguous() and cache.shape[-1] == C + R
    assert cache.shape[1] == 1 and q_plain.dtype == cache.dtype and q_plain.is_contiguous()
    assert q_rot.dtype == (cache.dtype if rot_block else torch.float32)
    rows = q_plain.shape[1]
    assert tuple(q_plain.shape) == (H, rows, D) and tuple(q_rot.shape) == (H, rows, 64 if rot_block else R) and q_rot.is_contiguous()
    assert freq is None or (freq.dtype == torch.float64 and freq.is_contiguous())
    rot = 0 if freq is None else 2 * freq.numel()
    _check(lib().infero_latent_prepare_from(
        _ptr(proj), c_int(proj.stride(0)), _ptr(q_src), c_int(q_src.stride(0)), c_int(q_off), c_int(kv_off), _ptr(_f32(norm_w, "norm_w")), c_float(eps),
        _ptr(freq), c_int(rot), c_int(1 if pairing == "adjacent" else 0), c_float(amp),
        _ptr(_i32(positions, "positions")), _ptr(_i32(tok_entry, "tok_entry")), _ptr(_i32(block_table, "block_table")),
        c_int(block_table.shape[1]), c_int(page_size), _ptr(cache), c_int(_dt(cache)), c_int(1 if write_cache else 0),
        _ptr(q_plain), _ptr(None if rot_block else q_rot), _ptr(q_rot if rot_block else None), c_longlong(rows), c_int(n_tokens), c_int(H), c_int(D), c_int(R), c_int(C), _stream()))


def few_ok(ctx, cache: torch.Tensor, n_tokens: int, D: int, R: int, C: int, w_k: torch.Tensor, w_v: torch.Tensor) -> bool:
    """Do the first ``n_tokens`` tokens go through ``query_few`` and ``result_few``?  Up to 16 of them, each its request's only one,
    in bf16, in sizes those and the tensor-core attention take, with up-projections that start on 16 bytes."""
    from . import latent_mma
    return (n_tokens <= 16 and cache.dtype == w_k.dtype == w_v.dtype == torch.bfloat16 and D % 32 == 0 and D <= 128 and latent_mma.ENABLED
            and w_k.data_ptr() % 16 == 0 and w_v.data_ptr() % 16 == 0
            and getattr(ctx, "h_q_len", None) is not None and len(ctx.h_q_len) >= n_tokens and all(int(n) == 1 for n in ctx.h_q_len[:n_tokens])
            and latent_mma.supported(C, R))


def query_few(proj, q_off, kv_off, norm_w, eps, freq, pairing, amp, positions, tok_entry, block_table, cache, page_size, w_k, q_lat, q_rot,
              n_tokens, H, D, R, C, write_cache=True, q_src=None) -> None:
    """``prepare`` and the product of the plain query parts with Wuk^T (``w_k`` [H, C, D]) in one launch: q_lat float32 [H, rows, C],
    q_rot float32 [H, rows, R]."""
    if q_src is None:
        q_src = proj
    assert proj.dtype == q_src.dtype == torch.float32 and proj.stride(1) == q_src.stride(1) == 1 and cache.is_contiguous()
    assert cache.dtype == w_k.dtype == torch.bfloat16 and tuple(w_k.shape) == (H, C, D) and w_k.is_contiguous() and cache.shape[-1] == C + R
    rows = q_lat.shape[1]
    assert tuple(q_lat.shape) == (H, rows, C) and tuple(q_rot.shape) == (H, rows, R) and q_lat.is_contiguous() and q_rot.is_contiguous()
    assert q_lat.dtype == q_rot.dtype == torch.float32 and (freq is None or (freq.dtype == torch.float64 and freq.is_contiguous()))
    _check(lib().infero_latent_query_few(
        _ptr(proj), c_int(proj.stride(0)), _ptr(q_src), c_int(q_src.stride(0)), c_int(q_off), c_int(kv_off), _ptr(_f32(norm_w, "norm_w")),
        c_float(eps), _ptr(freq), c_int(0 if freq is None else 2 * freq.numel()), c_int(1 if pairing == "adjacent" else 0), c_float(amp),
        _ptr(_i32(positions, "positions")), _ptr(_i32(tok_entry, "tok_entry")), _ptr(_i32(block_table, "block_table")),
        c_int(block_table.shape[1]), c_int(page_size), _ptr(cache), c_int(1 if write_cache else 0), _ptr(w_k), _ptr(q_lat), _ptr(q_rot),
        c_longlong(rows), c_int(n_tokens), c_int(H), c_int(D), c_int(R), c_int(C), _stream()))


def result_few(o_lat, splits: int, part_o, part_ml, sinks_log2, w_v, gate, out, n_tokens: int, H: int, D: int, C: int, V: int) -> None:
    """The attention's ranges merged (``splits`` > 1; else o_lat [H, rows, C] as it is), the product with Wuv (``w_v`` [H, V, C]) and the
    gate (float32 [tokens, H] or None) in one launch; out [tokens, H V] bf16."""
    assert w_v.dtype == out.dtype == torch.bfloat16 and tuple(w_v.shape) == (H, V, C) and w_v.is_contiguous()
    assert out.shape[1] == H * V and out.stride(1) == 1 and (gate is None or (gate.dtype == torch.float32 and gate.stride(1) == 1))
    _check(lib().infero_latent_result_few(_ptr(o_lat), c_longlong(o_lat.shape[1]), _ptr(part_o), _ptr(part_ml), c_int(splits), _ptr(sinks_log2),
                                          _ptr(w_v), _ptr(gate), c_int(gate.stride(0) if gate is not None else 0), _ptr(out),
                                          c_int(out.stride(0)), c_int(n_tokens), c_int(H), c_int(D), c_int(C), c_int(V), _stream()))


def grouped_ok(a: torch.Tensor, w: torch.Tensor) -> bool:
    """Can the tcgen05 grouped product take a [H, rows, K] x w [H, N, K]?"""
    from .tc_gemm import supported
    return (a.dtype == torch.bfloat16 and a.shape[1] % TILE == 0 and supported(a.view(-1, a.shape[2]), w.view(-1, w.shape[2])))


_TILE_HEAD = {}


def _tile_heads(H: int, rows: int, device) -> torch.Tensor:
    """tile -> head for [H, rows] in 128-row tiles, followed by the number of rows in use."""
    key = (H, rows, str(device))
    t = _TILE_HEAD.get(key)
    if t is None:
        per = rows // TILE
        # (made by device operations: a step that is being captured into a graph may meet a new size)
        t = torch.cat([torch.arange(H * per, dtype=torch.int32, device=device) // per,
                       torch.full((1,), H * rows, dtype=torch.int32, device=device)])
        if len(_TILE_HEAD) > 256:
            _TILE_HEAD.clear()
        _TILE_HEAD[key] = t
    return t


def per_head_product(a: torch.Tensor, w: torch.Tensor, out: torch.Tensor, n_rows: int) -> None:
    """out[n] = a[n] @ w[n]^T for every head n; a [H, rows, K], w [H, N, K], out float32 [H, rows, N].  The tcgen05
    grouped product where it applies (bf16, whole tiles), else one product per head on the first ``n_rows`` rows."""
    H, rows, Kd = a.shape
    N = w.shape[1]
    assert out.dtype == torch.float32 and tuple(out.shape) == (H, rows, N) and w.is_contiguous() and a.is_contiguous()
    if grouped_ok(a, w):
        from .tc_gemm import sm_count
        _check(lib().infero_gemm_tc_grouped(_ptr(a), _ptr(w), _ptr(out), c_int(0), c_int(H * rows), c_int(N), c_int(Kd),
                                            c_int(Kd), c_int(N), _ptr(_tile_heads(H, rows, a.device)), c_int(H),
                                            c_int(sm_count(a.device)), *_act_args(None), _stream()))
        return
    for n in range(H):
        gemm_tiled(a[n, :n_rows], w[n], None, out[n, :n_rows])


def attention(ctx, q_lat: torch.Tensor, q_rot: torch.Tensor, out: torch.Tensor, kv, table, n_tokens: int, H: int, C: int,
              R: int, scale: float, window: Optional[int] = None, sinks: Optional[torch.Tensor] = None,
              sinks_log2: Optional[torch.Tensor] = None, singles_only: bool = False) -> None:
    """Causal softmax attention of every token over its request's cached latent rows: q_lat float32 [H, rows, C],
    q_rot float32 [H, rows, R], out [H, rows, C] of the cache's type.  ``window``: a token sees that many keys up to its own.
    ``sinks`` float32 [H] (``sinks_log2``: times log2 e, made here when absent): one more term exp(sinks[h]) in head h's sum,
    without a value.  ``singles_only``: only the requests in front that bring one token each (``n_tokens`` of them)."""
    assert sinks is None or (sinks.dtype == torch.float32 and sinks.is_contiguous() and sinks.numel() == H)
    cache = kv.k
    rows = q_lat.shape[1]
    assert q_lat.dtype == torch.float32 and q_rot.dtype == torch.float32 and q_lat.is_contiguous() and q_rot.is_contiguous()
    assert out.dtype == cache.dtype and out.is_contiguous() and tuple(out.shape) == (H, rows, C) and cache.is_contiguous()
    from . import latent_mma
    if latent_mma.run(ctx, q_lat, q_rot, out, kv, table, n_tokens, H, C, R, scale, window, sinks, sinks_log2,
                      singles_only):
        return
    _check(lib().infero_latent_attention_generic(
        _ptr(q_lat), _ptr(q_rot), c_longlong(rows), _ptr(out), _ptr(cache), c_int(_dt(cache)),
        _ptr(_i32(table, "block_table")), c_int(table.shape[1]), _ptr(_i32(ctx.tok_entry, "tok_entry")),
        _ptr(_i32(ctx.positions, "positions")), c_int(0), c_int(n_tokens), c_int(H), c_int(C), c_int(R),
        c_int(kv.page_size), c_float(scale), c_int(window or 0), _ptr(sinks), _stream()))


def finish(val: torch.Tensor, gate: Optional[torch.Tensor], out: torch.Tensor, n_tokens: int, H: int, V: int) -> None:
    """out[t, n * V + v] = val[n, t, v] * sigmoid(gate[t, n]); val float32 [H, rows, V], gate float32 [T, H] (a column
    slice is fine) or None."""
    assert val.dtype == torch.float32 and val.is_contiguous() and out.stride(1) == 1 and out.shape[1] == H * V
    assert gate is None or (gate.dtype == torch.float32 and gate.stride(1) == 1 and gate.shape[1] == H)
    _check(lib().infero_latent_finish(_ptr(val), c_longlong(val.shape[1]), _ptr(gate), c_int(gate.stride(0) if gate is not None else 0),
                                      _ptr(out), c_int(out.stride(0)), c_int(_dt(out)), c_int(n_tokens), c_int(H), c_int(V),
                                      _stream()))
