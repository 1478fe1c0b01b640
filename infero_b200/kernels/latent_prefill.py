"""Latent attention of prompt portions with their keys and values written out (``csrc/latent_prefill_tc.cu``).

``plan`` says whether a step's portions go this way; the leading run of single-token requests never does."""
from __future__ import annotations

from ctypes import c_float, c_int
from typing import NamedTuple, Optional

import torch

from . import _check, _i32, _ptr, _stream, lib

KTILE, QROWS, BLOCK = 64, 128, 64
MIN_TOKENS = 16            # of all portions together
MAX_KEYS_PER_TOKEN = 4
launches = {"steps": 0}    # (tests look at it)


class Plan(NamedTuple):
    first_entry: int        # = the first token: the requests in front bring one each
    key_tiles: int
    query_tiles: int


def supported(D: int, V: int, R: int, C: int) -> bool:
    return (D in (64, 128) and V == D and 0 <= R <= BLOCK and R % 8 == 0 and C >= 2 * D and C % 8 == 0)


def values_fit(up_v: torch.Tensor, norm_w: torch.Tensor, C: int) -> bool:
    """Can no value of these weights leave the range of IEEE halves?  A latent row is norm_w times a row of 2-norm sqrt(C) at most
    (rounded to bf16: 1 + 2^-8), a value its product with a row of Wuv."""
    rows = (up_v.float() * norm_w.float()).norm(dim=1)
    return bool(float(rows.max()) * C ** 0.5 * (1 + 2.0 ** -8) < 65504.0)


def plan(ctx, dtype, H: int, D: int, V: int, R: int, C: int, window: Optional[int]) -> Optional[Plan]:
    """None, or how the portions behind the leading single tokens are cut.  Writing keys and values out costs 2 C (D + V)
    a key and head and saves about 2 (2 C - D - V) a (query, key) pair, so not a short portion behind a long cached prefix.
    Measured as whole prompts of four layers of 16 heads of 128 + 64, latent 512: 8 tokens 1.30 ms through the latents, 1.17 written out (the
    host's launches bind both), 512: 1.32 and 1.10, 1,024: 1.79 and 1.16, 2,048: 3.75 and 1.71; no length was slower.  MIN_TOKENS
    keeps the few tokens that fill no tile on the latent rows.  MAX_KEYS_PER_TOKEN also bounds
    the memory: at most 16 D bytes a token and head, where the latent queries and results take 6 C + 4 V (C >= 2 D)."""
    if dtype != torch.bfloat16 or getattr(ctx, "h_q_len", None) is None or not supported(D, V, R, C):
        return None
    E, n = ctx.n_entries, 0
    while n < E and ctx.h_q_len[n] == 1:
        n += 1
    tokens = keys = tiles = 0
    for e in range(n, E):
        q, p0 = int(ctx.h_q_len[e]), int(ctx.h_pos0[e])
        start = max(0, p0 - window + 1) // KTILE * KTILE if window else 0
        tokens += q
        keys += -(-(p0 + q - start) // KTILE)
        tiles += -(-q // QROWS)
    if tokens < MIN_TOKENS or keys * KTILE > MAX_KEYS_PER_TOKEN * tokens + KTILE * (E - n):
        return None
    return Plan(n, keys, tiles)


def run(ctx, p: Plan, q: torch.Tensor, q_rot: torch.Tensor, kv, table: torch.Tensor, w_kv: torch.Tensor, gate: Optional[torch.Tensor],
        out: torch.Tensor, H: int, D: int, R: int, C: int, scale: float, window: Optional[int], sinks_log2: Optional[torch.Tensor]) -> None:
    """out[t, n D + v] of the portions' tokens.  q [H, rows, D] and q_rot [H, rows, 64] (bf16) of these tokens; w_kv [2 H D, C]: the
    heads' key projections, then their value projections; gate float32 [tokens, H] (a column slice is fine) or None; out
    [tokens, H D] bf16."""
    from . import tc_gemm
    launches["steps"] += 1
    cache, dev, rows = kv.k, q.device, q.shape[1]
    assert cache.is_contiguous() and cache.shape[1] == 1 and cache.shape[-1] == C + R and w_kv.shape == (2 * H * D, C) and w_kv.is_contiguous()
    assert q.dtype == q_rot.dtype == out.dtype == cache.dtype == torch.bfloat16 and q.is_contiguous() and q_rot.is_contiguous()
    assert tuple(q.shape) == (H, rows, D) and tuple(q_rot.shape) == (H, rows, BLOCK) and out.shape[1] == H * D and out.stride(1) == 1
    assert gate is None or (gate.dtype == torch.float32 and gate.stride(1) == 1 and gate.shape == (out.shape[0], H))
    keys = p.key_tiles * KTILE
    lat = torch.empty((keys, C), dtype=torch.bfloat16, device=dev)
    k_rot = torch.empty((keys, BLOCK), dtype=torch.bfloat16, device=dev)
    entry = tuple(_ptr(_i32(t, n)) for t, n in ((ctx.entry_q_start, "entry_q_start"), (ctx.entry_q_len, "entry_q_len"), (ctx.entry_pos0, "entry_pos0")))
    where = (c_int(p.first_entry), c_int(ctx.n_entries))
    _check(lib().infero_latent_gather(_ptr(cache), _ptr(_i32(table, "block_table")), c_int(table.shape[1]), c_int(kv.page_size), entry[1], entry[2],
                                      *where, c_int(p.key_tiles), c_int(window or 0), c_int(C), c_int(R), _ptr(lat), _ptr(k_rot), _stream()))
    wide = torch.empty((keys, 2 * H * D), dtype=torch.bfloat16, device=dev)
    tc_gemm.gemm_halves(lat, w_kv, wide)                 # keys bf16, values halves
    _check(lib().infero_latent_prefill_tc(_ptr(q), _ptr(q_rot), c_int(rows), _ptr(wide), _ptr(k_rot), c_int(p.key_tiles), _ptr(out),
                                          c_int(out.stride(0)), _ptr(gate), c_int(gate.stride(0) if gate is not None else 0), *entry, *where,
                                          c_int(p.first_entry), c_int(p.query_tiles), c_int(H), c_int(D), c_int(D), c_int(R), c_int(C),
                                          c_float(scale), c_int(window or 0), _ptr(sinks_log2), _stream()))
