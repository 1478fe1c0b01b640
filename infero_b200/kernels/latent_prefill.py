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
MIN_BESIDE = 1 << 31       # multiply-adds that writing out has to save where single tokens stand in front
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
    lens, starts = [int(n) for n in ctx.h_q_len], [int(p) for p in ctx.h_pos0]
    n = 0
    while n < len(lens) and lens[n] == 1:
        n += 1
    tokens = sum(lens[n:])
    if tokens < MIN_TOKENS:
        return None
    keys = tiles = 0
    for q, p0 in zip(lens[n:], starts[n:]):
        start = max(0, p0 - window + 1) // KTILE * KTILE if window else 0
        keys += -(-(p0 + q - start) // KTILE)
        tiles += -(-q // QROWS)
    if keys * KTILE > MAX_KEYS_PER_TOKEN * tokens + KTILE * (len(lens) - n):
        return None
    return Plan(n, keys, tiles)


def worth_it(ctx, p: Plan, H: int, D: int, V: int, C: int, window: Optional[int]) -> bool:
    """Beside single tokens the portions' four launches come on top of the single tokens' own three to six, where everything
    through the latent rows is seven together; such steps are never captured, so the host's launches bound them, and writing out has to
    save more than these cost.  Four layers, through the latent rows and written out: 16 heads of 128, latent 512 (the line lies at 591
    prompt tokens): 17 single tokens and 100 prompt tokens 1.61 and 1.92 ms, 17 + 400 1.64 and 1.85, 17 + 700 2.06 and 1.92, 2 + 400 1.55 and
    1.58, 64 + 1,500 3.38 and 2.25; 8 of 64, latent 256 (1,182): 64 + 24 1.72 and 2.01, 17 + 700 1.45 and 1.73, 17 + 1,500 1.92 and 1.78."""
    if p.first_entry == 0:
        return True
    pairs = 0
    for q, p0 in zip(ctx.h_q_len[p.first_entry:], ctx.h_pos0[p.first_entry:]):
        q, p0 = int(q), int(p0)
        pairs += q * min(p0 + (q + 1) // 2, window or p0 + q)
    return H * (2 * C - D - V) * pairs >= MIN_BESIDE


def step_plan(ctx, dtype, H: int, D: int, V: int, R: int, C: int, window: Optional[int]) -> Optional[Plan]:
    """The plan that the step's layers of these sizes go by, worked out by the first of them."""
    memo = getattr(ctx, "_latent_plans", None)
    if memo is None:
        memo = {}
        try:
            ctx._latent_plans = memo
        except AttributeError:          # a context that takes no new attributes
            pass
    key = (dtype, H, D, V, R, C, window)
    if key not in memo:
        p = plan(ctx, *key)
        memo[key] = p if p is not None and worth_it(ctx, p, H, D, V, C, window) else None
    return memo[key]


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
