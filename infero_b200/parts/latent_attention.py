"""Latent attention over the paged cache: one small cached row per token makes the keys and values of all heads."""
from __future__ import annotations

from typing import Dict, List, Optional

import torch

from ..config.spec import MixerSpec
from ..registry import part_class
from .base import KvCacheSpec, Mixer, TensorDecl
from .linear import Linear


class LatentAttention(Mixer):
    """H heads; a query head is [D plain | R rotated] wide.  The input product also gives C + R numbers per token:
    the first C, RMS-normed with a weight, are the latent c, the last R a rotated key part shared by all heads.
    Head n's key is [Wuk_n c | rotated part] and its value Wuv_n c (V wide); causal softmax of q . k * scale; with
    ``out_gate`` head n's result is multiplied by sigmoid((Wg h)_n); heads side by side, output product.

    The cache holds the row [c | rotated part] only (one kv head of width C + R, no separate values), and the
    up-projections are carried to the query side: (Wuk_n^T q_plain,n) . c gives the same score as q_plain,n . (Wuk_n c),
    and Wuv_n applied to the softmax-weighted sum of latents the same result as the sum of values.  A step is

        stacked product [q; down; gate]  ->  prepare (norm, rotation, cache append, head-major queries)
        ->  per-head product with Wuk^T  ->  attention over latent rows  ->  per-head product with Wuv
        ->  finish (gate, heads side by side)  ->  output product.

    In bf16 steps, prompt portions of many tokens have the keys and values they see written out per head instead
    (``kernels/latent_prefill.py``); the requests in front that bring one token each keep to the latent rows.

    Rotation: the position part's table (with any stretching of the frequencies and its amplitude) and pairing; R may
    be 0 (no rotated part: positions enter through the causal mask alone).

    ``q_latent_dim`` = Q > 0: the queries have a latent of their own.  The stacked product gives [dq | down (| gate)], the
    first Q columns are RMS-normed with a weight (32-bit) and a second product with Wuq [H (D + R), Q] gives the queries.

    ``window``: a token sees that many keys up to its own; ``sink_per_head``: a learned sink in every head's softmax."""

    def __init__(self, spec: MixerSpec, prefix: str):
        self.spec, self.prefix = spec, prefix
        self.H, self.D, self.R, self.V, self.C = spec.num_heads, spec.head_dim, spec.rot_dim, spec.v_dim, spec.latent_dim
        self.Q = int(spec.q_latent_dim)
        if min(self.H, self.D, self.V, self.C) <= 0 or self.R < 0 or self.Q < 0:
            raise ValueError("latent attention needs heads, head_dim, value_dim and latent_dim")
        self.names = spec.tensor_names()
        self.rope, self.pairing, self.amp = None, "half", 1.0
        if spec.position is not None and spec.position.rotary_dim > 0:
            if spec.position.rotary_dim > self.R:
                raise ValueError(f"{spec.position.rotary_dim} rotated coordinates in a part of {self.R}")
            self.rope = part_class("position", spec.position.kind)(spec.position)
            if not hasattr(self.rope, "inv_freq64"):
                raise ValueError(f"latent attention needs a rotary table; position kind '{spec.position.kind}' has none")
            self.pairing = getattr(self.rope, "pairing", "half")
            self.amp = float(getattr(self.rope, "amplitude", 1.0))
        self.qkv: Linear = None
        self.out: Linear = None

    def _n(self, role: str) -> str:
        leaf = self.names[role]
        return f"{self.prefix}.{leaf}" + ("" if role in ("latent_norm", "q_norm", "sink") else self.spec.weight_suffix)

    def cache_spec(self) -> Optional[KvCacheSpec]:
        return KvCacheSpec(1, self.C + self.R, self.spec.window, v_head_dim=0)        # the values are the first C columns of a key row

    def declare(self) -> List[TensorDecl]:
        d, H, D, R, V, C = self.spec.hidden, self.H, self.D, self.R, self.V, self.C
        if self.Q:
            q = [TensorDecl(self._n("q_down"), (self.Q, d)), TensorDecl(self._n("q_norm"), (self.Q,), role="norm", init="ones"),
                 TensorDecl(self._n("q_up"), (H * (D + R), self.Q))]
        else:
            q = [TensorDecl(self._n("q"), (H * (D + R), d))]
        out = q + [TensorDecl(self._n("down"), (C + R, d)),
               TensorDecl(self._n("latent_norm"), (C,), role="norm", init="ones"),
               TensorDecl(self._n("up_k"), (H * D, C)), TensorDecl(self._n("up_v"), (H * V, C)),
               TensorDecl(self._n("o"), (d, H * V))]
        if self.spec.out_gate:
            out.append(TensorDecl(self._n("gate"), (H, d)))
        if self.spec.sink_per_head:
            out.append(TensorDecl(self._n("sink"), (H,), role="bias"))
        return out

    def bind(self, tensors: Dict[str, torch.Tensor]) -> None:
        from ..kernels import latent_prefill as P
        H, D, R, V, C = self.H, self.D, self.R, self.V, self.C
        rows = [tensors[self._n("q_down" if self.Q else "q")], tensors[self._n("down")]]
        if self.spec.out_gate:
            rows.append(tensors[self._n("gate")])
        if len({t.dtype for t in rows}) > 1:
            rows = [t.float() for t in rows]
        self.qkv = Linear(torch.cat(rows, dim=0), None, f"{self.prefix}.q_down")
        nq = self.Q or H * (D + R)
        self.q_off, self.kv_off, self.gate_off = 0, nq, nq + C + R
        self.q_norm = self.q_up = None
        if self.Q:
            self.q_norm = tensors[self._n("q_norm")].float().contiguous()
            self.q_up = Linear(tensors[self._n("q_up")], None, self._n("q_up"))
        self.latent_norm = tensors[self._n("latent_norm")].float().contiguous()
        self.sinks = self.sinks_log2 = None
        if self.spec.sink_per_head:
            self.sinks = tensors[self._n("sink")].float().contiguous()
            self.sinks_log2 = (self.sinks * 1.4426950408889634).contiguous()
        # [H, C, D]: head n's rows of Wuk, transposed, so that the product with the plain query parts is a @ w^T
        self.up_k_t = tensors[self._n("up_k")].view(H, D, C).transpose(1, 2).contiguous()
        # where prompts are written out: both up-projections as one matrix
        up_k, up_v = tensors[self._n("up_k")], tensors[self._n("up_v")]
        out = up_k.dtype == up_v.dtype == torch.bfloat16 and P.supported(D, V, R, C) and P.values_fit(up_v, self.latent_norm, C)
        self.kv_up = torch.cat([up_k, up_v]) if out else None
        self.up_v = (up_v if self.kv_up is None else self.kv_up[H * D:]).view(H, V, C).contiguous()
        self.out = Linear(tensors[self._n("o")], None, self._n("o"))

    def forward(self, ctx, h, slot):
        from ..kernels import latent_attention as A
        from ..kernels import latent_prefill as P
        H, D, R, V, C = self.H, self.D, self.R, self.V, self.C
        T, dev = h.shape[0], h.device
        proj = self.qkv.forward(h, out_dtype=torch.float32)             # [T, H (D + R) + C + R (+ H)], never rounded
        kv = ctx.kv_cache(slot.cache)
        table = ctx.block_table(kv.group)
        q_src = None
        if self.Q:
            from ..kernels import layer_ops as L
            cq = torch.empty((T, self.Q), dtype=h.dtype, device=dev)
            L.gated_group_norm(proj[:, :self.Q], None, self.q_norm, self.spec.norm_eps, 1, cq)
            q_src = self.q_up.forward(cq, out_dtype=torch.float32)
        attn = torch.empty((T, H * V), dtype=h.dtype, device=dev)
        plan = P.step_plan(ctx, h.dtype, H, D, V, R, C, self.spec.window) if self.kv_up is not None else None
        singles = T if plan is None else plan.first_entry
        if singles:
            self._through_latents(ctx, A, proj, q_src, kv, table, slot, attn, singles, plan is not None)
        if plan is not None:
            self._written_out(ctx, A, P, plan, proj, q_src, kv, table, slot, attn)
        return self.out.forward(attn, defer=True, residual=True)

    def _prepare(self, ctx, A, proj, q_src, kv, table, slot, t0, t1, rows, rot_block):
        """Norm, rotation and cache append of tokens t0 .. t1 - 1; their queries, head-major."""
        H, D, R, C = self.H, self.D, self.R, self.C
        n, positions, tok_entry = t1 - t0, ctx.positions, ctx.tok_entry
        if n < proj.shape[0]:                           # (steps that the host's work bounds come whole: no views of everything)
            proj, positions, tok_entry = proj[t0:t1], positions[t0:t1], tok_entry[t0:t1]
            q_src = None if q_src is None else q_src[t0:t1]
        q_plain = torch.empty((H, rows, D), dtype=kv.k.dtype, device=proj.device)
        q_rot = torch.empty((H, rows, 64 if rot_block else R), dtype=kv.k.dtype if rot_block else torch.float32, device=proj.device)
        freq = self.rope.inv_freq64(proj.device) if self.rope is not None else None
        A.prepare(proj, self.q_off, self.kv_off, self.latent_norm, self.spec.norm_eps, freq, self.pairing, self.amp,
                  positions, tok_entry, table, kv.k, kv.page_size, q_plain, q_rot, n, H, D, R, C,
                  write_cache=slot.write_cache, q_src=q_src, rot_block=rot_block)
        return q_plain, q_rot

    def _gate(self, proj, t0, t1):
        if not self.spec.out_gate:
            return None
        gate = proj[:, self.gate_off:self.gate_off + self.H]
        return gate if t1 - t0 == proj.shape[0] else gate[t0:t1]

    def _through_latents(self, ctx, A, proj, q_src, kv, table, slot, attn, n, singles_only):
        """Tokens 0 .. n - 1 against the latent rows where they lie, the up-projections carried to the query side."""
        H, D, R, V, C = self.H, self.D, self.R, self.V, self.C
        dt, dev = kv.k.dtype, proj.device
        if A.few_ok(ctx, kv.k, n, D, R, C, self.up_k_t, self.up_v):
            from ..kernels import latent_mma
            q_lat = torch.empty((H, n, C), dtype=torch.float32, device=dev)
            q_rot = torch.empty((H, n, R), dtype=torch.float32, device=dev)
            freq = self.rope.inv_freq64(dev) if self.rope is not None else None
            A.query_few(proj[:n], self.q_off, self.kv_off, self.latent_norm, self.spec.norm_eps, freq, self.pairing, self.amp,
                        ctx.positions[:n], ctx.tok_entry[:n], table, kv.k, kv.page_size, self.up_k_t, q_lat, q_rot, n, H, D, R, C,
                        write_cache=slot.write_cache, q_src=None if q_src is None else q_src[:n])
            o_lat = torch.empty((H, n, C), dtype=dt, device=dev)
            parts = latent_mma.single(ctx, q_lat, q_rot, o_lat, kv, table, n, H, C, R, self.spec.scale, self.spec.window, self.sinks_log2,
                                      merge=False)
            A.result_few(o_lat, *parts, self.sinks_log2, self.up_v, self._gate(proj, 0, n), attn[:n], n, H, D, C, V)
            return
        # whole 128-row tiles per head where the grouped tensor-core product runs
        rows = -(-n // A.TILE) * A.TILE if (dt == torch.bfloat16 and D % 8 == 0 and C % 8 == 0) else n
        q_plain, q_rot = self._prepare(ctx, A, proj, q_src, kv, table, slot, 0, n, rows, False)
        q_lat = torch.empty((H, rows, C), dtype=torch.float32, device=dev)
        A.per_head_product(q_plain, self.up_k_t, q_lat, n)
        o_lat = torch.empty((H, rows, C), dtype=dt, device=dev)
        A.attention(ctx, q_lat, q_rot, o_lat, kv, table, n, H, C, R, self.spec.scale, self.spec.window, self.sinks, self.sinks_log2,
                    singles_only=singles_only)
        val = torch.empty((H, rows, V), dtype=torch.float32, device=dev)
        A.per_head_product(o_lat, self.up_v, val, n)
        A.finish(val, self._gate(proj, 0, n), attn if n == attn.shape[0] else attn[:n], n, H, V)

    def _written_out(self, ctx, A, P, plan, proj, q_src, kv, table, slot, attn):
        """The portions behind the single tokens, their visible keys and values written out per head."""
        t0, T = plan.first_entry, proj.shape[0]
        q_plain, q_rot = self._prepare(ctx, A, proj, q_src, kv, table, slot, t0, T, T - t0, True)
        P.run(ctx, plan, q_plain, q_rot, kv, table, self.kv_up, self._gate(proj, t0, T), attn[t0:], self.H, self.D, self.R, self.C,
              self.spec.scale, self.spec.window, self.sinks_log2)
