"""Attention of the resident decode kernel over keys that many blocks share, against 64 bits: segments of more slots than the ring
has, several pieces and tokens a block, pairs that begin inside a block.  Values are zero but for the keys on both sides of every
edge between two blocks, which share the weight: a slice that is lost, taken twice or read too early changes the result by more
than a tenth."""
import ctypes

import pytest
import torch

import plain_qwen2 as P
from test_resident_gpu import _config

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SLICE = 16


def _edges(lengths, kv, blocks):
    """Per token and kv head the keys at the edges of the blocks' pieces where every block has an equal share of all slices."""
    slices = [n // SLICE + 1 for n in lengths]
    per = -(-sum(slices) * kv // blocks)
    out, off = [], 0
    for n, s in zip(lengths, slices):
        heads = []
        for h in range(kv):
            first = [i * SLICE for i in range(1, s) if (off + h * s + i) % per == 0]
            heads.append(sorted({k for f in first for k in (f - 1, f)} | {0, n - 1}))
        out.append(heads)
        off += s * kv
    return out, per


def _row(cfg, w, token, n, k_cache, v_cache):
    """Logits of the token at position n in 64 bits; k_cache, v_cache: per layer [kv, n, dim]."""
    H, G, D = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    pos, eps = torch.tensor([n], device=DEV), cfg["rms_norm_eps"]
    x = w["model.embed_tokens.weight"][token].double()[None]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        m = {name: w[p + name].double() for name in ("input_layernorm.weight", "post_attention_layernorm.weight", "self_attn.o_proj.weight",
                                                     "mlp.gate_proj.weight", "mlp.up_proj.weight", "mlp.down_proj.weight")}
        h = P.rms_norm(x, m["input_layernorm.weight"], eps)
        q, k, v = (h @ w[p + f"self_attn.{c}_proj.weight"].double().T + w[p + f"self_attn.{c}_proj.bias"].double() for c in "qkv")
        q = P.rope_neox(q.view(1, H, D), pos, cfg["rope_theta"], D)[0].view(G, H // G, D)
        k = P.rope_neox(k.view(1, G, D), pos, cfg["rope_theta"], D)[0].view(G, 1, D)
        keys, values = torch.cat([k_cache[i].double(), k], 1), torch.cat([v_cache[i].double(), v.view(G, 1, D)], 1)
        a = torch.softmax(q @ keys.transpose(1, 2) * D ** -0.5, -1) @ values
        x = x + a.reshape(1, H * D) @ m["self_attn.o_proj.weight"].T
        h = P.rms_norm(x, m["post_attention_layernorm.weight"], eps)
        x = x + P.swiglu_mlp(h, m["mlp.gate_proj.weight"], m["mlp.up_proj.weight"], m["mlp.down_proj.weight"])
    return (P.rms_norm(x, w["model.norm.weight"].double(), eps) @ w["lm_head.weight"].double().T)[0]


@pytest.mark.parametrize("shape,lengths", [
    (dict(hidden=640, heads=6, kv=6, dim=64, ff=2752), [15000]),           # 39 slices a block, three a slot: 14 slots
    (dict(hidden=640, heads=6, kv=6, dim=64, ff=2752), [9001, 40]),
    (dict(hidden=640, heads=12, kv=6, dim=128, ff=1344), [5000]),          # 13 slices a block, a slot each
    (dict(hidden=640, heads=12, kv=6, dim=128, ff=1344), [700, 9001]),
    (dict(hidden=896, heads=14, kv=2, dim=64, ff=4864), [36000]),           # 31 slices a block, 11 slots
], ids=["64", "64-two", "128", "128-two", "two-kv-heads"])
def test_keys_at_every_edge_between_blocks(shape, lengths):
    from infero_b200 import kernels as K
    from infero_b200.config import EngineConfig
    from infero_b200.engine import ModelRunner, StepEntry
    from infero_b200.models.decoder import DecoderModel
    from infero_b200.registry import resolve_architecture
    from infero_b200.weights import random_tensors
    cfg = dict(_config(**shape, layers=2), max_position_embeddings=65536)
    arch = resolve_architecture(cfg)
    model = DecoderModel(arch.to_spec(arch.read_config(cfg)))
    w = random_tensors(model.declare(), 3, torch.bfloat16, 0.02, 0.1, device=DEV)
    model.bind(dict(w))
    blocks = torch.cuda.get_device_properties(0).multi_processor_count
    edges, per = _edges(lengths, shape["kv"], blocks)
    assert per > 7
    runner = ModelRunner(model, EngineConfig(dtype="bfloat16", num_pages=sum(n // 16 + 2 for n in lengths), max_seqs=len(lengths), ctx=max(lengths) + 3,
                                             max_batch_tokens=64, max_logit_rows=8), DEV)
    g = torch.Generator(device=DEV).manual_seed(5)
    caches = []
    for i, n in enumerate(lengths):
        rc = runner.open(i)
        runner.manager.reserve(rc, n)
        runner.manager.commit(rc, n)
        table = torch.tensor(rc.tables[0], device=DEV)
        per_layer = []
        for layer in range(2):
            kv = runner.storage.layer_kv(layer)
            k = (torch.randn((shape["kv"], n, shape["dim"]), generator=g, device=DEV) * 0.5).bfloat16()
            v = torch.zeros_like(k)
            for h, keys in enumerate(edges[i]):
                v[h, keys] = (torch.randn((len(keys), shape["dim"]), generator=g, device=DEV) * n / len(keys) ** 0.5).bfloat16()
            at = torch.arange(n, device=DEV)
            for cache, rows in ((kv.k, k), (kv.v, v)):
                cache[table[at // 16], :, at % 16] = rows.transpose(0, 1)
            per_layer.append((k, v))
        caches.append(per_layer)
    toks = torch.randint(512, (len(lengths),), generator=torch.Generator().manual_seed(7)).tolist()
    want = torch.stack([_row(cfg, w, t, n, [c[0] for c in kv], [c[1] for c in kv]) for t, n, kv in zip(toks, lengths, caches)])

    def steps(resident):
        K.lib().infero_block_set_resident(ctypes.c_int(resident))
        runner.drop_graphs()
        out = []
        try:
            before = K.launch_count()
            for _ in range(3):                                          # eager, captured, replayed
                out.append(runner.step([StepEntry(i, [t], [0]) for i, t in enumerate(toks)]).clone())
                launches = K.launch_count() - before if len(out) == 1 else launches
                for i, n in enumerate(lengths):
                    runner.truncate(i, n)
        finally:
            K.lib().infero_block_set_resident(ctypes.c_int(2))
        if resident:                                                    # (the launches cut the keys by a captured step's bound)
            assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
        return out[0].double(), launches

    resident, few = steps(1)
    plain, many = steps(0)
    assert few < many, "the resident kernel was meant to run this step"
    # About ten bf16 roundings a layer (normed rows, q, k, v, weights of the softmax, activations), 2^-9 at most and half of that in the
    # root mean square, each of the whole row; three times what they add up to at random.
    bound = 3 * (2 * 10) ** 0.5 * 2.0 ** -10
    for name, got in (("resident", resident), ("launches", plain)):
        for a, b in zip(want, got):
            assert float((a - b).norm() / a.norm()) <= bound, name
    from infero_b200.kernels import tc_gemm
    assert tc_gemm.error_flag() == 0
