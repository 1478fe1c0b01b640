"""The resident decode kernel against the launches layer by layer, through the runner: requests of lengths at the edges of its slices
(16 keys), of a block's share (112) and of the pages, one and two tokens, shares of rows that end in units of one to seven, K in
several pieces, windows, biases."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _config(hidden, heads, kv, dim, ff, window=None, layers=3, vocab=512):
    return {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": layers, "hidden_size": hidden,
            "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": dim, "intermediate_size": ff, "vocab_size": vocab,
            "rope_theta": 10000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": False, "use_sliding_window": window is not None,
            "sliding_window": window, "max_window_layers": 0, "max_position_embeddings": 8192, "hidden_act": "silu"}


@pytest.mark.parametrize("shape", [dict(hidden=896, heads=14, kv=2, dim=64, ff=4864),
                                   dict(hidden=1408, heads=8, kv=1, dim=128, ff=1344),
                                   dict(hidden=640, heads=6, kv=6, dim=64, ff=2752, window=100)],
                         ids=["groups-of-7", "one-kv-head", "window"])
@pytest.mark.parametrize("cached", [[300], [15, 16], [112, 1], [113, 700], [4090],
                                    [4000, 2500]], ids=["one", "slices", "share", "shares", "long", "two-long"])
def test_resident_steps_give_what_the_launches_give(shape, cached):
    from infero_b200 import kernels as K
    from infero_b200.config import EngineConfig
    from infero_b200.engine import ModelRunner, StepEntry
    from infero_b200.loading import random_model
    model, _ = random_model(_config(**shape), seed=1, dtype="bfloat16", device=DEV, generate_on_device=True)
    gen = torch.Generator().manual_seed(len(cached))
    toks = [torch.randint(512, (n + 3,), generator=gen).tolist() for n in cached]

    def run(resident):
        K.lib().infero_block_set_resident(ctypes.c_int(resident))
        try:
            runner = ModelRunner(model, EngineConfig(dtype="bfloat16", num_pages=sum(n // 16 + 2 for n in cached), max_seqs=len(cached),
                                                     ctx=max(cached) + 3, max_batch_tokens=4096, max_logit_rows=8), DEV)
            for i, n in enumerate(cached):
                runner.open(i)
                runner.step([StepEntry(i, toks[i][:n], [])])
            before = K.launch_count()
            out = [runner.step([StepEntry(i, toks[i][n + j:n + j + 1], [0]) for i, n in enumerate(cached)]).clone() for j in range(3)]
            return torch.stack(out).double(), K.launch_count() - before
        finally:
            K.lib().infero_block_set_resident(ctypes.c_int(2))

    plain, n_plain = run(0)
    resident, n_resident = run(1)
    assert n_resident < n_plain, "the resident kernel was meant to run these steps"
    # Both paths round the same values to bf16 (normed rows, q, k, v, weights of the softmax, activations), in places that differ: at
    # most 2^-9 each, 0.41 of that in the root mean square; per layer about ten roundings enter a row of the residual stream at
    # random, of a share of it below one: 4.4e-3 in all.  Two and a half times that.
    bound = 2.5 * (10 * 3) ** 0.5 * 0.41 * 2.0 ** -9
    for a, b in zip(plain.flatten(0, 1), resident.flatten(0, 1)):
        assert float((a - b).norm() / a.norm()) <= bound
    again, _ = run(1)
    assert torch.equal(resident, again)
    assert int(K.lib().infero_tc_error_flag()) == 0


@pytest.mark.parametrize("page,rotary,norms", [(32, 0.5, "bfloat16"), (64, 1.0, "float32"), (16, 0.25, "float32")], ids=["32-half", "64-norms32", "16-quarter"])
def test_other_pages_partial_rotary_and_norms_with_the_samplers_token(page, rotary, norms):
    from infero_b200 import kernels as K
    from infero_b200.config import EngineConfig
    from infero_b200.engine import ModelRunner, StepEntry
    from infero_b200.engine.step import FROM_DEVICE
    from infero_b200.models.decoder import DecoderModel
    from infero_b200.registry import resolve_architecture
    from infero_b200.weights import random_tensors
    cfg = dict(_config(896, 14, 2, 64, 1344), partial_rotary_factor=rotary)
    arch = resolve_architecture(cfg)
    model = DecoderModel(arch.to_spec(arch.read_config(cfg)))
    tensors = random_tensors(model.declare(), 2, torch.bfloat16, 0.02, 0.1, device=DEV)
    model.bind({name: t.to(getattr(torch, norms)) if "norm" in name else t for name, t in tensors.items()})
    gen = torch.Generator().manual_seed(page)
    cached, toks = [page * 3 - 1, page * 5], torch.randint(512, (2, 400), generator=gen).tolist()

    def run(resident):
        K.lib().infero_block_set_resident(ctypes.c_int(resident))
        try:
            runner = ModelRunner(model, EngineConfig(dtype="bfloat16", num_pages=32, page_size=page, max_seqs=2, ctx=512, max_batch_tokens=512, max_logit_rows=8), DEV)
            for i, n in enumerate(cached):
                runner.open(i)
                runner.step([StepEntry(i, toks[i][:n], [])])
            runner.device_tokens.copy_(torch.tensor([toks[0][350], toks[1][351]], dtype=torch.int32))
            before = K.launch_count()
            out = [runner.step([StepEntry(i, [FROM_DEVICE], [0]) for i in range(2)]).clone() for _ in range(3)]
            return torch.stack(out).double(), K.launch_count() - before
        finally:
            K.lib().infero_block_set_resident(ctypes.c_int(2))

    plain, n_plain = run(0)
    resident, n_resident = run(1)
    assert n_resident < n_plain, "the resident kernel was meant to run these steps"
    bound = 2.5 * (10 * 3) ** 0.5 * 0.41 * 2.0 ** -9                             # (as above)
    for a, b in zip(plain.flatten(0, 1), resident.flatten(0, 1)):
        assert float((a - b).norm() / a.norm()) <= bound
