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
            K.lib().infero_block_set_resident(ctypes.c_int(1))

    plain, n_plain = run(0)
    resident, n_resident = run(1)
    assert n_resident < n_plain, "the resident kernel was meant to run these steps"
    # Both paths round the same values to bf16 (normed rows, q, k, v, weights of the softmax, activations), 2^-9 each, in places that
    # differ; per layer about ten roundings enter a row of the residual stream at random, of a share of it below one.
    bound = 3 * (10 * 3) ** 0.5 * 2.0 ** -9
    for a, b in zip(plain.flatten(0, 1), resident.flatten(0, 1)):
        assert float((a - b).norm() / a.norm()) <= bound
    again, _ = run(1)
    assert torch.equal(resident, again)
    assert int(K.lib().infero_tc_error_flag()) == 0
