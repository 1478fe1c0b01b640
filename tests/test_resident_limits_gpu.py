"""The resident decode kernel where it cannot run."""
import ctypes

import pytest
import torch

from test_resident_gpu import _config

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _runner(layers=2):
    from infero_b200.config import EngineConfig
    from infero_b200.engine import ModelRunner
    from infero_b200.loading import random_model
    model, _ = random_model(_config(hidden=896, heads=14, kv=2, dim=64, ff=1024, layers=layers), seed=1, dtype="bfloat16", device=DEV, generate_on_device=True)
    return ModelRunner(model, EngineConfig(dtype="bfloat16", num_pages=16, max_seqs=1, ctx=128, max_batch_tokens=64, max_logit_rows=8), DEV)


def _step(runner, resident):
    from infero_b200 import kernels as K
    from infero_b200.engine import StepEntry
    K.lib().infero_block_set_resident(ctypes.c_int(resident))
    try:
        runner.open(0)
        runner.step([StepEntry(0, list(range(40)), [])])
        before = K.launch_count()
        return runner.step([StepEntry(0, [7], [0])]).clone(), K.launch_count() - before
    finally:
        runner.close(0)
        K.lib().infero_block_set_resident(ctypes.c_int(2))


def test_more_blocks_than_multiprocessors_keep_the_launches(monkeypatch):
    from infero_b200.kernels import tc_gemm
    real = tc_gemm.sm_count(DEV)
    monkeypatch.setitem(tc_gemm._SM_COUNT, 0, real + 12)
    plain, many = _step(_runner(), 0)
    other, launches = _step(_runner(), 1)
    assert launches == many and torch.equal(plain, other)


def test_a_wait_that_runs_out_names_the_kernel(monkeypatch):
    """A token at position -1 sees no keys: nobody writes its attention, the wait for it ends at its limit and the step returns."""
    from infero_b200.kernels import tc_gemm
    runner = _runner()
    good, launches = _step(runner, 1)
    assert launches < 6, "the resident kernel was meant to run this step (the launches layer by layer must not see such a position)"
    build = runner._build_context

    def nowhere(entries, rcs):
        ctx, rows = build(entries, rcs)
        if len(entries[0].tokens) == 1:
            ctx.positions.fill_(-1)
        return ctx, rows

    with monkeypatch.context() as m:
        m.setattr(runner, "_build_context", nowhere)
        runner.drop_graphs()
        _step(runner, 1)
        torch.cuda.synchronize()
    assert tc_gemm.error_flag() == 10
    assert tc_gemm.error_flag() == 0
    runner.drop_graphs()
    again, _ = _step(runner, 1)
    assert torch.equal(good, again) and tc_gemm.error_flag() == 0
