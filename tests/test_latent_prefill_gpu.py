"""Latent attention of prompt portions with their keys and values written out (``csrc/latent_prefill_tc.cu``), against the plain
implementation in 64 bits; the rule that picks it."""
import types

import numpy as np
import pytest
import torch

from infero_b200.kernels import latent_prefill as P

TOL = 2.5e-2          # bf16 operands, as the kernels that attend over the latent rows are held to


def _ctx(lens, pos0):
    return types.SimpleNamespace(h_q_len=np.array(lens, dtype=np.int32), h_pos0=np.array(pos0, dtype=np.int32), n_entries=len(lens))


@pytest.mark.parametrize("lens,pos0,window,want", [
    ([16], [0], None, (0, 1, 1)), ([15], [0], None, None), ([1, 1, 300], [9, 900, 0], None, (2, 5, 3)),
    ([1, 1], [9, 900], None, None),                                  # single tokens only
    ([100], [400], None, None), ([100], [300], None, (0, 7, 1)),     # behind too long a prefix; within the bound
    ([100], [4000], 128, (0, 5, 1)),                                 # the window leaves 100 + 127 keys, from 3,840 on
    ([40, 1, 129], [0, 5, 64], None, (0, 1 + 1 + 4, 1 + 1 + 2)),     # a single token behind a portion goes with it
])
def test_the_rule(lens, pos0, window, want):
    got = P.plan(_ctx(lens, pos0), torch.bfloat16, 4, 64, 64, 32, 128, window)
    assert got == (None if want is None else P.Plan(*want))
    assert P.plan(_ctx(lens, pos0), torch.float32, 4, 64, 64, 32, 128, window) is None
    for D, V, R, C in ((32, 32, 16, 128), (64, 128, 32, 256), (64, 64, 72, 256), (64, 64, 12, 256), (128, 128, 64, 128), (64, 64, 32, 132)):
        assert P.plan(_ctx(lens, pos0), torch.bfloat16, 4, D, V, R, C, window) is None


@pytest.mark.parametrize("lens,pos0,window,want", [
    ([600], [0], None, True), ([1, 600], [40, 0], None, True), ([1, 500], [40, 0], None, False), ([1] * 64 + [24], [99] * 64 + [0], None, False),
    ([1, 200, 300, 220], [7, 0, 0, 0], None, False), ([1, 200], [7, 500], None, False), ([1, 300], [7, 900], None, True),       # (pairs count)
    ([1, 600], [40, 0], 256, False), ([1, 1500], [40, 0], 256, True),                  # a window bounds them
])
def test_beside_single_tokens_only_portions_that_are_worth_it(lens, pos0, window, want):
    """16 heads of 128 with a latent of 512 save 12,288 multiply-adds a pair: from about 174,763 pairs on."""
    args = (torch.bfloat16, 16, 128, 128, 64, 512, window)
    ctx = _ctx(lens, pos0)
    p = P.step_plan(ctx, *args)
    assert (p is not None) == want and P.plan(ctx, *args) is not None
    ctx.h_q_len = None                                               # (the layers behind the first one ask no more)
    assert P.step_plan(ctx, *args) is p


@pytest.mark.gpu
@pytest.mark.parametrize("H,D,R,C,page", [(16, 128, 64, 512, 16), (3, 64, 32, 256, 64), (2, 128, 8, 256, 16), (5, 64, 64, 136, 16)])
def test_portions_at_the_edges_of_tiles(H, D, R, C, page, monkeypatch):
    """Portions of 1 to 300 tokens beside each other and behind prefixes, single tokens in front of them; shuffled pages."""
    from test_gositar_gpu import _Latent, _rel
    from infero_b200.kernels import tc_gemm
    g = torch.Generator().manual_seed(D + R)
    cuts = {"s": [2, 1, 1], "a": [64, 65, 128], "b": [129, 300], "c": [127, 1, 63], "d": [193, 192]}
    hs = None
    for least in (1, 1 << 30):                          # written out, and through the latent rows
        # (queries and keys grow with the input's width here: the scale leaves scores a spread of a few units)
        a = _Latent("bfloat16", H, D, R, D, C, gated=H != 3, pairing="half" if H == 3 else "adjacent", seed=H, page=page, pages=120,
                    scale=3.0 / (max(64, H * D) * C * (D + R)) ** 0.5)
        if hs is None:
            hs = {r: torch.randn(sum(n), a.d, generator=g).to(torch.bfloat16).float() for r, n in cuts.items()}
            want = {r: a.plain(h) for r, h in hs.items()}
        monkeypatch.setattr(P, "MIN_TOKENS", least)
        monkeypatch.setattr(P, "MIN_BESIDE", 0)         # (single tokens in front or not)
        got, before = {r: [] for r in cuts}, P.launches["steps"]
        for i in range(3):
            entries = [(r, hs[r][sum(n[:i]):sum(n[:i]) + n[i]]) for r, n in cuts.items() if i < len(n)]
            for r, rows in a.step(entries).items():
                got[r].append(rows)
        assert P.launches["steps"] == before + (3 if least == 1 else 0) and tc_gemm.error_flag() == 0
        for r in hs:
            assert _rel(torch.cat(got[r]), want[r]) < TOL, (r, least)


@pytest.mark.gpu
@pytest.mark.parametrize("H,D,R,C", [(16, 128, 64, 512), (8, 64, 32, 256)])
@pytest.mark.parametrize("n", [16, 130])
def test_written_out_is_no_further_from_64_bits(H, D, R, C, n, monkeypatch):
    from test_gositar_gpu import _Latent
    g = torch.Generator().manual_seed(n)
    errors = []
    for least in (1, 1 << 30):                          # written out, and through the latent rows
        monkeypatch.setattr(P, "MIN_TOKENS", least)
        a = _Latent("bfloat16", H, D, R, D, C, pairing="half", pages=n // 16 + 8, scale=2.0 / (H * D * C * (D + R)) ** 0.5)
        if not errors:
            h = torch.randn(n, a.d, generator=g).to(torch.bfloat16).float()
            want = a.plain(h).cpu()
        got = a.step([("x", h)])["x"].double().cpu()
        errors.append(float((got - want).norm() / want.norm()))
    assert errors[0] <= errors[1]


def test_values_that_halves_hold():
    w, norm = torch.full((3, 64), 10.0), torch.ones(64)              # 2-norm of a row: 80; of a latent row: 8
    assert P.values_fit(w, norm, 64) and P.values_fit(w * 100, norm, 64)
    w[1] *= 102                                                      # 65,280 in exact numbers, more with the latents rounded up
    assert not P.values_fit(w, norm, 64) and P.values_fit(w, norm * 0.9, 64) and not P.values_fit(w * 0.9, norm * 2, 64)
    assert not P.values_fit(w * float("nan"), norm, 64)


@pytest.mark.gpu
def test_values_that_halves_do_not_hold_keep_to_the_latent_rows():
    from test_gositar_gpu import DEV, _Latent, _rel
    for times in (1.0, 3.0e4):
        a = _Latent("bfloat16", 2, 64, 32, 64, 128, seed=3, scale=0.06, pages=40)
        name = a.part._n("up_v")
        a.w[name] = a.w[name] * times
        a.part.bind({k: v.to(DEV) for k, v in a.w.items()})
        before = P.launches["steps"]
        h = torch.randn(70, a.d, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).float()
        assert _rel(a.step([("x", h)])["x"], a.plain(h)) < TOL
        assert P.launches["steps"] == before + (times == 1.0)


@pytest.mark.gpu
@pytest.mark.parametrize("window", [1, 64, 100, 129])
def test_windows_and_sinks(window, monkeypatch):
    import plain_dukolorn as PD
    from test_dukolorn_gpu import EPS, _inputs, _latent_alone, _rel, latent
    from infero_b200.kernels import tc_gemm
    monkeypatch.setattr(P, "MIN_TOKENS", 1)
    H, D, R, C, scale = 3, 64, 32, 128, 0.08
    a = _latent_alone(H, D, R, D, C, scale, window, "bfloat16", pages=128)
    m, w, d = latent(H, D, R, D, C, scale, 500.0, window), a.weights(), a.spec.hidden
    hs = {r: _inputs(n, d, "bfloat16", n, 0.4) for r, n in (("a", 500), ("b", 90))}
    before = P.launches["steps"]
    first = a.step([("a", hs["a"][:201]), ("b", hs["b"])])
    then = a.step([("a", hs["a"][201:])])
    assert P.launches["steps"] == before + 2 and tc_gemm.error_flag() == 0
    for r, rows in (("a", torch.cat([first["a"], then["a"]])), ("b", first["b"])):
        assert _rel(rows[:, :H * D], PD.latent_inner(hs[r].double(), w, "mix", m, EPS)) < TOL, r


@pytest.mark.gpu
def test_one_requests_infinities_stay_its_own():
    """Tiles of a request end in rows of zeros, not in the next request's keys."""
    from test_gositar_gpu import _Latent, _rel
    a = _Latent("bfloat16", 2, 64, 32, 64, 128, seed=3, scale=0.06, pages=40)
    g = torch.Generator().manual_seed(1)
    h = torch.randn(70, a.d, generator=g).to(torch.bfloat16).float()
    got = a.step([("x", h), ("y", torch.full((64, a.d), float("inf")))])
    assert _rel(got["x"], a.plain(h)) < TOL and not bool(torch.isfinite(got["y"]).all())


@pytest.mark.gpu
@pytest.mark.parametrize("H,D,R,V,C", [(16, 128, 64, 128, 512), (3, 96, 16, 20, 64), (5, 32, 0, 72, 256)])
@pytest.mark.parametrize("n", [1, 8, 9, 16, 17])
def test_few_single_tokens_in_two_launches(H, D, R, V, C, n, monkeypatch):
    """Steps of 1 to 17 single tokens behind prefixes of 3 to 200 tokens: 16 and fewer without the grouped products, 17 with them; against
    64 bits and, where both can run, no further from it than by a quarter (the roundings are the same ones, in another order of sums)."""
    from test_gositar_gpu import _Latent, _rel
    from infero_b200.kernels import latent_attention as A, tc_gemm
    g = torch.Generator().manual_seed(n + D)
    lens = [3 + (197 * i) // max(1, n - 1) for i in range(n)]
    a = None
    calls, errors = [], []
    real = A.query_few
    monkeypatch.setattr(A, "query_few", lambda *x, **k: (calls.append(1), real(*x, **k))[1])
    for few in (True, False):
        a = _Latent("bfloat16", H, D, R, V, C, gated=H != 3, pairing="half", seed=H, pages=16 * n + 16, scale=3.0 / (max(64, H * V) * C * (D + R)) ** 0.5)
        if few:
            hs = [torch.randn(m + 2, a.d, generator=g).to(torch.bfloat16).float() for m in lens]
            want = torch.cat([a.plain(h)[-2:] for h in hs])
        else:
            monkeypatch.setattr(A, "few_ok", lambda *x: False)
        for i, h in enumerate(hs):
            a.step([(i, h[:-2])])
        calls.clear()
        got = [a.step([(i, h[h.shape[0] - 2 + k:h.shape[0] - 1 + k]) for i, h in enumerate(hs)]) for k in range(2)]
        assert len(calls) == (2 if few and n <= 16 else 0) and tc_gemm.error_flag() == 0
        out = torch.cat([torch.cat([got[0][i], got[1][i]]) for i in range(n)])
        errors.append(float((out.double().cpu() - want.double().cpu()).norm() / want.double().cpu().norm()))
        assert _rel(out, want) < TOL, few
    assert errors[0] <= 1.25 * errors[1]


@pytest.mark.gpu
def test_up_projections_that_start_anywhere():
    """Values of another width than the keys keep the caller's own projection, here two bytes behind a multiple of 16."""
    from test_gositar_gpu import DEV, _Latent, _rel
    a = _Latent("bfloat16", 3, 64, 16, 20, 64, seed=2, scale=0.05, pages=40)
    bound = {k: v.to(DEV) for k, v in a.w.items()}
    name = a.part._n("up_v")
    up_v = bound[name]
    moved = torch.empty(up_v.numel() + 8, dtype=up_v.dtype, device=DEV)[1:1 + up_v.numel()].view(up_v.shape)
    assert moved.data_ptr() % 16
    bound[name] = moved.copy_(up_v)
    a.part.bind(bound)
    g = torch.Generator().manual_seed(1)
    hs = [torch.randn(n + 1, a.d, generator=g).to(torch.bfloat16).float() for n in (5, 30)]
    first = a.step([(i, h[:-1]) for i, h in enumerate(hs)])
    last = a.step([(i, h[-1:]) for i, h in enumerate(hs)])
    for i, h in enumerate(hs):
        assert _rel(torch.cat([first[i], last[i]]), a.plain(h)) < TOL
