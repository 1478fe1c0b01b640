"""Gated linear attention over long portions cut into segments that run side by side (csrc/channel_memory.cuh)."""
import pytest
import torch

from infero_b200.kernels import layer_ops as L

DEV = "cuda:0"


def test_which_portions_are_cut():
    cut = lambda lens: L._segments(lens, 2, 4, 8, "cpu")[:2]                      # noqa: E731
    assert cut(None) == cut([]) == cut([1023]) == (0, 0) and cut([1024]) == (256, 4) and cut([3, 1201, 257, 256]) == (256, 1 + 5 + 2 + 1)
    assert cut([1200, 1300]) == (256, 5 + 6) and cut([1100, 600, 600]) == (0, 0)
    starts, totals = L._segments([3, 1201, 257, 256], 2, 4, 8, "cpu")[2:]
    assert tuple(starts.shape) == (7, 2, 4, 8) and tuple(totals.shape) == (7, 2, 8)


@pytest.mark.gpu
@pytest.mark.parametrize("K,V", [(128, 128), (64, 36), (32, 5), (20, 16), (200, 8)])
def test_segments_against_whole_portions_and_64_bits(K, V, monkeypatch):
    """Portions around multiples of a segment, beside short ones, from states of their own: read-outs and the states left."""
    H, lens = 2, [1, 49, 32, 0, 127, 33]
    T, E = sum(lens), len(lens)
    g = torch.Generator().manual_seed(K)
    Kp = int(L.lib().infero_channel_rows(K))
    rec = torch.zeros(H, T, 3, Kp)
    rec[:, :, 0, :K] = torch.rand(H, T, K, generator=g) * 0.3 + 0.7
    rec[0, 60:64, 0, :K] = 0.0                                                     # a decay of nothing wipes what was before
    rec[:, :, 1:, :K] = torch.randn(H, T, 2, K, generator=g)
    v, state = torch.randn(T, H * V, generator=g), torch.randn(E + 1, H * V * K, generator=g)
    starts = [sum(lens[:e]) for e in range(E)]
    slots = [3, 0, 5, 6, 1, 4]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)                # noqa: E731
    want_y, want_s = torch.zeros(T, H, V, dtype=torch.float64), state.double().view(E + 1, H, V, K).clone()
    for e, n in enumerate(lens):
        S = want_s[slots[e]]
        for t in range(starts[e], starts[e] + n):
            a, k, q = (rec[:, t, i, :K].double() for i in range(3))
            S = S * a[:, None] + v[t].double().view(H, V, 1) * k[:, None]
            want_y[t] = (S * q[:, None]).sum(-1) * K ** -0.5
        want_s[slots[e]] = S
    for seg in (0, 16, 48):
        monkeypatch.setattr(L, "SEGMENT", seg or 1 << 20)
        if seg:                                          # (the rule wants one long portion; the kernels take any)
            counts = [-(-n // seg) if n > seg else 1 for n in lens]
            many = sum(c for c in counts if c > 1)
            plan = (seg, sum(counts), torch.full((many, H, V, K), float("nan"), device=DEV), torch.full((many, H, K), float("nan"), device=DEV))
            monkeypatch.setattr(L, "_segments", lambda *a, plan=plan: plan)
        st = state.to(DEV).clone()
        y = L.decayed_scan(v.to(DEV), rec.view(H, T, 3 * Kp).to(DEV), st, 0, i32(starts), i32(lens), i32(slots), E, H, K, V, False, lens)
        for got, want in ((y.double().cpu().view(T, H, V), want_y), (st.double().cpu().view(E + 1, H, V, K), want_s)):
            # (sums of a few dozen live terms in 32 bits)
            assert float((got - want).abs().max() / want.abs().max()) < 5e-6, seg
