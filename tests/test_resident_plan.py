"""Host side of the resident decode kernel: where its scratch lies."""
import ctypes
from ctypes import c_float, c_int, c_longlong, c_void_p

import pytest


class _Step(ctypes.Structure):
    _fields_ = [(n, c_int) for n in ("n_tok", "n_layers", "hidden", "n_heads", "n_kv", "ff", "rotary_dim", "page_size", "max_blocks", "norm_dtype",
                                     "qkv_bias_dtype", "o_bias_dtype")] + [("inv_hidden", c_float)] + \
               [(n, c_void_p) for n in ("positions", "tok_entry", "x", "h0", "h1", "sums0", "sums1", "qkv", "attn", "act", "part_o", "part_ml", "stop",
                                        "counters")]


@pytest.mark.parametrize("n_kv,heads,dim", [(1, 8, 128), (2, 14, 64), (16, 16, 64)])
def test_every_layer_counts_arrivals_on_its_own(n_kv, heads, dim):
    from infero_b200 import kernels as K
    f = K.lib().infero_resident_scratch
    f.restype = c_longlong
    s = _Step(hidden=896, n_heads=heads, n_kv=n_kv, ff=4864)
    base = 1 << 30
    end = base + f(ctypes.byref(s), c_void_p(base), c_int(dim), c_int(148))
    layers, tokens = 48, 2
    assert end - s.counters >= layers * tokens * n_kv * 4
    places = sorted(getattr(s, n) for n, t in s._fields_[16:])
    assert places[0] == base and places[-1] == s.counters and len(set(places)) == len(places)


@pytest.mark.parametrize("hidden,ff,heads,kv,dim,tokens,visible,want", [
    (896, 4864, 14, 2, 64, 1, 20, 1), (896, 4864, 14, 2, 64, 1, 4096, 1), (896, 4864, 14, 2, 64, 1, 4097, 0), (896, 4864, 14, 2, 64, 2, 2048, 1),
    (896, 4864, 14, 2, 64, 2, 2049, 0), (896, 4864, 14, 2, 64, 1, 32768, 0),
    (640, 8192, 10, 2, 64, 1, 2048, 1), (640, 8192, 10, 2, 64, 1, 4090, 0), (1024, 5120, 16, 4, 64, 1, 2048, 1), (1024, 5120, 16, 4, 64, 2, 2040, 0),
    (1024, 6912, 16, 4, 64, 1, 20, 0),
    (1024, 4096, 8, 8, 128, 1, 1000, 1), (1024, 4096, 8, 8, 128, 1, 2048, 0), (640, 2560, 10, 10, 64, 1, 4090, 1), (640, 1024, 16, 16, 128, 1, 2040, 1),
    (640, 1024, 16, 16, 128, 1, 4090, 0), (640, 1024, 16, 16, 128, 2, 2040, 0),
])
def test_long_contexts_and_large_layers_keep_the_launches(hidden, ff, heads, kv, dim, tokens, visible, want):
    from infero_b200 import kernels as K
    s = _Step(n_tok=tokens, n_layers=24, hidden=hidden, n_heads=heads, n_kv=kv, ff=ff, page_size=16)
    assert K.lib().infero_resident_worth(ctypes.byref(s), c_int(dim), c_int(148), c_int(visible)) == want
