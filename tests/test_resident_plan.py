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
