"""The many-row norm at a width whose ring takes exactly the shared memory that a launch gets without asking."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_rows_of_1536():
    from infero_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(1)
    x, delta = torch.randn((300, 1536), generator=g, device="cuda"), torch.randn((300, 1536), generator=g, device="cuda")
    w, out = torch.randn((1536,), generator=g, device="cuda").bfloat16(), torch.empty((300, 1536), dtype=torch.bfloat16, device="cuda")
    want = x.double() + delta.double()
    K.add_rmsnorm(x, delta, w, 1e-6, out)
    assert float((x.double() - want).abs().max()) < 1e-6
    want = want * torch.rsqrt(want.pow(2).mean(1, keepdim=True) + 1e-6) * w.double()
    assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -8
