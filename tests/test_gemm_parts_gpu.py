"""32-bit products over K cut into parts: every row count, tile and way of adding the parts up gives the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("N,K,lda", [(70, 640, 640), (1100, 644, 644), (1152, 896, 900), (130, 1281, 1281), (896, 4864, 4864), (200, 5120, 5124),
                                     (200, 5124, 5124), (5000, 1924, 1924)],
                         ids=["one-part", "two", "two-896", "three-odd", "eight", "eight-full", "nine", "wide"])
def test_products_over_parts_of_k(N, K, lda):
    from infero_b200 import kernels as Kn
    g = torch.Generator(device=DEV).manual_seed(K)
    big = 640
    a = torch.randn((big, lda), generator=g, device=DEV)[:, :K]
    w, bias = torch.randn((N, K), generator=g, device=DEV), torch.randn((N,), generator=g, device=DEV)
    full = torch.empty((big, N), device=DEV)
    Kn.gemm_tiled(a, w, bias, full)
    ref = a.double() @ w.double().T + bias.double()
    # two chains of at most 340 roundings a part, the parts' sums and the bias: |error| <= (340 + parts + 2) 2^-24 (sum |a w| + |bias|)
    bound = (340 + K / 640 + 3) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T + bias.double().abs())
    assert bool(((full.double() - ref).abs() <= bound).all())
    for M in (1, 2, 4, 5, 8, 9, 16, 17, 31, 40, 64, 65, 150, 301):
        out = torch.empty((M, N), device=DEV)
        Kn.gemm_tiled(a[:M], w, bias, out)
        assert torch.equal(out, full[:M]), M
    wide = torch.empty((3, N), device=DEV, dtype=torch.bfloat16)               # operands that are widened on the way
    Kn.gemm_tiled(a[:3].bfloat16(), w, bias, wide)
    ref = (a[:3].bfloat16().double() @ w.double().T + bias.double())
    assert float((wide.double() - ref).norm() / ref.norm()) < 2.0 ** -8


@pytest.mark.parametrize("N,K", [(70, 641), (1152, 896), (9000, 300), (200, 1925), (19000, 72)])
@pytest.mark.parametrize("ta,tw", [("bfloat16", "bfloat16"), ("float32", "bfloat16"), ("bfloat16", "float32")])
def test_widened_operands_over_the_tiles(N, K, ta, tw):
    from infero_b200 import kernels as Kn
    g = torch.Generator(device=DEV).manual_seed(N)
    big = 301
    a = torch.randn((big, K), generator=g, device=DEV).to(getattr(torch, ta))
    w = torch.randn((N, K), generator=g, device=DEV).to(getattr(torch, tw))
    bias = torch.randn((N,), generator=g, device=DEV)
    full = torch.empty((big, N), device=DEV)
    Kn.gemm_tiled(a, w, bias, full)
    ref = a.double() @ w.double().T + bias.double()
    bound = (340 + K / 640 + 3) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T + bias.double().abs())     # (as above)
    assert bool(((full.double() - ref).abs() <= bound).all())
    for M in (1, 8, 9, 16, 17, 33, 63, 64, 65, 100, 128, 200):
        out = torch.full((M, N), 7.0, device=DEV)
        Kn.gemm_tiled(a[:M], w, bias, out)
        assert torch.equal(out, full[:M]), M
