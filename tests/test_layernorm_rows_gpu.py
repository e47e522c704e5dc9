"""LayerNorm with one and with two rows per warp, at an odd number of rows and at every register shape, against PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [8, 256, 264, 768, 1000, 1032, 2048])
@pytest.mark.parametrize("rows", [1, 9472, 9473, 9475])
def test_rows_per_warp(rows, D):
    import gtr_b200 as G
    gen = torch.Generator(device="cuda").manual_seed(D)
    x = torch.randn(1, rows, D, generator=gen, device="cuda").half()
    w, b = (torch.randn(D, generator=gen, device="cuda").half() for _ in range(2))
    got = G.layernorm(x, w, b, 1e-6)
    mean, var = x.double().mean(-1, keepdim=True), x.double().var(-1, unbiased=False, keepdim=True)
    scaled = (x.double() - mean) * (var + 1e-6).rsqrt() * w.double()
    # the result's rounding to fp16 (2^-11 of it, 2^-25 below the normals) and fp32 sums of D terms
    bound = (scaled + b.double()).abs() * 2 ** -11 + (scaled.abs() + b.double().abs() + w.double().abs()) * 2 ** -16 + 2 ** -24
    assert ((got.double() - scaled - b.double()).abs() <= bound).all()
