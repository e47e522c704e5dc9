"""The depthwise-conv + SwiGLU kernel at the edges of its tiles, channel slabs and ring: grids on either side of a tile,
grids that take another tile shape, channels on either side of a slab, and more blocks than there are SMs, against PyTorch
in fp32."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,hg,wg,C,with_bias", [(1, 16, 16, 64, True), (1, 17, 15, 72, True), (1, 15, 17, 56, False), (2, 33, 100, 128, True),
                                                 (1, 1, 300, 64, False), (1, 300, 1, 8, True), (5, 65, 19, 648, True)])
def test_tiles(B, hg, wg, C, with_bias):
    import gtr_b200 as G
    gen = torch.Generator().manual_seed(hg * 131 + wg)
    gate, y = (torch.randn(B, hg * wg, C, generator=gen).half().cuda() for _ in range(2))
    taps = (torch.randn(3, 3, C, generator=gen) * 0.3).half().cuda()
    bias = torch.randn(C, generator=gen).half().cuda() if with_bias else None
    out = torch.full_like(y, float("nan"))
    G.swiglu_dwconv(gate, y, taps, bias, (hg, wg), out=out)
    img = y.double().view(B, hg, wg, C).permute(0, 3, 1, 2)
    kernel = taps.double().permute(2, 0, 1).unsqueeze(1)
    conv = F.conv2d(img, kernel, None if bias is None else bias.double(), padding=1, groups=C).permute(0, 2, 3, 1).reshape(B, -1, C)
    size = F.conv2d(img.abs(), kernel.abs(), None if bias is None else bias.double().abs(), padding=1, groups=C)
    size = size.permute(0, 2, 3, 1).reshape(B, -1, C)
    g = gate.double()
    # the result's rounding to fp16 (2^-11 of it, 2^-25 below the normals), the tanh approximation (2^-11 absolute, taken times
    # |g| / 2 and the conv) and nine fp32 roundings of the conv's partial sums
    bound = F.silu(g).abs() * conv.abs() * 2 ** -10.9 + g.abs() * conv.abs() * 2 ** -11 + g.abs() * size * 2 ** -20 + 2 ** -24
    assert ((out.double() - F.silu(g) * conv).abs() <= bound).all()
