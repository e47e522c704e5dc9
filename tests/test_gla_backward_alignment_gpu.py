"""Gradients into buffers that start on 16-byte but not on 32-byte boundaries: other stores, the same bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [64, 32])
def test_outputs_between_sectors(K):
    import gtr_b200 as G
    from gtr_b200 import _lib
    B, T, H = 2, 100, 3
    gen = torch.Generator().manual_seed(K)
    q, k, v, do = (torch.randn(B, T, H, d, generator=gen).mul(0.5).half().cuda() for d in (K, K, 64, 64))
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, H, K, generator=gen)).div(16).half().cuda()
    want = G.chunk_gla_backward(q, k, v, g, do)[:4]

    def between(x):
        size, skip = x.numel(), 16 // x.element_size()
        flat = torch.full((size + 64,), float("nan"), dtype=x.dtype, device="cuda")
        return flat[skip:skip + size].view(x.shape)

    got = [between(x) for x in want]
    assert all(x.data_ptr() % 32 == 16 for x in got)
    ws = torch.empty(G.ops.backward_workspace_bytes(B, T, H, K), dtype=torch.uint8, device="cuda")
    a = _lib.BwdArgs()
    a.q, a.k, a.v, a.g, a.d_o = (x.data_ptr() for x in (q, k, v, g, do))
    a.dq, a.dk, a.dv, a.dg = (x.data_ptr() for x in got)
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    a.B, a.T, a.H, a.K, a.V, a.scale = B, T, H, K, 64, K ** -0.5
    _lib.check(_lib.lib().gla_b200_backward(ctypes.byref(a), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(want, got))
