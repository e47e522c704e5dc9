"""States updated in place: `final_state` over `initial_state`, in every decomposition such a call can take, against the same call
with arrays of their own."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,T,K,direction,fused,segments,repeats", [
    (4, 12, 1600, 64, 0, False, 0, 200),         # three segments of a sequence, and spans of several sequences on the small kernels
    (4, 12, 700, 64, 1, False, 0, 200),
    (1, 6, 1600, 64, 2, False, 0, 50),           # fewer segments than there are SMs for
    (4, 12, 6400, 64, 3, True, 0, 20),
    (16, 12, 640, 32, 0, False, 0, 50),          # more sequences than SMs: relayed segments
    (64, 12, 130, 64, 1, True, 0, 50),           # whole sequences
    (3, 3, 1050, 32, 0, False, 2, 50),
    (2, 3, 24, 64, 0, False, 0, 5),              # the token-by-token kernel
    (2, 3, 25, 64, 0, False, 0, 5),
])
def test_in_place(B, H, T, K, direction, fused, segments, repeats):
    import gtr_b200 as G
    gen = torch.Generator(device="cuda").manual_seed(T)
    draw = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    q, k, v = (draw(B, T, H, d).mul(0.3).half() for d in (K, K, 64))
    g = torch.nn.functional.logsigmoid(draw(B, T, H, K)).div(16).half()
    gate, w = draw(B, T, H, 64).half(), draw(64).half()
    s0 = draw(B, H, K, 64) * 10                  # large: a state read after it was replaced shows
    grid = (5, T // 5) if direction >= 2 else None
    ws = G.make_workspace(B, T, H, "cuda")

    def call(initial, final):
        o = torch.empty(B, T, H, 64, dtype=torch.float16, device="cuda")
        kw = dict(direction=direction, grid_hw=grid, initial_state=initial, final_state=final, segments=segments)
        if fused:
            G.chunk_gla_run_gated(q, k, v, g, gate, w, K ** -0.5, 1e-5, ws, o, **kw)
        else:
            G.chunk_gla_run(q, k, v, g, K ** -0.5, ws, o, **kw)
        return o.float()

    final = torch.empty_like(s0)
    want = call(s0, final)
    # both calls are within 5e-4 of the exact operator each
    for _ in range(repeats):
        state = s0.clone()
        got = call(state, state)
        assert float((got - want).norm() / want.norm()) <= 1e-3 and float((state - final).norm() / final.norm()) <= 1e-3
    G.check_status(ws)


def test_packed_sequences_refuse_it():
    from gtr_b200 import _lib
    x = torch.zeros(1, 64, 1, 64, dtype=torch.float16, device="cuda")
    state = torch.zeros(1, 1, 64, 64, device="cuda")
    ws = torch.zeros(1 << 20, device="cuda")
    a = _lib.Args()
    a.q = a.k = a.v = a.g = x.data_ptr()
    o = torch.empty_like(x)
    a.o = o.data_ptr()
    a.initial_state = a.final_state = state.data_ptr()
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel() * 4
    a.B, a.T, a.H, a.K, a.V, a.scale = 1, 64, 1, 64, 64, 0.125
    offsets = (ctypes.c_int32 * 2)(0, 64)
    assert _lib.lib().gla_b200_forward_packed(ctypes.byref(a), offsets, 1, None) == -9
