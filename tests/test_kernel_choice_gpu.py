"""Calls on either side of the line between the operator's two small kernels and the persistent one, plain and with the fused
epilogue, against the CPU oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,grid,direction,K,states,fused", [
    (8, 12, (41, 77), 1, 64, True, False),        # 96 x 50 chunks: past 32 chunks per SM
    (8, 12, (41, 75), 1, 64, True, False),        # 96 x 49: short of it
    (1, 16, (128, 148), 3, 32, False, False),     # 16 x 296: just there, staggered segments
    (16, 13, (37, 41), 2, 64, True, False),       # 208 x 24: relayed segments
    (12, 12, (96, 64), 0, 64, False, True),       # 144 x 96: the fused line
    (12, 12, (95, 64), 0, 64, False, True),
])
def test_either_side(B, H, grid, direction, K, states, fused):
    import gtr_b200 as G
    from oracle import c_oracle, gla_ref
    T = grid[0] * grid[1]
    q, k, v, g = gla_ref.make_inputs(B, T, H, K=K, seed=T)
    gen = torch.Generator().manual_seed(1)
    s0 = torch.randn(B, H, K, 64, generator=gen) * 0.25 if states else None
    want, want_s = c_oracle.forward(q, k, v, g, initial_state=s0, output_final_state=states, direction=direction, grid_hw=grid)
    ws = G.make_workspace(B, T, H, "cuda")
    y = torch.full((B, T, H, 64), float("nan"), dtype=torch.float16, device="cuda")
    x = [t.cuda() for t in (q, k, v, g)]
    if fused:
        gate = torch.randn(B, T, H, 64, generator=gen).half()
        w = (torch.rand(64, generator=gen) + 0.5).half()
        want = gla_ref.rmsnorm_swish_gate(want, gate, w, 1e-5)
        G.chunk_gla_run_gated(*x, gate.cuda(), w.cuda(), K ** -0.5, 1e-5, ws, y, direction=direction, grid_hw=grid)
    else:
        final = torch.empty(B, H, K, 64, device="cuda") if states else None
        G.chunk_gla_run(*x, K ** -0.5, ws, y, direction=direction, grid_hw=grid, initial_state=None if s0 is None else s0.cuda(),
                        final_state=final)
        if states:
            assert float((final.cpu() - want_s).norm() / want_s.norm()) < 5e-4
    G.check_status(ws)
    m = gla_ref.error_metrics(want, y.float().cpu())
    assert m["finite"] and m["rel_l2"] <= 1e-3, m           # the operator's own bound
