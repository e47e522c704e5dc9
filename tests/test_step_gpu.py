"""The token-by-token kernel for short sequences: tile edges of its staging (16 tokens), its range (1 .. 24 tokens) and the
first length the chunk kernel takes, in every scan order, on strided views, with log gates and raw logits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [64, 32])
@pytest.mark.parametrize("grid,direction,logits", [((1, 1), 0, False), ((1, 2), 1, True), ((3, 5), 2, False), ((4, 4), 3, True),
                                                   ((17, 1), 3, False), ((4, 6), 2, True), ((1, 24), 1, False),
                                                   ((5, 5), 3, False)])
def test_short_sequences(K, grid, direction, logits):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import gtr_b200 as G
    from oracle import c_oracle, gla_ref
    B, H, T = 3, 5, grid[0] * grid[1]
    q, k, v, g = gla_ref.make_inputs(B, T, H, K=K, seed=T + K)
    s0 = torch.randn(B, H, K, 64, generator=torch.Generator().manual_seed(1))
    norm = 0.0
    log_gates = g
    if logits:
        norm, g = 16.0, (torch.randn(B, T, H, K, generator=torch.Generator().manual_seed(2)) * 2).half()
        log_gates = gla_ref.gate_from_logits(g.float(), norm).half()
    ref, ref_s = c_oracle.forward(q, k, v, log_gates, direction=direction, grid_hw=grid, initial_state=s0, output_final_state=True)
    packed = torch.cat([x.reshape(B, T, -1) for x in (q, k, g, v)], dim=-1).cuda()
    qd, kd, gd, vd = (x.unflatten(-1, (H, -1)) for x in packed.split([H * K] * 3 + [H * 64], dim=-1))
    ws = G.make_workspace(B, T, H, "cuda")
    o = torch.full((B, T, H, 64), float("nan"), dtype=torch.float16, device="cuda")
    s = torch.full((B, H, K, 64), float("nan"), device="cuda")
    G.chunk_gla_run(qd, kd, vd, gd, K ** -0.5, ws, o, norm, direction=direction, grid_hw=grid, initial_state=s0.cuda(), final_state=s)
    G.check_status(ws)
    rel = lambda a, b: float((a - b).norm() / b.norm())
    short = T <= 24
    # fp32 throughout: the outputs carry only their own rounding (at most 2^-11 each, 2^-11 / sqrt(3) in the mean), the state
    # only fp32 sums and, for logits, log gates one fp16 rounding off where logsigmoid's two forms straddle a tie
    assert rel(o.float().cpu(), ref) <= (3.5e-4 if short else 1e-3)
    assert rel(s.cpu(), ref_s) <= ((5e-5 if logits else 5e-6) if short else 5e-4)
