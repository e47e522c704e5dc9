"""Calls that the two models' comparison sends to one or the other of the forward's kernels, on either side of where they meet and
with segments of the caller's own, against the CPU oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,chunks,K,direction,fused,logits,segments", [
    (18, 12, 20, 64, 1, False, True, 0),         # more sequences than SMs: relayed
    (37, 4, 40, 32, 0, True, False, 0),          # as many: whole sequences
    (37, 4, 40, 64, 3, True, True, 0),
    (74, 8, 4, 64, 2, False, False, 0),          # many short ones: the small kernels
    (37, 8, 12, 64, 0, False, False, 0),         # whole sequences in two rounds
    (1, 1, 1500, 64, 1, False, False, 0),        # one long sequence
    (2, 3, 100, 64, 0, False, False, 1),         # the caller's segments: many spans to a sequence,
    (1, 3, 200, 64, 3, True, False, 50),         # few long ones,
    (8, 12, 25, 32, 0, False, True, 4),          # enough for four to an SM
])
def test_against_the_oracle(B, H, chunks, K, direction, fused, logits, segments):
    import gtr_b200 as G
    from oracle import c_oracle, gla_ref
    T = chunks * 64 - (0 if direction >= 2 else 13)
    grid = (64, chunks) if direction >= 2 else None
    q, k, v, g = gla_ref.make_inputs(B, T, H, K=K, seed=T)
    norm, gates = 0.0, g
    if logits:
        norm = 16.0
        g = torch.randn(B, T, H, K, generator=torch.Generator().manual_seed(T)).half()
        gates = (torch.nn.functional.logsigmoid(g.float()) / norm).half()
    want, want_s = c_oracle.forward(q, k, v, gates, output_final_state=True, direction=direction, grid_hw=grid)
    ws = torch.zeros(max(G.workspace_floats(B, T, H), B * H * 8400 * (chunks // max(segments, 1) + 2) if segments else 0), device="cuda")
    y = torch.full((B, T, H, 64), float("nan"), dtype=torch.float16, device="cuda")
    final = torch.empty(B, H, K, 64, device="cuda")
    x = [t.cuda() for t in (q, k, v, g)]
    kw = dict(direction=direction, grid_hw=grid, final_state=final, segments=segments)
    if fused:
        gen = torch.Generator().manual_seed(1)
        gate, w = torch.randn(B, T, H, 64, generator=gen).half(), (torch.rand(64, generator=gen) + 0.5).half()
        want = gla_ref.rmsnorm_swish_gate(want, gate, w, 1e-5)
        G.chunk_gla_run_gated(*x, gate.cuda(), w.cuda(), K ** -0.5, 1e-5, ws, y, norm, **kw)
    else:
        G.chunk_gla_run(*x, K ** -0.5, ws, y, norm, **kw)
    G.check_status(ws)
    m = gla_ref.error_metrics(want, y.float().cpu())
    assert m["finite"] and m["rel_l2"] <= 1e-3, m           # the operator's own bounds
    assert float((final.cpu() - want_s).norm() / want_s.norm()) < 5e-4
