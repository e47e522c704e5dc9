"""The gradient where gates cut the state off, down to -inf, among weak ones: several to a chunk, in every scan order, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [-30.0, -200.0, -1000.0, -60000.0, -float("inf")])
@pytest.mark.parametrize("T,K,direction,share", [(20, 64, 0, 0.05), (64, 32, 1, 0.3), (130, 64, 1, 0.02), (500, 64, 2, 0.03), (1500, 32, 3, 0.3)])
def test_resets(value, T, K, direction, share):
    import gtr_b200 as G
    from oracle import gla_bwd_ref, gla_ref
    B, H = 2, 3
    grid = (5, T // 5) if direction >= 2 else (1, T)
    gen = torch.Generator().manual_seed(T)
    q, k, v, do = (torch.randn(B, T, H, d, generator=gen).mul(0.125).half() for d in (K, K, 64, 64))
    g = torch.nn.functional.logsigmoid(torch.randn(B, T, H, K, generator=gen)).div(16).half()
    g[torch.rand(B, T, H, K, generator=gen) < share] = value
    s0, dht = torch.randn(B, H, K, 64, generator=gen) * 0.25, torch.randn(B, H, K, 64, generator=gen) * 0.25
    order = gla_ref.scan_order(direction, *grid)
    want = gla_bwd_ref.recurrent_gla_backward(*(x[:, order] for x in (q, k, v, g, do)), initial_state=s0, d_final_state=dht)
    got = G.chunk_gla_backward(*(x.cuda() for x in (q, k, v, g, do)), initial_state=s0.cuda(), d_final_state=dht.cuda(),
                               want_d_initial_state=True, direction=direction, grid_hw=grid)
    for name, w, x in zip(("dq", "dk", "dv", "dg", "ds0"), want, got):
        x = x.cpu().double()
        if name != "ds0":
            x = x[:, order]
        assert torch.isfinite(x).all(), name
        # fp16 rounding of the outputs is 2.1e-4; dg and the state's gradient are fp32 sums over the sequence
        most = 3e-4 if name in ("dq", "dk", "dv") else 2e-5
        assert float((x - w).norm()) <= most * float(w.norm()) + 1e-30, name
