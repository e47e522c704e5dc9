"""Every score at or before its query counts, none after it: with unit queries, keys and values and no decay an output is the number of
tokens so far whose value lies in its channel, exactly."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("in_place", (False, True))           # states updated in place go to the persistent kernel
@pytest.mark.parametrize("direction", (0, 1, 2, 3))
@pytest.mark.parametrize("grid", ((8, 8), (5, 13), (16, 9)))
def test_counts(grid, direction, in_place):
    import gtr_b200
    hg, wg = grid
    T, H = hg * wg, 2
    q = torch.zeros(1, T, H, 64, dtype=torch.float16, device="cuda")
    q[..., 5] = 1
    g = torch.zeros_like(q)
    order = torch.arange(T, device="cuda")
    if direction >= 2:
        order = order.view(hg, wg).t().reshape(-1)
    if direction & 1:
        order = order.flip(0)                                   # order[p]: the token at scan position p
    v = torch.zeros_like(q)
    v[:, order, :, torch.arange(T, device="cuda") % 64] = 1
    want = torch.empty_like(q)
    want[:, order] = v[:, order].float().cumsum(1).half()
    state = torch.zeros(1, H, 64, 64, device="cuda")
    final = state if in_place else torch.empty_like(state)
    out = torch.full_like(q, float("nan"))
    gtr_b200.chunk_gla_run(q, q.clone(), v, g, 1.0, gtr_b200.make_workspace(1, T, H, "cuda"), out, direction=direction, grid_hw=grid,
                           initial_state=state, final_state=final)
    assert torch.equal(out, want)
    torch.testing.assert_close(final[0, :, 5], v[0].float().sum(0), rtol=1e-6, atol=0)     # exponentials of whole numbers, a few units of 2^-23
