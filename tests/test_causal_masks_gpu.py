"""Every score at or before its query counts, none after it: with unit queries, keys and values and no decay an output is the number of
tokens so far whose value lies in its channel, exactly; in both forwards (which one ran is looked up), with every epilogue and kind of gate,
and in packed sequences."""
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


def _kernels_of(call, tmp_path):
    """The names of the kernels that a call launches."""
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    graph.enable_debug_mode()
    with torch.cuda.graph(graph):
        call()
    graph.debug_dump(str(tmp_path / "call.dot"))
    return (tmp_path / "call.dot").read_text()


def _inputs(T, H, K, order, logits):
    q = torch.zeros(1, T, H, K, dtype=torch.float16, device="cuda")
    q[..., 5] = 1
    v = torch.zeros(1, T, H, 64, dtype=torch.float16, device="cuda")
    v[:, order, :, torch.arange(T, device="cuda") % 64] = 1
    want = torch.empty(1, T, H, 64, dtype=torch.float64, device="cuda")
    want[:, order] = v[:, order].double().cumsum(1)
    return q, v, torch.full_like(q, 100. if logits else 0.), want           # logsigmoid(100) is 0 in fp32


def _order(hg, wg, direction):
    order = torch.arange(hg * wg, device="cuda")
    if direction >= 2:
        order = order.view(hg, wg).t().reshape(-1)
    return order.flip(0) if direction & 1 else order


@pytest.mark.filterwarnings("ignore:DEBUG")
@pytest.mark.parametrize("logits", (False, True))
@pytest.mark.parametrize("fused", (False, True))
@pytest.mark.parametrize("in_place", (False, True))
@pytest.mark.parametrize("direction", (0, 1, 2, 3))
@pytest.mark.parametrize("grid,K", (((7, 9), 64), ((5, 13), 32), ((16, 9), 64)))       # one chunk, one and a row, three
def test_counts_in_every_variant(grid, K, direction, in_place, fused, logits, tmp_path):
    import gtr_b200
    hg, wg = grid
    T, H = hg * wg, 2
    q, v, g, want = _inputs(T, H, K, _order(hg, wg, direction), logits)
    state = torch.zeros(1, H, K, 64, device="cuda")
    final = state if in_place else torch.empty_like(state)
    out = torch.full_like(v, float("nan"))
    ws = gtr_b200.make_workspace(1, T, H, "cuda")
    gate = torch.randn(v.shape, generator=torch.Generator(device="cuda").manual_seed(T), device="cuda").half()
    weight = torch.linspace(0.5, 1.5, 64, device="cuda").half()
    kw = dict(direction=direction, grid_hw=grid, initial_state=state, final_state=final)

    def call():
        if fused:
            gtr_b200.chunk_gla_run_gated(q, q, v, g, gate, weight, 1.0, 1e-5, ws, out, float(logits), **kw)
        else:
            gtr_b200.chunk_gla_run(q, q, v, g, 1.0, ws, out, float(logits), **kw)

    names = _kernels_of(call, tmp_path)
    assert ("gla_block_kernel" in names) == in_place and ("gla_out_kernel" in names) != in_place
    call()
    if fused:
        before = want * torch.rsqrt(want.square().mean(-1, keepdim=True) + 1e-5) * weight.double()
        want = before * torch.nn.functional.silu(gate.double())
        # silu = h + h tanh h, h = gate / 2, with a tanh good to 2^-11 of its value (twice that allowed); the result in fp16
        assert bool(((out.double() - want).abs() <= 2 ** -11 * (want.abs() + (before * gate.double()).abs()) + 2 ** -24).all())
    else:
        assert torch.equal(out, want.half())
    torch.testing.assert_close(final[0, :, 5], v[0].float().sum(0), rtol=1e-6, atol=0)


@pytest.mark.parametrize("on_gpu", (False, True))
@pytest.mark.parametrize("K", (64, 32))
def test_counts_of_packed_sequences(K, on_gpu):
    import gtr_b200
    lens = [1, 64, 65, 130, 17, 63]
    T, H = sum(lens), 2
    q, v, g, _ = _inputs(T, H, K, torch.arange(T, device="cuda"), False)
    want = torch.cat([x.float().cumsum(1) for x in v.split(lens, dim=1)], dim=1).half()
    ends = torch.tensor([0] + lens, device="cuda" if on_gpu else "cpu").cumsum(0)
    out, _ = gtr_b200.chunk_gla(q, q, v, g, scale=1.0, cu_seqlens=ends)
    assert torch.equal(out, want)
