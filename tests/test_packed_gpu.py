"""Packed sequences in one launch: lengths around the chunk size, empty ones, one long sequence cut into segments among short
ones, more sequences than a launch's table holds (96), with log gates and raw logits, states in and out."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,H,K,logits", [
    ([1, 63, 64, 65, 0, 128, 129], 3, 64, False),
    ([5000, 20, 300, 64, 1], 2, 64, False),            # few heads: the long one is cut into many segments
    ([3000, 2900, 700], 12, 32, True),
    ([0, 0, 40], 1, 64, False),
    ([(7 * i) % 90 for i in range(200)], 2, 64, False),
    ([640] * 40, 12, 64, True),                        # more items than SMs
])
def test_packed(lens, H, K, logits):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import gtr_b200 as G
    from oracle import c_oracle, gla_ref
    T = sum(lens)
    q, k, v, g = gla_ref.make_inputs(1, T, H, K=K, seed=len(lens))
    s0 = torch.randn(len(lens), H, K, 64, generator=torch.Generator().manual_seed(3)) * 0.5
    norm, log_gates = 0.0, g
    if logits:
        norm, g = 16.0, (torch.randn(1, T, H, K, generator=torch.Generator().manual_seed(2)) * 2).half()
        log_gates = gla_ref.gate_from_logits(g.float(), norm).half()
    ends = torch.tensor([0] + lens).cumsum(0)
    o, s = G.chunk_gla(q.cuda(), k.cuda(), v.cuda(), g.cuda(), initial_state=s0.cuda(), output_final_state=True,
                       cu_seqlens=ends.cuda(), gk_normalizer=norm)
    assert o.shape == (1, T, H, 64) and s.shape == (len(lens), H, K, 64)
    o, s = o.float().cpu(), s.cpu()
    want_o, want_s = torch.empty_like(o), torch.empty_like(s)
    for i, (a, b) in enumerate(zip(ends[:-1].tolist(), ends[1:].tolist())):
        if a == b:
            assert torch.equal(s[i], s0[i])
            want_s[i] = s0[i]
            continue
        want_o[:, a:b], want_s[i:i + 1] = c_oracle.forward(*(x[:, a:b].contiguous() for x in (q, k, v, log_gates)),
                                                           initial_state=s0[i:i + 1], output_final_state=True)
    # the operator's own bounds: fp16 operands of the tensor cores, fp32 state
    assert torch.isfinite(o).all() and float((o - want_o).norm() / want_o.norm()) <= 1e-3
    assert float((s - want_s).norm() / want_s.norm()) < 5e-4
    assert float((o - want_o).abs().max()) <= 4e-3 * float(want_o.abs().max())


@pytest.mark.parametrize("ends", [
    torch.tensor([0, 2 ** 32 + 30, 100]), torch.tensor([2 ** 32, 30, 100]), torch.tensor([0, 30, 2 ** 33 + 100]),   # good in their low halves
    [0, 2 ** 32 + 30, 100], [0, 2 ** 70, 100], [0, 40, 30, 100], [0], [],
])
def test_offsets_that_are_no_good_as_they_came(ends):
    import gtr_b200 as G
    x = torch.zeros(1, 100, 2, 64, dtype=torch.float16, device="cuda")
    with pytest.raises(ValueError):
        G.chunk_gla(x, x, x, x, cu_seqlens=ends)


def test_offsets_may_come_as_any_iterable():
    import gtr_b200 as G
    gen = torch.Generator().manual_seed(0)
    x = torch.randn(1, 100, 2, 64, generator=gen).half().cuda()
    g = -torch.rand(1, 100, 2, 64, generator=gen).half().cuda()
    want, state = G.chunk_gla(x, x, x, g, output_final_state=True, cu_seqlens=torch.tensor([0, 30, 60, 90, 100]))
    for ends in ([0, 30, 60, 90, 100], (0, 30, 60, 90, 100), iter([0, 30, 60, 90, 100]), np.array([0, 30, 60, 90, 100]), torch.tensor([0., 30, 60, 90, 100])):
        got, final = G.chunk_gla(x, x, x, g, output_final_state=True, cu_seqlens=ends)
        assert torch.equal(want, got) and torch.equal(state, final)
