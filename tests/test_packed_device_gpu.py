"""Packed sequences whose offsets lie on the GPU (the table is made there) against the same call with offsets on the host."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(lens, H, K):
    gen = torch.Generator().manual_seed(len(lens))
    T = sum(lens)
    q, k, v = (torch.randn(1, T, H, d, generator=gen).mul(0.2).half().cuda() for d in (K, K, 64))
    g = torch.nn.functional.logsigmoid(torch.randn(1, T, H, K, generator=gen)).div(16).half().cuda()
    s0 = torch.randn(len(lens), H, K, 64, generator=gen).cuda()
    return q, k, v, g, s0


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("lens,H,K", [
    ([1], 1, 64),                                     # one block, no exchange of states
    ([0, 65, 0, 64, 63, 0], 3, 64),
    ([37] * 96, 2, 32),                               # a full table
    ([37] * 97, 2, 64),                               # one more: the host's table
    ([9000, 1, 700], 2, 64),
    ([640] * 31 + [0] * 33 + [129], 6, 64),           # empty ones on both sides of a warp's entries
])
def test_against_offsets_on_the_host(lens, H, K, dtype):
    import gtr_b200 as G
    q, k, v, g, s0 = _case(lens, H, K)
    ends = torch.tensor([0] + lens).cumsum(0).to(dtype)
    want = G.chunk_gla(q, k, v, g, initial_state=s0, output_final_state=True, cu_seqlens=ends)
    got = G.chunk_gla(q, k, v, g, initial_state=s0, output_final_state=True, cu_seqlens=ends.cuda())
    # the spans may be cut elsewhere: the operator's own bounds (fp16 operands of the tensor cores, fp32 state)
    for x, y, most in ((want[0], got[0], 1e-3), (want[1], got[1], 5e-4)):
        assert torch.isfinite(y).all() and float((x.double() - y.double()).norm() / x.double().norm()) <= most
    zero = G.chunk_gla(q, k, v, g, output_final_state=True, cu_seqlens=ends.cuda())[1]
    assert all(not zero[i].any() and torch.equal(got[1][i], s0[i]) for i, n in enumerate(lens) if n == 0)


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("ends", [[0, 30, 20, 100], [1, 30, 100], [0, 30, 99], [0, 101], [0, -1, 100], [0, 2 ** 31 - 1, 100]])
def test_offsets_that_do_not_rise_through_the_row(ends, dtype):
    import gtr_b200 as G
    q, k, v, g, _ = _case([100], 2, 64)
    good = torch.tensor([0, 40, 100], dtype=dtype, device="cuda")
    want = G.chunk_gla(q, k, v, g, cu_seqlens=good)[0]
    with pytest.raises(ValueError):
        G.chunk_gla(q, k, v, g, cu_seqlens=torch.tensor(ends, dtype=dtype, device="cuda"))
    assert torch.equal(want, G.chunk_gla(q, k, v, g, cu_seqlens=good)[0])
