"""The chunk-by-chunk gradient kernels where they can go wrong: every scan order with ragged and mirrored chunks, segments that
hand states on, chunks whose decay needs the pair-by-pair path between ordinary ones, and gradients far from unit size (the
tensor cores' fp16 operand pairs are scaled per chunk).

Bounds as for the other gradient tests: 1e-3 (fp16 outputs; their own rounding is 2.8e-4) and 1e-4 (fp32) relative L2 against the
float64 oracle on the same fp16 inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import gtr_b200
    return gtr_b200


def _rel(want, got):
    got = got.double().cpu()
    assert bool(torch.isfinite(got).all())
    return float((got - want).norm() / want.norm().clamp_min(1e-300))


def _case(B, T, H, K, seed, do_scale=0.125):
    from oracle import gla_ref
    q, k, v, g = gla_ref.make_inputs(B, T, H, K=K, seed=seed)
    gen = torch.Generator().manual_seed(seed + 7)
    do = (torch.randn(B, T, H, 64, generator=gen) * do_scale).half()
    s0 = torch.randn(B, H, K, 64, generator=gen) / 8
    dht = torch.randn(B, H, K, 64, generator=gen) * do_scale
    return q, k, v, g, do, s0, dht


def _check(G, q, k, v, g, do, s0, dht, direction=0, grid=None):
    from oracle import gla_bwd_ref, gla_ref
    perm = torch.arange(q.shape[1]) if grid is None else gla_ref.scan_order(direction, *grid)
    want = gla_bwd_ref.recurrent_gla_backward(q[:, perm], k[:, perm], v[:, perm], g[:, perm], do[:, perm], initial_state=s0,
                                              d_final_state=dht)
    got = G.chunk_gla_backward(*(x.cuda() for x in (q, k, v, g, do)), None, s0.cuda(), dht.cuda(), True, direction=direction,
                               grid_hw=grid)
    torch.cuda.synchronize()
    for i, n in enumerate(("dq", "dk", "dv", "dg")):
        back = torch.empty_like(want[i])
        back[:, perm] = want[i]
        assert _rel(back, got[i]) <= (1e-3 if i < 3 else 1e-4), n
    assert _rel(want[4], got[4]) <= 1e-4


@pytest.mark.parametrize("K", [64, 32])
@pytest.mark.parametrize("grid,direction", [((1, 65), 1), ((9, 7), 2), ((8, 8), 3), ((5, 26), 3), ((11, 36), 1), ((23, 17), 2)])
def test_scan_orders_and_ragged_chunks(G, K, grid, direction):
    _check(G, *_case(2, grid[0] * grid[1], 3, K, seed=grid[0] + K), direction=direction, grid=grid)


@pytest.mark.parametrize("direction", [0, 3])
def test_strong_chunks_between_ordinary_ones(G, direction):
    grid = (20, 32)
    q, k, v, g, do, s0, dht = _case(1, 640, 2, 64, seed=3)
    g = g.clone()
    g[:, 100:260] = -2.0                  # chunks that decay by e^-128
    g[:, 400:410, :, :8] = -30.0          # a burst in a few channels
    g[:, 500:564] = -0.2                  # 2^-18 over a chunk: just beyond the common reference's range
    _check(G, q, k, v, g, do, s0, dht, direction, grid)


@pytest.mark.parametrize("do_scale", [2.0 ** -17, 64.0])
def test_gradient_sizes(G, do_scale):
    """fp16 outputs of subnormal size cannot be compared relatively, so the small case looks at dg, d initial_state only."""
    from oracle import gla_bwd_ref
    q, k, v, g, do, s0, dht = _case(1, 300, 2, 64, seed=5, do_scale=do_scale)
    want = gla_bwd_ref.recurrent_gla_backward(q, k, v, g, do, initial_state=s0, d_final_state=dht)
    got = G.chunk_gla_backward(*(x.cuda() for x in (q, k, v, g, do)), None, s0.cuda(), dht.cuda(), True)
    if do_scale > 1:
        assert max(_rel(want[i], got[i]) for i in range(3)) <= 1e-3
    assert _rel(want[3], got[3]) <= 1e-4 and _rel(want[4], got[4]) <= 1e-4


@pytest.mark.parametrize("K", [64, 32])
@pytest.mark.parametrize("grid,direction", [((1, 64), 1), ((7, 13), 2), ((1, 300), 0), ((20, 33), 3)])
def test_nothing_but_strong_chunks(G, K, grid, direction):
    q, k, v, _, do, s0, dht = _case(2, grid[0] * grid[1], 3, K, seed=11)
    x = torch.randn(q.shape, generator=torch.Generator().manual_seed(12))
    _check(G, q, k, v, torch.nn.functional.logsigmoid(x - 2).half(), do, s0, dht, direction, grid)
