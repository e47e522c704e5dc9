"""First calls from threads that have no CUDA context yet, with their memory from the allocator's cache."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["forward", "backward", "autograd", "swiglu"])
def test_first_call_of_a_thread(what):
    import gtr_b200 as G
    from gtr_b200 import workloads
    q, k, v, g = (x.cuda() for x in workloads.make_inputs(1, 64, 3, K=64))
    y = torch.randn(1, 64, 64, device="cuda").half()
    taps = torch.randn(3, 3, 64, device="cuda").half()
    leaves = [x.clone().requires_grad_() for x in (q, k, v, g)]          # clones: tensor maps of their own
    calls = {
        "forward": lambda q, k, v, g: G.chunk_gla(q, k, v, g)[0],
        "backward": lambda q, k, v, g: G.chunk_gla_backward(q, k, v, g, v)[0],
        "autograd": lambda *_: torch.autograd.grad(G.chunk_gla(*leaves)[0], leaves, v)[0],
        "swiglu": lambda *_: G.swiglu_dwconv(y, y.clone(), taps, None, (8, 8)),
    }
    want = calls[what](q, k, v, g)
    del want
    fresh = [x.clone() for x in (q, k, v, g)]
    torch.cuda.synchronize()
    got, failed = [], []

    def work():
        try:
            got.append(calls[what](*fresh))
            torch.cuda.synchronize()
        except Exception as e:                                            # noqa: BLE001 (reported by the assertion below)
            failed.append(e)

    thread = threading.Thread(target=work)
    thread.start()
    thread.join()
    assert not failed, failed
    assert torch.isfinite(got[0]).all() and torch.equal(got[0], calls[what](q, k, v, g))
