"""The workloads this framework's speed is judged on: what its users call, at the sizes they call it with.

Seven kinds of call, each through the public entry point a program would use:

* ``step``      ``fused_recurrent_gla`` on one or a few new tokens with the state carried from call to call;
* ``scan``      ``chunk_gla_run``, the operator on caller-owned workspace and output, any scan order;
* ``block``     ``chunk_gla_run_gated`` as a backbone block calls it: strided views of one packed projection, raw gate
                logits, RMSNorm * w * silu(gate) fused;
* ``packed``    ``chunk_gla`` on sequences of different lengths packed in one row (``cu_seqlens``);
* ``train``     ``chunk_gla`` recorded by autograd, and its gradient;
* ``mlp``       ``swiglu_dwconv``, the middle of the backbone's MLP;
* ``backbone``  ``GraphedBackbone``: stem and twelve blocks, deploy form.

All inputs are synthetic and made on the GPU from a seed.
"""
import math

import torch

import gtr_b200
from gtr_b200.backbone import GraphedBackbone, GTRBackbone

V = 64


def listed():
    return [
        # one new token for each of 32 sequences, state carried: the smallest call, all latency
        dict(name="step_one_token", kind="step", B=32, T=1, H=12, K=64),
        # one 640 x 640 image's tokens (40 x 40 patches) through a six-head layer: a single low-latency forward
        dict(name="scan_one_image", kind="scan", B=1, H=6, hg=40, wg=40, K=64, direction=1, gates="weak", states=False),
        # the high-resolution throughput point (80 x 80 patches, 12 heads), on a column scan
        dict(name="scan_high_resolution", kind="scan", B=4, H=12, hg=80, wg=80, K=64, direction=2, gates="weak", states=False),
        # the released models' 32-channel key heads on an odd grid whose last chunk is ragged, states in and out
        dict(name="scan_k32_ragged_states", kind="scan", B=3, H=3, hg=25, wg=42, K=32, direction=3, gates="weak", states=True),
        # large values and almost no forgetting over very long spans: the numerically hard end
        dict(name="scan_open_gates", kind="scan", B=2, H=8, hg=64, wg=128, K=64, direction=0, gates="open", states=False),
        # what a block of the 1024 x 2048 backbone hands the operator for eight images
        dict(name="block_fused", kind="block", B=8, H=12, hg=64, wg=128, K=64, direction=1),
        # images of different sizes packed back to back
        dict(name="packed_sequences", kind="packed", H=12, K=64, states=True,
             lens="1600 196 2304 1024 49 640 1225 400 3136 256 900 1 1450 576 784 64"),
        # a training step of the operator: small images, row scan
        dict(name="train_small_images", kind="train", B=8, H=6, hg=40, wg=40, K=64, direction=0),
        # a training step at high resolution on a reversed column scan
        dict(name="train_high_resolution", kind="train", B=4, H=12, hg=80, wg=80, K=64, direction=3),
        # depthwise convolution and gating of the MLP on eight 1024 x 2048 images
        dict(name="mlp_middle", kind="mlp", B=8, hg=64, wg=128, C=3072),
        # detection on one 640 x 640 image with the released small model's width
        dict(name="backbone_one_image", kind="backbone", B=1, height=640, width=640, dim=192, heads=3, expand_k=0.5),
        # throughput inference on 1024 x 2048 images
        dict(name="backbone_high_resolution", kind="backbone", B=4, height=1024, width=2048, dim=768, heads=12, expand_k=1.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "scan", "scan", "block", "packed", "train", "train", "mlp", "backbone"))
    K = rng.choice((64, 64, 32))
    direction = rng.randrange(4)
    if kind == "step":
        return dict(kind=kind, B=_log_int(rng, 1, 96), T=rng.choice((1, 1, _log_int(rng, 2, 64))), H=rng.randint(2, 16), K=K)
    if kind == "scan":
        hg, wg = rng.randint(12, 100), rng.randint(12, 100)
        H = rng.choice((3, 6, 8, 12))
        B = _log_int(rng, 1, max(1, min(16, 780000 // (hg * wg * H))))
        return dict(kind=kind, B=B, H=H, hg=hg, wg=wg, K=K, direction=direction, gates=rng.choice(("weak", "weak", "open")),
                    states=rng.random() < 0.3)
    if kind == "block":
        hg, wg = rng.randint(20, 96), rng.randint(20, 128)
        H = rng.choice((3, 6, 12))
        B = _log_int(rng, 1, max(1, min(16, 780000 // (hg * wg * H))))
        return dict(kind=kind, B=B, H=H, hg=hg, wg=wg, K=K, direction=direction)
    if kind == "packed":
        lens = [_log_int(rng, 1, 4096) for _ in range(rng.randint(2, 32))]
        while sum(lens) > 24000:
            lens.pop()
        return dict(kind=kind, H=rng.choice((3, 6, 12)), K=K, states=rng.random() < 0.5, lens=" ".join(map(str, lens)))
    if kind == "train":
        hg, wg = rng.randint(10, 80), rng.randint(10, 80)
        H = rng.choice((3, 6, 12))
        B = _log_int(rng, 1, max(1, min(16, 300000 // (hg * wg * H))))
        return dict(kind=kind, B=B, H=H, hg=hg, wg=wg, K=K, direction=direction)
    if kind == "mlp":
        hg, wg, C = rng.randint(12, 96), rng.randint(12, 128), 256 * rng.randint(2, 12)
        B = _log_int(rng, 1, max(1, min(16, 200000000 // (hg * wg * C))))
        return dict(kind=kind, B=B, hg=hg, wg=wg, C=C)
    dim, heads, expand_k = rng.choice(((192, 3, 0.5), (384, 6, 0.5), (384, 6, 1.0), (768, 12, 1.0)))
    h, w = 16 * rng.randint(20, 64), 16 * rng.randint(20, 64)
    B = _log_int(rng, 1, max(1, min(8, 32768 * 256 // (h * w))))
    return dict(kind="backbone", B=B, height=h, width=w, dim=dim, heads=heads, expand_k=expand_k)


def _lens(case):
    return [int(x) for x in case["lens"].split()]


def _values(gen, shape, std):
    return (torch.randn(shape, generator=gen, device="cuda") * std).half()


def _log_gates(gen, shape, kind):
    # "weak": a layer at initialisation, normaliser 16; "open": near-zero decay, normaliser 1
    x = torch.randn(shape, generator=gen, device="cuda")
    x = torch.nn.functional.logsigmoid(x) / 16 if kind == "weak" else torch.nn.functional.logsigmoid(2 * x + 4)
    return x.half()


def _qkvg(gen, B, T, H, K, gates="weak"):
    std = 0.125 if gates == "weak" else 3.0
    q, k, v = (_values(gen, (B, T, H, d), std) for d in (K, K, V))
    return q, k, v, _log_gates(gen, (B, T, H, K), gates)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "backbone":
        torch.manual_seed(seed)
        with torch.device("cuda"):
            model = GTRBackbone(embed_dim=case["dim"], num_heads=case["heads"], expand_k=case["expand_k"])
        model = model.half().eval().convert_to_deploy()
        image = torch.rand(case["B"], 3, case["height"], case["width"], generator=gen, device="cuda").half()
        return dict(case=case, runner=GraphedBackbone(model), image=image)
    if kind == "mlp":
        shape = (case["B"], case["hg"] * case["wg"], case["C"])
        gate, y = _values(gen, shape, 1.0), _values(gen, shape, 1.0)
        return dict(case=case, gate=gate, y=y, taps=_values(gen, (3, 3, case["C"]), 1 / 3), bias=_values(gen, (case["C"],), 0.1),
                    out=torch.empty_like(y))
    H, K = case["H"], case["K"]
    if kind == "step":
        x = _qkvg(gen, case["B"], case["T"], H, K)
        return dict(case=case, x=x, state=torch.randn(case["B"], H, K, V, generator=gen, device="cuda") * 0.25)
    if kind == "packed":
        lens = _lens(case)
        ends = torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32)
        state = torch.randn(len(lens), H, K, V, generator=gen, device="cuda") * 0.25 if case["states"] else None
        return dict(case=case, x=_qkvg(gen, 1, sum(lens), H, K), ends=ends, state=state)
    B, T = case["B"], case["hg"] * case["wg"]
    if kind == "train":
        x = [t.requires_grad_(True) for t in _qkvg(gen, B, T, H, K)]
        return dict(case=case, x=x, do=_values(gen, (B, T, H, V), 0.125))
    ws = gtr_b200.make_workspace(B, T, H, "cuda")
    out = torch.empty(B, T, H, V, dtype=torch.float16, device="cuda")
    if kind == "scan":
        state = final = None
        if case["states"]:
            state = torch.randn(B, H, K, V, generator=gen, device="cuda") * 0.25
            final = torch.empty_like(state)
        return dict(case=case, x=_qkvg(gen, B, T, H, K, case["gates"]), ws=ws, out=out, state=state, final=final)
    # block: one fused projection's output, split into strided views; q and k small, the rest of order one
    widths = (H * K, H * K, H * V, H * V, H * K)
    packed = torch.randn(B, T, sum(widths), generator=gen, device="cuda", dtype=torch.float16)
    packed[..., :2 * H * K] *= 0.125
    q, k, v, gate, logits = (t.unflatten(-1, (H, -1)) for t in packed.split(widths, dim=-1))
    weight = (torch.rand(V, generator=gen, device="cuda") + 0.5).half()
    return dict(case=case, q=q, k=k, v=v, gate=gate, logits=logits, weight=weight, ws=ws, out=out)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "backbone":
        return state["runner"](state["image"])
    if kind == "mlp":
        return gtr_b200.swiglu_dwconv(state["gate"], state["y"], state["taps"], state["bias"], (case["hg"], case["wg"]),
                                      state["out"])
    if kind == "step":
        return gtr_b200.fused_recurrent_gla(*state["x"], initial_state=state["state"], output_final_state=True)
    if kind == "packed":
        return gtr_b200.chunk_gla(*state["x"], initial_state=state["state"], output_final_state=case["states"],
                                  cu_seqlens=state["ends"])
    grid = (case["hg"], case["wg"])
    if kind == "train":
        o, _ = gtr_b200.chunk_gla(*state["x"], direction=case["direction"], grid_hw=grid)
        return (o,) + torch.autograd.grad(o, state["x"], state["do"])
    scale = case["K"] ** -0.5
    if kind == "scan":
        gtr_b200.chunk_gla_run(*state["x"], scale, state["ws"], state["out"], direction=case["direction"], grid_hw=grid,
                               initial_state=state["state"], final_state=state["final"])
        return state["out"], state["final"]
    gtr_b200.chunk_gla_run_gated(state["q"], state["k"], state["v"], state["logits"], state["gate"], state["weight"], scale, 1e-5,
                                 state["ws"], state["out"], 16.0, direction=case["direction"], grid_hw=grid)
    return state["out"]


def work(case):
    """Bytes and operations of one pass: each input read once, each output written once; the recurrence's own
    multiply-adds (decay and update of the state, read-out), the MLP's taps, the backbone's products."""
    kind = case["kind"]
    if kind == "mlp":
        n = case["B"] * case["hg"] * case["wg"] * case["C"]
        return {"bytes": 6 * n + 20 * case["C"], "flops": 22 * n}
    if kind == "backbone":
        B, dim, heads, depth = case["B"], case["dim"], case["heads"], 12
        L = (case["height"] // 16) * (case["width"] // 16)
        key, inter = int(dim * case["expand_k"]), 256 * ((dim * 4 + 255) // 256)
        per_token = dim * (3 * key + 2 * dim) + dim * dim + 3 * dim * inter            # multiply-adds of a block's products
        stem = sum(256 // 4 ** (i + 1) * 9 * a * b for i, (a, b) in
                   enumerate(zip((3, dim // 8, dim // 4, dim // 2), (dim // 8, dim // 4, dim // 2, dim))))
        flops = B * L * (depth * (2 * per_token + 18 * inter + heads * 5 * (key // heads) * V) + 2 * stem)
        return {"bytes": 2 * (depth * per_token + B * 3 * case["height"] * case["width"] + 3 * B * L * dim), "flops": flops}
    H, K = case["H"], case["K"]
    n = sum(_lens(case)) if kind == "packed" else case["B"] * (case["T"] if kind == "step" else case["hg"] * case["wg"])
    rows = n * H                                                                         # (token, head) pairs
    if kind == "train":
        return {"bytes": 2 * rows * (6 * K + 4 * V), "flops": rows * 17 * K * V}
    sequences = 0
    if kind == "step":
        sequences = case["B"]
    elif case.get("states"):
        sequences = len(_lens(case)) if kind == "packed" else case["B"]
    values = 3 * V if kind == "block" else 2 * V
    return {"bytes": 2 * rows * (3 * K + values) + 8 * sequences * H * K * V, "flops": rows * 5 * K * V}


def tolerance(case):
    # outputs are fp16, and the operator's tensor-core operands are: a few half units of 2^-11 each.  The backbone rounds
    # to fp16 some eighty times in a row.
    if case["kind"] == "backbone":
        return {"rel": 1e-2}
    if case["kind"] == "mlp":
        return {"rel": 1e-3}
    return {"rel": 2e-3}
