"""Workloads the library is timed on: what a program that computes separable flow with it runs, through the public
entry points, over the sizes the benchmark and the tests of this repository use.

``listed()`` names them, ``draw(rng)`` gives further ones of the same ranges; ``prepare(case, seed)`` makes what such a
program holds before the call, ``run(state)`` is one pass, ``work(case)`` the operations and bytes a pass cannot do
without and ``tolerance(case)`` how far two correct implementations of the same precision may lie apart.

A case's ``kind`` is the entry point:

* ``separate``   ``AlternateCorrBlockSepflow`` (the call site): pyramid of image 2, separation with two Conv3d attention
  modules, and when ``backward`` is set the gradients of both feature maps and of the attention parameters.  One pass is
  one pair of image batches.
* ``functions``  the three autograd Functions under their drop-in names on channels-last features, attention weights
  given; forward, and backward when set.
* ``maxavg``     the inference Function alone: max and mean channels, no attention.
* ``lookup``     ``CorrBlock1D``: displacement pyramids of the two aggregated volumes and ``iterations`` refinement
  lookups on them, with the volumes' gradients when ``backward`` is set.
* ``lookup4d``   ``AlternateCorrBlockSepflow`` as the lookup on the 4D volume: ``iterations`` refinement lookups, with the
  feature maps' gradients when ``backward`` is set.
"""
import math

import torch

import separableflowthesis_b200 as sfb

RADIUS = 4

# Every field a case of the kind has; the fields of a listed case override these.
_DEFAULTS = {
    "separate": dict(kind="separate", channels=256, attention=4, levels=4, backward=True, operands="fp16"),
    "functions": dict(kind="functions", channels=256, attention=2, backward=True, operands="fp16"),
    "maxavg": dict(kind="maxavg", channels=256, backward=False, operands="fp16"),
    "lookup": dict(kind="lookup", levels=4, iterations=12, backward=False),
    "lookup4d": dict(kind="lookup4d", channels=256, levels=4, iterations=4, backward=True),
}


def _case(name, kind, batch, height, width, **fields):
    case = dict(_DEFAULTS[kind], batch=batch, height=height, width=width, **fields)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest call: max/mean channels of one 384x512 pair (1/8 resolution), inference
        _case("maxavg_b1_48x64", "maxavg", 1, 48, 64),
        # the drop-in operators of a training step on small crops
        _case("functions_train_b2_48x64", "functions", 2, 48, 64),
        # one 440x1024 pair served alone: latency
        _case("infer_b1_55x128", "separate", 1, 55, 128, backward=False),
        # the same as a validation batch
        _case("infer_b4_55x128", "separate", 4, 55, 128, backward=False),
        # one 1080x1920 pair served alone, the case the 4D volume does not fit for
        _case("infer_b1_135x240", "separate", 1, 135, 240, backward=False),
        # a training step on small crops, where launches count
        _case("train_b2_48x64", "separate", 2, 48, 64, attention=2),
        # a training step on crops of odd size, three attention channels, full-range operands
        _case("train_b3_47x155_tf32", "separate", 3, 47, 155, attention=3, operands="tf32"),
        # a training step on 376x1248 crops with bfloat16 operands, one pyramid level
        _case("train_b8_47x156_bf16", "separate", 8, 47, 156, attention=2, levels=1, operands="bf16"),
        # the largest: a training step on full 1080x1920 frames, one pyramid level
        _case("train_b8_135x240", "separate", 8, 135, 240, levels=1),
        # twelve refinement iterations on the aggregated volumes, inference
        _case("lookup_b4_55x128", "lookup", 4, 55, 128),
        # twelve refinement iterations of a training step
        _case("lookup_train_b8_47x156", "lookup", 8, 47, 156, backward=True),
        # refinement iterations that read the 4D volume, in a training step
        _case("lookup4d_train_b2_55x128", "lookup4d", 2, 55, 128),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    """Sizes spread over the logarithm of the listed range (odd ones included), options as often as they are met in
    use, the batch cut back until the case has at most half the work of the largest listed one (pyramids and the
    drop-in Functions take up to twice the time per operation)."""
    kind = rng.choices(("separate", "functions", "maxavg", "lookup", "lookup4d"), (6, 1.5, 1, 2, 1.5))[0]
    fields = {"batch": _log_int(rng, 1, 8)}
    if kind == "lookup4d":
        fields.update(height=_log_int(rng, 16, 60), width=_log_int(rng, 24, 160), iterations=rng.randint(1, 6))
    else:
        fields.update(height=_log_int(rng, 16, 135), width=_log_int(rng, 24, 240))
    if kind == "lookup":
        fields.update(iterations=rng.randint(4, 16))
    if kind in ("separate", "functions", "maxavg"):
        fields.update(operands=rng.choices(("fp16", "tf32", "bf16"), (4, 1, 1))[0])
    if kind in ("separate", "functions"):
        fields.update(attention=rng.choices((1, 2, 3, 4), (1, 3, 1, 3))[0])
    if kind == "separate":
        fields.update(levels=rng.choices((1, 2, 3, 4), (3, 1, 1, 5))[0])
    if kind != "lookup":
        fields.update(channels=rng.choices((256, 192, 128, 96, 64), (6, 1, 2, 1, 1))[0])
    if kind != "maxavg":
        fields.update(backward=rng.random() < 0.6)
    case = dict(_DEFAULTS[kind], **fields)
    most = work(_case("", "separate", 8, 135, 240, levels=1))
    while case["batch"] > 1 and any(work(case)[k] > 0.5 * most[k] for k in most):
        case["batch"] -= 1
    return case


# ------------------------------------------------------------------------------------------------- inputs
def _coordinates(case, generator):
    """Per iteration the estimated positions (B, 2, H, W): the pixel grid plus a flow field that is smooth up to
    sub-pixel noise and moves a little from iteration to iteration, as refinement does."""
    B, H, W, dev = case["batch"], case["height"], case["width"], "cuda"
    ys, xs = torch.meshgrid(torch.arange(H, device=dev), torch.arange(W, device=dev), indexing="ij")
    yy, xx = ys.float() / H, xs.float() / W
    phase = 6.28 * torch.rand(B, 2, 1, 1, generator=generator, device=dev)
    wave = torch.stack((xx + 0.5 * yy, yy - 0.3 * xx))[None]
    flow = torch.tensor([8.0, 6.0], device=dev).view(1, 2, 1, 1) * torch.sin(6.28 * wave + phase)
    grid = torch.stack((xs, ys)).float()[None]
    coords = []
    for _ in range(case["iterations"]):
        flow = flow + 0.25 * torch.randn(B, 2, H, W, generator=generator, device=dev)
        coords.append(grid + flow)
    return coords


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, H, W, kind, backward = case["batch"], case["height"], case["width"], case["kind"], case["backward"]

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    state = {"case": case}
    if kind == "lookup":
        state["volumes"] = [randn(B, 1, W, H, W).requires_grad_(backward), randn(B, 1, H, H, W).requires_grad_(backward)]
        state["coords"] = _coordinates(case, g)
        if backward:
            rows = case["levels"] * (2 * RADIUS + 1)
            state["upstream"] = [randn(B, rows, H, W) for _ in range(2 * case["iterations"])]
        return state
    C = case["channels"]
    if kind in ("separate", "lookup4d"):
        state["fmaps"] = [randn(B, C, H, W).requires_grad_(backward) for _ in range(2)]
    if kind == "lookup4d":
        state["coords"] = _coordinates(case, g)
        if backward:
            rows = case["levels"] * (2 * RADIUS + 1) ** 2
            state["upstream"] = [randn(B, rows, H, W) for _ in range(case["iterations"])]
    elif kind == "separate":
        K = case["attention"]
        modules = [torch.nn.Conv3d(2, K, 3, padding=1, device="cuda") for _ in range(2)]
        bound = 1.0 / math.sqrt(2 * 27)    # Conv3d's own initial range, from this generator
        with torch.no_grad():
            for p in (p for m in modules for p in m.parameters()):
                p.copy_((2 * torch.rand(p.shape, generator=g, device="cuda") - 1) * bound)
        state["attention"] = modules
        if backward:
            rows = (2 + K) * case["levels"]
            state["upstream"] = [randn(B, rows, W, H, W), randn(B, rows, H, H, W)]
    else:
        state["features"] = [(randn(B, H, W, C) / math.sqrt(C)).requires_grad_(backward), randn(B, H, W, C).requires_grad_(backward)]
        if kind == "functions":
            K = case["attention"]
            state["weights"] = [randn(B, H, W, K, D).softmax(-1).requires_grad_(backward) for D in (W, H)]
            if backward:
                state["upstream"] = [randn(B, H, W, k, D) for k, D in ((2, H), (2, W), (K, H), (K, W))]
    return state


# --------------------------------------------------------------------------------------------------- passes
def run(state):
    case = state["case"]
    with torch.set_grad_enabled(case["backward"]):
        if "operands" not in case:
            return _PASSES[case["kind"]](case, state)
        with sfb.MemorySaver.sweep_operands(case["operands"]):
            return _PASSES[case["kind"]](case, state)


def _separate(case, state):
    f1, f2 = state["fmaps"]
    block = sfb.AlternateCorrBlockSepflow(f1, f2, None, num_levels=case["levels"], radius=RADIUS,
                                          support_backward=case["backward"])
    outputs = block(None, sep=True, attention_weights=state["attention"])
    if not case["backward"]:
        return outputs
    parameters = [p for m in state["attention"] for p in m.parameters()]
    grads = torch.autograd.grad(outputs, [f1, f2] + parameters, state["upstream"])
    # the parameter gradients as the one flat vector an all-reduce or a clipped step takes (a softmax does not see its
    # biases: their gradients are zero up to rounding and mean something only beside the others)
    return outputs, grads[:2], torch.cat([g.reshape(-1) for g in grads[2:]])


def _functions(case, state):
    F1, F2 = state["features"]
    first = sfb.ComputeMaxArgmaxAvgFunction if case["backward"] else sfb.ComputeMaxAvgFunction
    outputs = list(first.apply(F1, F2)) + list(sfb.ComputeSelfCompressionFunction.apply(F1, F2, *state["weights"]))
    if not case["backward"]:
        return outputs
    return outputs, torch.autograd.grad(outputs, [F1, F2] + state["weights"], state["upstream"])


def _maxavg(case, state):
    return sfb.ComputeMaxAvgFunction.apply(*state["features"])


def _lookup(case, state):
    block = sfb.CorrBlock1D(*state["volumes"], num_levels=case["levels"], radius=RADIUS)
    outputs = [out for coords in state["coords"] for out in block(coords)]
    if not case["backward"]:
        return outputs
    return outputs, torch.autograd.grad(outputs, state["volumes"], state["upstream"])


def _lookup4d(case, state):
    block = sfb.AlternateCorrBlockSepflow(*state["fmaps"], None, num_levels=case["levels"], radius=RADIUS,
                                          support_backward=case["backward"])
    outputs = [block(coords) for coords in state["coords"]]
    if not case["backward"]:
        return outputs
    return outputs, torch.autograd.grad(outputs, state["fmaps"], state["upstream"])


_PASSES = {"separate": _separate, "functions": _functions, "maxavg": _maxavg, "lookup": _lookup, "lookup4d": _lookup4d}


# ----------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes: every input read once, every output (gradients among them) written once.  Operations: a contraction of the
    features per cell of the correlation volume for the max/mean channels, one for the compression channels (whose
    weights depend on the former) and three in the backward; the Conv3d stencils; the dot products under the lookup
    windows."""
    B, H, W, kind, backward = case["batch"], case["height"], case["width"], case["kind"], case["backward"]
    pixels = B * H * W
    if kind == "lookup":
        taps = 2 * RADIUS + 1
        entries = 2 * pixels * case["levels"] * taps * case["iterations"]
        volume = pixels * (H + W)
        coords = 2 * pixels * case["iterations"]
        floats = volume + coords + entries + (entries + volume if backward else 0)
        return {"bytes": 4.0 * floats, "flops": 3.0 * entries * (2 if backward else 1)}
    C = case["channels"]
    features = 2 * pixels * C
    if kind == "lookup4d":
        window = (2 * RADIUS + 1) ** 2
        entries = pixels * case["levels"] * window * case["iterations"]
        dots = pixels * case["levels"] * (2 * RADIUS + 2) ** 2 * case["iterations"]
        floats = features + 2 * pixels * case["iterations"] + entries + (entries + features if backward else 0)
        return {"bytes": 4.0 * floats, "flops": 2.0 * C * dots * (3 if backward else 1)}
    K, levels = case.get("attention", 0), case.get("levels", 1)
    cells = sum(pixels * (H >> l) * (W >> l) for l in range(levels))
    contractions = (2 if K else 1) + ((3 if K else 2) if backward else 0)
    flops = 2.0 * C * cells * contractions
    outputs = pixels * (2 + K) * levels * (H + W)
    floats = features + outputs
    if kind == "separate":
        flops += 2.0 * 54 * K * sum(pixels * ((H >> l) + (W >> l)) for l in range(levels)) * (3 if backward else 1)
    else:
        floats += pixels * K * (H + W) * (2 if backward else 1)
    if backward:
        floats += features + outputs
    return {"bytes": 4.0 * floats, "flops": flops}


def tolerance(case):
    """FP32 lookups: sums of at most a few hundred products.  Contractions: operands of 10 mantissa bits (FP16, TF32) or
    7 (BF16), FP32 accumulation; in the backward a near tie of two cells may put a maximum's gradient on either, which
    moves whole values of a pixel's feature gradient (measured between FP16 and TF32 operands: 4.5e-3 of the norm)."""
    if case["kind"] in ("lookup", "lookup4d"):
        return {"rel": 1e-5}
    if case["backward"]:
        return {"rel": 1e-2, "max": 0.99}
    return {"rel": 5e-3 if case["operands"] == "bf16" else 1e-3}
