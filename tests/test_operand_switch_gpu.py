"""GPU: a call computes with one operand type from its preparation to its last kernel, also when another thread moves the
process-wide switch (``ops.sweep_operands``) while the call is being enqueued: every result equals, bit for bit, the result
under one of the types."""
import threading

import pytest
import torch

from separableflowthesis_b200 import _lib, ops

pytestmark = pytest.mark.gpu

KINDS = ("tf32", "bf16", "fp16")


def inputs(dev):
    g = torch.Generator().manual_seed(77)
    B, H, W, C, K = 1, 20, 36, 64, 6   # six channels: two chunks, so every operand-dependent step runs more than once
    F1 = torch.randn(B, H, W, C, generator=g) / C ** 0.5
    F2 = torch.randn(B, H, W, C, generator=g)
    A = [torch.randn(B, H, W, K, D, generator=g).softmax(-1) for D in (W, H)]
    up = [torch.randn(B, H, W, k, D, generator=g) for k, D in ((2, H), (2, W), (K, H), (K, W))]
    F1, F2, a_u, a_v, gm_u, gm_v, gc_u, gc_v = (t.to(dev) for t in (F1, F2, *A, *up))
    _, _, am_u, am_v = ops.max_argmax_avg_forward(F1, F2)
    cf = lambda t: t.permute(0, 3, 4, 1, 2).contiguous()
    am_cf = [t.squeeze(3).permute(0, 3, 1, 2).contiguous() for t in (am_u, am_v)]
    return {
        "max/avg backward": lambda: ops.max_argmax_avg_backward(F1, F2, am_u, am_v, gm_u, gm_v),
        "compression backward": lambda: ops.compression_backward(F1, F2, a_u, a_v, gc_u, gc_v),
        "separation backward": lambda: ops.separation_backward(F1, F2, am_u, am_v, gm_u, gm_v, a_u, a_v, gc_u, gc_v),
        "feature backward, channels first": lambda: ops.separation_feature_backward_cf(
            F1, F2, *am_cf, cf(gm_u), cf(gm_v), cf(a_u), cf(a_v), cf(gc_u), cf(gc_v)),
    }


@pytest.mark.parametrize("name", ["max/avg backward", "compression backward", "separation backward",
                                  "feature backward, channels first"])
def test_a_call_keeps_its_operand_type(name, cuda_device):
    call = inputs(cuda_device)[name]
    want = []
    for kind in KINDS:
        with ops.sweep_operands(kind):
            want.append([t.clone() for t in call()])
    lib = _lib.load()
    before = lib.sfb_get_sweep_operands()
    stop = threading.Event()

    def flip():
        while not stop.is_set():
            for code in (0, 1, 2):
                lib.sfb_set_sweep_operands(code)

    other = threading.Thread(target=flip)
    other.start()
    seen, odd = set(), 0
    try:
        for _ in range(400):
            got = call()
            hits = [i for i, w in enumerate(want) if all(torch.equal(x, y) for x, y in zip(got, w))]
            seen.update(hits)
            odd += not hits
    finally:
        stop.set()
        other.join()
        lib.sfb_set_sweep_operands(before)
    assert odd == 0, f"{odd} of 400 calls mixed operand types"
    assert len(seen) > 1   # the switch did move between calls
