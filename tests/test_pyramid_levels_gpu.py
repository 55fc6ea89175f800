"""All pyramid levels in one call against the same levels one call at a time: the same bits, because neither the cut of a launch nor its
other levels enter a sum, around the edges of tiles (8 x 32 and 16 x 16), pixel tiles (128, 32 x 4), walks and softmax classes."""
import math

import pytest
import torch
import torch.nn.functional as F

from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu


def inputs(B, C, H, W, Kc, levels, seed, dev):
    g = torch.Generator().manual_seed(seed)
    f1, f2 = torch.randn(B, C, H, W, generator=g).to(dev), torch.randn(B, C, H, W, generator=g).to(dev)
    pyr = [f2]
    for _ in range(levels - 1):
        pyr.append(F.avg_pool2d(pyr[-1], 2, stride=2).contiguous())
    params = [p.to(dev) for _ in range(2) for p in (torch.randn(Kc, 2, 3, 3, 3, generator=g) * 0.2, torch.randn(Kc, generator=g) * 0.1)]
    return f1, pyr, params


def one_by_one(f1, pyr, params, with_argmax):
    B, C, H, W = f1.shape
    L, Kt = len(pyr), 2 + params[0].shape[0]
    sep_u = torch.empty(B, Kt * L, W, H, W, device=f1.device)
    sep_v = torch.empty(B, Kt * L, H, H, W, device=f1.device)
    saved = []
    for l, f2 in enumerate(pyr):
        place = (sep_u, sep_v, 0) if l == 0 else None
        su, sv, *rest = ops.separation_level_forward(f1, f2, *params, with_argmax, True, 1 / math.sqrt(C), place)
        if l > 0:
            ops.upsample_displacement_into(su, sep_u, l * Kt)
            ops.upsample_displacement_into(sv, sep_v, l * Kt)
        saved.append((su, sv, *rest))
    return sep_u, sep_v, saved


# (B, C, H, W, Kc, levels)
SHAPES = [(1, 32, 8, 32, 1, 2), (1, 64, 17, 33, 2, 3), (2, 64, 24, 40, 3, 4), (1, 256, 55, 128, 4, 4), (3, 40, 47, 155, 3, 2), (1, 128, 16, 24, 4, 4),
          (2, 256, 48, 64, 2, 4), (1, 36, 33, 31, 2, 2), (1, 64, 130, 36, 1, 4), (4, 64, 61, 130, 2, 3)]


@pytest.mark.parametrize("operands", ["fp16", "tf32", "bf16"])
@pytest.mark.parametrize("with_argmax", [True, False])
@pytest.mark.parametrize("shape", SHAPES)
def test_forward(shape, with_argmax, operands, cuda_device):
    B, C, H, W, Kc, levels = shape
    if operands == "bf16" and C % 8:
        pytest.skip("needs C % 8 == 0")
    f1, pyr, params = inputs(B, C, H, W, Kc, levels, H * W + Kc, cuda_device)
    with ops.sweep_operands(operands):
        sep_u, sep_v, buffer = ops.separation_pyramid_forward(f1, pyr, *params, with_argmax, 1 / math.sqrt(C))
        ref_u, ref_v, ref = one_by_one(f1, pyr, params, with_argmax)
    assert torch.equal(sep_u, ref_u) and torch.equal(sep_v, ref_v)
    for got, want in zip(ops.separation_pyramid_saved(buffer, f1, pyr, Kc, with_argmax), ref):
        for x, y in zip(got, want):
            assert (x is None) == (y is None) and (x is None or torch.equal(x, y))
