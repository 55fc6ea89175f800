"""Resampling along the displacement axis with four pixels a thread: planes that end inside a thread's pixels, planes and output offsets that are
and are not multiples of 16 bytes, columns walked whole and in pieces."""
import pytest
import torch
import torch.nn.functional as F

from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N1", [1, 127, 129, 385, 511, 513, 640])
@pytest.mark.parametrize("B,K,Dl,D0", [(1, 1, 2, 5), (2, 3, 9, 19), (60, 5, 4, 9), (60, 5, 9, 9)])
def test_matches_interpolate(B, K, Dl, D0, N1, cuda_device):
    g = torch.Generator().manual_seed(N1)
    src = torch.randn(B, K, Dl, N1, 1, generator=g).to(cuda_device)
    dst = torch.zeros(B, K + 2, D0, N1, 1, device=cuda_device)
    ops.upsample_displacement_into(src, dst, 1)
    x = src.double().requires_grad_(True)
    ref = F.interpolate(x, size=(D0, N1, 1), mode="trilinear", align_corners=True)
    # source positions in FP32, up to Dl * 2^-23 off, times a difference of neighbours; a few roundings of the sum
    assert (dst[:, 1:K + 1].double() - ref).abs().max().item() < 4e-6 * max(1, Dl)
    assert not dst[:, 0].any() and not dst[:, K + 1].any()
    grad = torch.randn(B, K + 2, D0, N1, 1, generator=g).to(cuda_device)
    got = ops.upsample_displacement_backward(grad, 1, K, Dl)
    (want,) = torch.autograd.grad(ref, x, grad[:, 1:K + 1].double())
    # the same for each of the up to 2 * ceil(D0 / Dl) + 1 rows that a source row reaches
    assert (got.double() - want).abs().max().item() < 4e-6 * max(1, Dl) * (2 * -(-D0 // Dl) + 1)
