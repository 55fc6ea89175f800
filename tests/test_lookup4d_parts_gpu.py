"""Gradients of the 4D lookup where two blocks share a tile's levels, with one and with two channels to a lane: every number of
levels, channel counts on both sides of what a lane, a warp and a block take."""
import pytest
import torch

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# as LOOKUP_TOL of tests/test_ops_gpu.py: FP32 products of up to 512 channels in sums of up to a few hundred
TOL = 5e-5


def relerr(a, b):
    return ((a.double().cpu() - b).norm() / b.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("levels", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("C", [8, 32, 36, 64, 68, 128, 196, 260, 512])
def test_levels_and_channels(levels, C, cuda_device):
    B, H, W, radius = 2, 6, 7, 3
    g = torch.Generator().manual_seed(C + levels)
    ys, xs = torch.meshgrid(torch.arange(H).float(), torch.arange(W).float(), indexing="ij")
    coords = (torch.stack((xs, ys)) * 1.5 + 2 + torch.rand(B, 2, H, W, generator=g)).contiguous()
    f1 = torch.randn(B, H, W, C, generator=g)
    F2s = [torch.randn(B, max(17 >> l, 2), max(22 >> l, 2), C, generator=g) for l in range(levels)]
    gout = torch.randn(B, levels * (2 * radius + 1) ** 2, H, W, generator=g)
    args = (f1.to(cuda_device), [t.to(cuda_device) for t in F2s], coords.to(cuda_device), gout.to(cuda_device), radius, C ** -0.5)
    stale = [torch.full((B * H * W * C,), float("nan"), device=cuda_device) for _ in range(4)]   # memory the results may come to lie in
    del stale
    gF1, gF2 = ops.lookup4d_backward(*args)
    rF1, rF2 = orc.lookup4d_backward(f1.double(), [t.double() for t in F2s], coords.double(), gout.double(), radius, C ** -0.5)
    assert relerr(gF1, rF1) < TOL
    for a, b in zip(gF2, rF2):
        assert relerr(a, b) < TOL
    assert torch.equal(gF1, ops.lookup4d_backward(*args)[0])
