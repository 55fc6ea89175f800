"""The 4D lookup's blocks of 2 x 2 pixels where the windows lie so far apart that a walk serves one pixel at a time, blocks cut
by the image border, and blocks of both kinds in one CTA, for one to four 128-channel chunks."""
import pytest
import torch
import torch.nn.functional as F

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# FP32 products of up to 512 channels in sums of up to a few hundred, positions replicated in FP32: as LOOKUP_TOL of
# tests/test_ops_gpu.py
TOL = 5e-5


def relerr(a, b):
    return ((a.double().cpu() - b).norm() / b.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("C", [64, 160, 260, 512])
@pytest.mark.parametrize("spread", ["rows", "columns", "all"])
@pytest.mark.parametrize("size", [(6, 11), (4, 8), (5, 25)])
def test_spread_windows(size, spread, C, cuda_device):
    H, W = size
    H2, W2, radius, levels = 40, 44, 4, 2
    g = torch.Generator().manual_seed(C + W)
    ys, xs = torch.meshgrid(torch.arange(H).float(), torch.arange(W).float(), indexing="ij")
    coords = torch.stack((xs + 14, ys + 14)) + torch.rand(2, H, W, generator=g)
    if spread in ("rows", "all"):       # every other row 18 below: the two rows of a block of 2 x 2 do not fit one walk
        coords[1] += 18 * (ys.long() % 2)
    if spread in ("columns", "all"):    # some columns far to the side: pixel by pixel there, together elsewhere
        coords[0] += 21 * (xs.long() % 5 == 3)
    coords = coords[None].contiguous()
    f1 = torch.randn(1, H, W, C, generator=g)
    f2 = torch.randn(1, C, H2, W2, generator=g)
    F2s = [t.permute(0, 2, 3, 1).contiguous() for t in (f2, F.avg_pool2d(f2, 2, stride=2))]
    scale = C ** -0.5
    dev = cuda_device
    out = ops.lookup4d_forward(f1.to(dev), [t.to(dev) for t in F2s], coords.to(dev), radius, scale)
    ref = orc.lookup4d_forward(f1.double(), [t.double() for t in F2s], coords.double(), radius, scale)
    assert out.shape == ref.shape and relerr(out, ref) < TOL
    gout = torch.randn(out.shape, generator=g)
    gF1, gF2 = ops.lookup4d_backward(f1.to(dev), [t.to(dev) for t in F2s], coords.to(dev), gout.to(dev), radius, scale)
    rF1, rF2 = orc.lookup4d_backward(f1.double(), [t.double() for t in F2s], coords.double(), gout.double(), radius, scale)
    assert relerr(gF1, rF1) < TOL
    assert len(gF2) == levels
    for a, b in zip(gF2, rF2):
        assert relerr(a, b) < TOL


@pytest.mark.parametrize("radius", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("C", [20, 132, 512])
def test_scattered_windows(radius, C, cuda_device):
    """Windows all over the image and beyond its edges, so that every walk is for one pixel, for every window size."""
    H, W, H2, W2, levels = 7, 19, 22, 37, 2
    g = torch.Generator().manual_seed(radius + C)
    coords = torch.rand(2, 2, H, W, generator=g) * torch.tensor([W2 + 30.0, H2 + 30.0]).view(1, 2, 1, 1) - 15
    f1 = torch.randn(2, H, W, C, generator=g)
    f2 = torch.randn(2, C, H2, W2, generator=g)
    F2s = [t.permute(0, 2, 3, 1).contiguous() for t in (f2, F.avg_pool2d(f2, 2, stride=2))]
    dev = cuda_device
    out = ops.lookup4d_forward(f1.to(dev), [t.to(dev) for t in F2s], coords.to(dev), radius, C ** -0.5)
    ref = orc.lookup4d_forward(f1.double(), [t.double() for t in F2s], coords.double(), radius, C ** -0.5)
    assert relerr(out, ref) < TOL
    gout = torch.randn(out.shape, generator=g)
    gF1, gF2 = ops.lookup4d_backward(f1.to(dev), [t.to(dev) for t in F2s], coords.to(dev), gout.to(dev), radius, C ** -0.5)
    rF1, rF2 = orc.lookup4d_backward(f1.double(), [t.double() for t in F2s], coords.double(), gout.double(), radius, C ** -0.5)
    assert relerr(gF1, rF1) < TOL and len(gF2) == levels
    for a, b in zip(gF2, rF2):
        assert relerr(a, b) < TOL
