"""The 4D lookup's walks for a whole 4 x 4 tile: boxes on both sides of the largest one that is walked as a whole, channel
counts that leave warps to share positions or need several passes, tiles cut by the image border."""
import pytest
import torch

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# as LOOKUP_TOL of tests/test_ops_gpu.py: FP32 products of up to 512 channels in sums of up to a few hundred
TOL = 5e-5


def relerr(a, b):
    return ((a.double().cpu() - b).norm() / b.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("C", [4, 36, 132, 256, 288, 420])
# the tile's pixels lie `step` apart in the volume: boxes of (3 * step + 2r + 2)^2 positions (some one more per side)
@pytest.mark.parametrize("radius,step", [(4, 0), (4, 1), (4, 2), (4, 3), (3, 2), (2, 1), (2, 2), (1, 1), (0, 1)])
def test_box_sizes(radius, step, C, cuda_device):
    H, W, H2, W2 = 9, 6, 40, 33
    g = torch.Generator().manual_seed(C + step)
    ys, xs = torch.meshgrid(torch.arange(H).float(), torch.arange(W).float(), indexing="ij")
    coords = (torch.stack((xs, ys)) * step + 2 + 0.9 * torch.rand(2, H, W, generator=g))[None].contiguous()
    f1, gen = torch.randn(1, H, W, C, generator=g), g
    F2s = [torch.randn(1, H2, W2, C, generator=gen), torch.randn(1, H2 // 2, W2 // 2, C, generator=gen)]
    gout = torch.randn(1, 2 * (2 * radius + 1) ** 2, H, W, generator=g)
    scale = C ** -0.5
    dev = cuda_device
    out = ops.lookup4d_forward(f1.to(dev), [t.to(dev) for t in F2s], coords.to(dev), radius, scale)
    ref = orc.lookup4d_forward(f1.double(), [t.double() for t in F2s], coords.double(), radius, scale)
    assert relerr(out, ref) < TOL
    gF1, gF2 = ops.lookup4d_backward(f1.to(dev), [t.to(dev) for t in F2s], coords.to(dev), gout.to(dev), radius, scale)
    rF1, rF2 = orc.lookup4d_backward(f1.double(), [t.double() for t in F2s], coords.double(), gout.double(), radius, scale)
    assert relerr(gF1, rF1) < TOL
    for a, b in zip(gF2, rF2):
        assert relerr(a, b) < TOL


@pytest.mark.parametrize("where", ["image 1", "image 2"])
def test_infinity_reaches_its_windows_only(where, cuda_device):
    H, W, C, radius = 4, 4, 64, 2
    g = torch.Generator().manual_seed(3)
    ys, xs = torch.meshgrid(torch.arange(H).float(), torch.arange(W).float(), indexing="ij")
    coords = (torch.stack((xs, ys)) + 4.5)[None].contiguous().to(cuda_device)
    f1, f2 = torch.randn(1, H, W, C, generator=g), torch.randn(1, 16, 16, C, generator=g)
    gout = torch.randn(1, 25, H, W, generator=g).to(cuda_device)
    clean1, clean2 = f1.clone().to(cuda_device), f2.clone().to(cuda_device)
    if where == "image 1":
        f1[0, 1, 2, 5] = float("inf")
    else:
        f2[0, 4, 2, 5] = float("inf")
    a1, (a2,) = ops.lookup4d_backward(f1.to(cuda_device), [f2.to(cuda_device)], coords, gout, radius, 1.0)
    b1, (b2,) = ops.lookup4d_backward(clean1, [clean2], coords, gout, radius, 1.0)
    other = torch.arange(C, device=cuda_device) != 5
    assert torch.equal(a1[..., other], b1[..., other]) and torch.allclose(a2[..., other], b2[..., other], rtol=1e-5, atol=1e-5)
    if where == "image 1":
        # window of pixel (1, 2), centre (6.5, 5.5)
        hit = torch.zeros(16, 16, dtype=torch.bool, device=cuda_device)
        hit[3:9, 4:10] = True
        assert torch.isfinite(a1).all() and not torch.isfinite(a2[0, ..., 5][hit]).any() and torch.isfinite(a2[0, ..., 5][~hit]).all()
    else:
        # pixels with column 2 and row 4 under their windows: columns x + 2 .. x + 7, rows y + 2 .. y + 7
        hit = torch.zeros(H, W, dtype=torch.bool, device=cuda_device)
        for y in range(H):
            for x in range(W):
                hit[y, x] = x + 2 <= 2 <= x + 7 and y + 2 <= 4 <= y + 7
        assert torch.isfinite(a2).all() and not torch.isfinite(a1[0, ..., 5][hit]).any() and torch.isfinite(a1[0, ..., 5][~hit]).all()


# boxes on both sides of the table's 384 positions at smaller radii: (3 * step + 2r + 2)^2 and one more per side
@pytest.mark.parametrize("C", [36, 256])
@pytest.mark.parametrize("radius,step", [(3, 3), (3, 4), (2, 3), (2, 4), (2, 5)])
def test_largest_boxes_of_smaller_radii(radius, step, C, cuda_device):
    test_box_sizes(radius, step, C, cuda_device)
