"""The 4D lookup's forward with 16 and with 32 lanes per position, all of them with channels or not, and features that are not finite outside
every window."""
import pytest
import torch

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# as LOOKUP_TOL of tests/test_ops_gpu.py: FP32 products of up to 512 channels, positions replicated in FP32
TOL = 5e-5


@pytest.mark.parametrize("C", [4, 64, 68, 128, 132, 192, 196, 256, 260, 384, 388, 512])
@pytest.mark.parametrize("spread", [0, 9])   # windows of 2 x 2 pixels together, and of one pixel
def test_forward(C, spread, cuda_device):
    H, W, H2, W2, radius = 5, 7, 12, 15, 4
    g = torch.Generator().manual_seed(C)
    ys, xs = torch.meshgrid(torch.arange(H).float(), torch.arange(W).float(), indexing="ij")
    # the last row and column look beyond the image
    coords = (torch.stack((xs, ys)) * 2 + 5 + spread * torch.rand(2, H, W, generator=g))[None].contiguous()
    f1, f2 = torch.randn(1, H, W, C, generator=g), torch.randn(1, H2, W2, C, generator=g)
    ref = orc.lookup4d_forward(f1.double(), [f2.double()], coords.double(), radius, C ** -0.5)
    out = ops.lookup4d_forward(f1.to(cuda_device), [f2.to(cuda_device)], coords.to(cuda_device), radius, C ** -0.5)
    assert ((out.double().cpu() - ref).norm() / ref.norm()).item() < TOL
    # positions beyond the image count as zero whatever the image holds: no window of these reaches row 0
    f2[0, 0] = float("inf")
    again = ops.lookup4d_forward(f1.to(cuda_device), [f2.to(cuda_device)], coords.to(cuda_device), radius, C ** -0.5)
    assert torch.equal(again, out)
