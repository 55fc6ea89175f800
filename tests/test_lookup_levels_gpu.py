"""Forward lookup on the aggregated volumes for every number of pyramid levels, which decides how a block's warps are shared
out over levels and groups of 32 pixels: pixel counts around the groups' edges, the compiled radius and another one."""
import pytest
import torch

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# FP32 interpolation of two values at positions of up to 260: as LOOKUP_TOL of tests/test_ops_gpu.py
TOL = 5e-5


@pytest.mark.parametrize("levels", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("radius", [2, 4])
@pytest.mark.parametrize("plane", [(1, 1), (1, 31), (4, 8), (3, 11), (1, 64), (5, 13), (1, 127), (8, 16), (3, 43)])
def test_levels(levels, radius, plane, cuda_device):
    (H1, W1), B, dim, D = plane, 2, 2, 260
    g = torch.Generator().manual_seed(levels * 100 + H1 * W1)
    corr = torch.randn(B, dim, D, H1, W1, generator=g)
    coords = torch.rand(B, H1, W1, generator=g) * (D + 12) - 6
    corr_d = corr.to(cuda_device)
    out = ops.lookup_forward(corr_d, ops.lookup_build_pyramid(corr_d, levels), coords.to(cuda_device), levels, radius, False)
    ref = orc.lookup_forward(corr.double(), coords.double(), levels, radius, False)
    assert out.shape == ref.shape
    assert ((out.double().cpu() - ref).abs().max() / ref.abs().max()).item() < TOL
