"""Displacement resampling and its adjoint at the edges of the eight-row pieces and of the four-pixel form: one row, seven to
nine and fifteen to seventeen rows, equal sizes, ratios from one to many, pixel counts that are and are not multiples of 4."""
import pytest
import torch
import torch.nn.functional as F

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# positions d*(Dl-1)/(D0-1) are formed in float32, as in torch's own float32 kernel: ~D0 * 2^-24
TOL = 2e-5


@pytest.mark.parametrize("plane", [(3, 5), (4, 6), (9, 60)])
@pytest.mark.parametrize("sizes", [(1, 1), (1, 9), (2, 3), (7, 8), (8, 8), (8, 9), (9, 17), (15, 31), (16, 33), (17, 240), (33, 34), (67, 135)])
def test_rows(sizes, plane, cuda_device):
    (Dl, D0), (H1, W1), (B, K) = sizes, plane, (2, 3)
    g = torch.Generator().manual_seed(Dl * 1000 + D0)
    src = torch.randn(B, K, Dl, H1, W1, generator=g)
    dst = torch.full((B, K + 2, D0, H1, W1), 7.0, device=cuda_device)
    ops.upsample_displacement_into(src.to(cuda_device), dst, 1)
    ref = F.interpolate(src.double(), [D0, H1, W1], mode="trilinear", align_corners=True)
    assert (dst[:, 1:1 + K].double().cpu() - ref).abs().max() < TOL * ref.abs().max()
    assert (dst[:, :1] == 7.0).all() and (dst[:, 1 + K:] == 7.0).all()
    gd = torch.randn(B, K + 2, D0, H1, W1, generator=g)
    gs = ops.upsample_displacement_backward(gd.to(cuda_device), 1, K, Dl)
    rs = orc.upsample_displacement_backward(gd.double(), 1, K, Dl)
    assert (gs.double().cpu() - rs).abs().max() < TOL * rs.abs().max()


@pytest.mark.parametrize("sizes", [(8, 9), (9, 17), (16, 16), (17, 240), (33, 34)])
def test_whole_columns_give_what_pieces_give(sizes, cuda_device):
    """Launches with blocks enough to fill the GPU walk whole columns, smaller ones pieces of rows: the same sums."""
    (Dl, D0), (H1, W1), (B, K) = sizes, (3, 5), (2, 444)   # 888 blocks: whole columns
    g = torch.Generator().manual_seed(Dl)
    gd = torch.randn(B, K + 1, D0, H1, W1, generator=g).to(cuda_device)
    whole = ops.upsample_displacement_backward(gd, 1, K, Dl)
    pieces = torch.cat([ops.upsample_displacement_backward(gd, 1 + k0, K // 4, Dl) for k0 in range(0, K, K // 4)], 1)
    assert torch.equal(whole, pieces)
    rs = orc.upsample_displacement_backward(gd.double().cpu(), 1, K, Dl)
    assert (whole.double().cpu() - rs).abs().max() < TOL * rs.abs().max()
