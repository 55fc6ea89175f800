"""The mean channels of a level on feature maps, whose mean rows keep a lane's columns in registers (widths up to 32, 64, 128,
256) or walk the plane twice (wider), around those widths and around the rows that eight warps take two at a time."""
import pytest
import torch

from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# operands rounded to 10 mantissa bits (2^-11 each way), FP32 accumulation: as tests/test_ops_gpu.py
TOL = 1e-3


@pytest.mark.parametrize("operands", ["fp16", "tf32"])
@pytest.mark.parametrize("size", [(1, 1), (7, 31), (8, 32), (9, 33), (16, 64), (17, 65), (15, 128), (33, 129), (8, 256), (5, 257), (40, 300)])
def test_means(size, operands, cuda_device):
    (H2, W2), (H1, W1), B, C, K = size, (3, 7), 2, 24, 1
    g = torch.Generator().manual_seed(H2 * 1000 + W2)
    f1, f2 = torch.randn(B, C, H1, W1, generator=g), torch.randn(B, C, H2, W2, generator=g) + 0.5
    params = [torch.zeros(K, 2, 3, 3, 3), torch.zeros(K), torch.zeros(K, 2, 3, 3, 3), torch.zeros(K)]
    with ops.sweep_operands(operands):
        sep_u, sep_v = ops.separation_level_forward(f1.to(cuda_device), f2.to(cuda_device), *[p.to(cuda_device) for p in params],
                                                    fmaps=True, scale1=0.25)[:2]
    S = torch.einsum("bcij,bcuv->buvij", f1.double() * 0.25, f2.double())
    for got, want in ((sep_v[:, 1], S.mean(2)), (sep_u[:, 1], S.mean(1))):
        assert ((got.double().cpu() - want).abs().max() / want.abs().max()).item() < TOL
