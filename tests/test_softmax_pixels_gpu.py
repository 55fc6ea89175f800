"""The softmax over the displacement axis with one, two and four pixels a lane: launches that fill the device and planes of a
multiple of four pixels take more than one up to 192 displacements; a sample alone and planes of other sizes take one."""
import pytest
import torch

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# FP32 sums of 54 products, then a softmax.
TOL = 2e-5


# last displacement of each class of lengths (8 warps of 4, 8, 16, 20, 24, 32 values, or any number), and the first of the next
@pytest.mark.parametrize("D", [9, 32, 33, 64, 65, 128, 129, 160, 161, 192, 193, 256, 257])
@pytest.mark.parametrize("H1,W1", [(40, 64), (39, 66), (41, 63), (44, 59)])
def test_pixels_of_a_lane(D, H1, W1, cuda_device):
    B, Kc = 4, 2
    g = torch.Generator().manual_seed(D + W1)
    x = torch.randn(B, 2, D, H1, W1, generator=g)
    weight, bias = torch.randn(Kc, 2, 3, 3, 3, generator=g) * 0.3, torch.randn(Kc, generator=g)
    x[0, :, :, 3, 5] = 40.0   # logits of some tens
    args = (weight.to(cuda_device), bias.to(cuda_device))
    a = ops.attention_forward(x.to(cuda_device), *args)
    ref = orc.attention_forward(x[:1].double(), weight.double(), bias.double())
    error = (a[:1].double().cpu() - ref).abs().amax(dim=(1, 2)) / ref.abs().amax(dim=(1, 2))
    assert error.max().item() < 50 * TOL   # the logits beside the spike are ten times the others'
    for b in range(B):
        assert torch.equal(a[b:b + 1], ops.attention_forward(x[b:b + 1].to(cuda_device), *args))
    x[1, 0, D // 2, 7, 9] = float("nan")
    x[2, 1, D - 1, 8, 8] = float("inf")
    b = ops.attention_forward(x.to(cuda_device), *args)
    for i in range(B):
        assert torch.equal(b[i:i + 1].nan_to_num(7.0), ops.attention_forward(x[i:i + 1].to(cuda_device), *args).nan_to_num(7.0))
