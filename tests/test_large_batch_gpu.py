"""Batches of many small images through the fused channels-first backward, where a launch that puts several operands on one grid
axis with the batch would run out of that axis (65535 blocks).  Whole numbers throughout: the results are exact."""
import pytest
import torch

from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Kc", [(10922, 4), (10923, 4), (16384, 2), (20000, 6)])
def test_fused_backward(B, Kc, cuda_device):
    H1, W1, H2, W2, C = 1, 2, 2, 4, 8
    g = torch.Generator(device=cuda_device).manual_seed(B)
    ints = lambda lo, hi, *s: torch.randint(lo, hi + 1, s, generator=g, device=cuda_device).float()
    F1, F2 = ints(-2, 2, B, H1, W1, C), ints(-2, 2, B, H2, W2, C)
    a_u, a_v = ints(0, 2, B, Kc, W2, H1, W1), ints(0, 2, B, Kc, H2, H1, W1)
    gc_u, gc_v = ints(-2, 2, B, Kc, H2, H1, W1), ints(-2, 2, B, Kc, W2, H1, W1)
    g_v, g_u = ints(-3, 3, B, 2, H2, H1, W1), ints(-3, 3, B, 2, W2, H1, W1)   # channel 0: maxima, 1: means
    am_u = torch.randint(0, W2, (B, H2, H1, W1), generator=g, device=cuda_device, dtype=torch.int32)
    am_v = torch.randint(0, H2, (B, W2, H1, W1), generator=g, device=cuda_device, dtype=torch.int32)
    gF1, gF2 = ops.separation_feature_backward_cf(F1, F2, am_u, am_v, g_v, g_u, a_u, a_v, gc_u, gc_v)
    G = torch.einsum("bkuij,bkvij->bijuv", gc_u, a_u) + torch.einsum("bkuij,bkvij->bijuv", a_v, gc_v)
    pixels_first = lambda t: t.permute(0, 2, 3, 1)
    G += pixels_first(g_v[:, 1])[..., None] / W2 + pixels_first(g_u[:, 1])[..., None, :] / H2
    G.scatter_add_(4, pixels_first(am_u)[..., None].long(), pixels_first(g_v[:, 0])[..., None])
    G.scatter_add_(3, pixels_first(am_v)[..., None, :].long(), pixels_first(g_u[:, 0])[..., None, :])
    G, F1, F2 = G.double(), F1.double(), F2.double()
    assert torch.equal(gF1.double(), (G[..., None] * F2[:, None, None]).sum((3, 4)))
    assert torch.equal(gF2.double(), (G[..., None] * F1[:, :, :, None, None]).sum((1, 2)))
