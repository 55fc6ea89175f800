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


# The gradients of image 1 are summed over the levels tile by tile: 16 384 x 4 of 128 pixels and more than 65535 of them.  C = 4 runs with
# TF32 operands and never hands G over, in parts of the batch or otherwise.
@pytest.mark.parametrize("B", [16384, 16390])
def test_pyramid_backward(B, cuda_device):
    C, H1, W1, Kc, sizes = 4, 16, 25, 1, [(2, 4), (1, 2)]
    Kt, dev = 2 + Kc, cuda_device
    g = torch.Generator(device=dev).manual_seed(B)
    randn = lambda *s: torch.randn(*s, generator=g, device=dev)
    f1, pyr = randn(B, C, H1, W1), [randn(B, C, h, w) for h, w in sizes]
    params = [randn(Kc, 2, 3, 3, 3) * 0.2, randn(Kc) * 0.1, randn(Kc, 2, 3, 3, 3) * 0.2, randn(Kc) * 0.1]
    gu, gv = randn(B, 2 * Kt, 4, H1, W1), randn(B, 2 * Kt, 2, H1, W1)

    def both(part):
        maps = f1[part].contiguous(), [f2[part].contiguous() for f2 in pyr]
        sep_u, sep_v, buffer = ops.separation_pyramid_forward(*maps, *params, True, 0.5)
        return ops.separation_pyramid_backward(*maps, params[0], params[2], sep_u, sep_v, buffer, gu[part].contiguous(), gv[part].contiguous(), 0.5)

    whole = both(slice(None))
    parts = [both(slice(i, i + 4100)) for i in range(0, B, 4100)]
    # per sample: the same products, sums of up to 400 or 10 of them in other pieces (2^-23 of the result each)
    relerr = lambda x, ref: ((x.double() - ref.double()).norm() / ref.double().norm()).item()
    assert relerr(whole[0], torch.cat([p[0] for p in parts])) < 400 * 2 ** -23
    for l in range(2):
        assert relerr(whole[1][l], torch.cat([p[1][l] for p in parts])) < 400 * 2 ** -23
    for i in (2, 4):   # parameters: sums over the batch, in the order of blocks and of parts (2^-24 of a few thousand terms that cancel)
        assert relerr(whole[i], sum(p[i].double() for p in parts)) < 1e-4
