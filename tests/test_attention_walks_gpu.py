"""The attention kernels where their work is cut along the displacement axis and where the softmax changes the number of
values a thread keeps: one displacement, the shortest piece, the edges of the register variants (32, 64, 128, 256
displacements) and beyond, for the gather form and for the TMA tiles (image-1 widths that are a multiple of 4)."""
import pytest
import torch

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# Weights relative to their norm.  A logit is an FP32 sum of 54 products of about 0.3: roundings of 2^-24 of a running sum of
# a few units, sqrt(54) of them, up to 2e-6, which is the relative error it gives its weight.  __expf(x) is within
# 2 + floor(abs(1.173 x)) ulp (its documented bound): 4 ulp = 5e-7 for the weights near a column's maximum, which carry the
# norm, 13 ulp at x = -10, where a weight is 5e-5 of them.  The sum of up to 300 weights adds sqrt(300) 2^-24 = 1e-6.  About
# 4e-6 in all; the gradients pass through two such sums more.
TOL = 2e-5
DS = [1, 2, 7, 8, 9, 17, 32, 33, 64, 65, 128, 129, 256, 257, 300]


def relerr(a, b):
    return ((a.double().cpu() - b).norm() / b.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("D", DS)
@pytest.mark.parametrize("shape", [(1, 2, 3, 5), (2, 5, 6, 33)])
def test_gather_form(shape, D, cuda_device):
    B, Kc, H1, W1 = shape
    g = torch.Generator().manual_seed(100 + D)
    x = torch.randn(B, 2, D, H1, W1, generator=g)
    weight, bias = torch.randn(Kc, 2, 3, 3, 3, generator=g) * 0.3, torch.randn(Kc, generator=g)
    a = ops.attention_forward(x.to(cuda_device), weight.to(cuda_device), bias.to(cuda_device))
    ref = orc.attention_forward(x.double(), weight.double(), bias.double())
    assert relerr(a, ref) < TOL
    assert (a.sum(dim=2) - 1).abs().max().item() < 1e-5
    ga, add = torch.randn(a.shape, generator=g), torch.randn(x.shape, generator=g)
    gx, gw, gb = ops.attention_backward(x.to(cuda_device), weight.to(cuda_device), a, ga.to(cuda_device),
                                        add.to(cuda_device))
    r_gx, r_gw, r_gb = orc.attention_backward(x.double(), weight.double(), a.double().cpu(), ga.double(), add.double())
    assert relerr(gx, r_gx) < TOL
    if D > 1:   # a softmax over one entry has no gradient: the reference is zero up to rounding
        assert relerr(gw, r_gw) < TOL
    assert (gb.double().cpu() - r_gb).abs().max().item() < TOL * max(r_gw.abs().max().item(), 1.0)


@pytest.mark.parametrize("size", [(5, 36, 1, 7), (8, 32, 9, 33), (4, 4, 17, 65), (6, 68, 64, 129), (9, 40, 130, 257)])
@pytest.mark.parametrize("Kc", [1, 3, 4, 6])
def test_tiles(size, Kc, cuda_device):
    """The weights a level call returns against the oracle's attention of the max/mean channels it returns."""
    H1, W1, H2, W2 = size
    g = torch.Generator().manual_seed(7 * Kc + H2)
    F1, F2 = torch.randn(1, H1, W1, 16, generator=g) / 4, torch.randn(1, H2, W2, 16, generator=g)
    params = [torch.randn(Kc, 2, 3, 3, 3, generator=g) * 0.3, torch.randn(Kc, generator=g),
              torch.randn(Kc, 2, 3, 3, 3, generator=g) * 0.3, torch.randn(Kc, generator=g)]
    sep_u, sep_v, _, _, a_u, a_v = ops.separation_level_forward(F1.to(cuda_device), F2.to(cuda_device),
                                                                *[p.to(cuda_device) for p in params])
    for sep, a, w, b in ((sep_u, a_u, params[0], params[1]), (sep_v, a_v, params[2], params[3])):
        ref = orc.attention_forward(sep[:, :2].double().cpu(), w.double(), b.double())
        assert relerr(a, ref) < TOL


@pytest.mark.parametrize("D", [1, 3, 8, 9, 16, 17, 31, 160, 161, 192, 193])
def test_a_sample_alone_and_in_a_batch(D, cuda_device):
    """How the forward's walk is cut, and whether it ends with the softmax itself (short columns, launches of many blocks) or
    leaves it to the kernel of its own, follows the number of blocks: the weights of a sample are the same bits either way.
    Its gradients depend on D only as well."""
    B, Kc, H1, W1 = 7, 3, 45, 131
    g = torch.Generator().manual_seed(D)
    x = torch.randn(B, 2, D, H1, W1, generator=g).to(cuda_device)
    weight, bias = (torch.randn(Kc, 2, 3, 3, 3, generator=g) * 0.3).to(cuda_device), torch.randn(Kc, generator=g).to(cuda_device)
    ga = torch.randn(B, Kc, D, H1, W1, generator=g).to(cuda_device)
    a = ops.attention_forward(x, weight, bias)
    gx = ops.attention_backward(x, weight, a, ga)[0]
    for b in (0, B - 1):
        ab = ops.attention_forward(x[b:b + 1].contiguous(), weight, bias)
        assert torch.equal(a[b:b + 1], ab)
        assert torch.equal(gx[b:b + 1], ops.attention_backward(x[b:b + 1].contiguous(), weight, ab, ga[b:b + 1].contiguous())[0])
    ref = orc.attention_forward(x[:1].double().cpu(), weight.double().cpu(), bias.double().cpu())
    assert relerr(a[:1], ref) < TOL
    r_gx = orc.attention_backward(x[:1].double().cpu(), weight.double().cpu(), a[:1].double().cpu(), ga[:1].double().cpu(), None)[0]
    if D > 1:
        assert relerr(gx[:1], r_gx) < TOL


@pytest.mark.parametrize("H1,W1,H2,W2,Kc", [(55, 128, 55, 128, 4), (55, 128, 20, 9, 1), (135, 240, 33, 135, 3), (135, 240, 135, 240, 2)])
def test_tiles_agree_between_repeated_calls(H1, W1, H2, W2, Kc, cuda_device):
    """Many planes through the rings of the tiled kernels (level calls on widths that are multiples of 4), on many blocks at once:
    the same weights, and the same gradients that pass through them, every time."""
    g = torch.Generator(device=cuda_device).manual_seed(9)
    randn = lambda *s: torch.randn(*s, generator=g, device=cuda_device)
    F1, F2 = randn(2, H1, W1, 16) / 4, randn(2, H2, W2, 16)
    w_u, b_u, w_v, b_v = randn(Kc, 2, 3, 3, 3) * 0.3, randn(Kc), randn(Kc, 2, 3, 3, 3) * 0.3, randn(Kc)
    g_u, g_v = randn(2, 2 + Kc, W2, H1, W1), randn(2, 2 + Kc, H2, H1, W1)

    def run():
        level = ops.separation_level_forward(F1, F2, w_u, b_u, w_v, b_v)
        return level + ops.separation_level_backward(F1, F2, w_u, w_v, *level, g_u, g_v)

    first = run()
    for _ in range(6):
        for p, q in zip(first, run()):
            assert torch.equal(p, q)
