"""All pyramid levels in one call against the same levels one call at a time: the same bits, because neither the cut of a launch nor its
other levels enter a sum, around the edges of tiles (8 x 32 and 16 x 16), pixel tiles (128, 32 x 4), walks and softmax classes."""
import math

import pytest
import torch
import torch.nn.functional as F

from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu


def inputs(B, C, H, W, Kc, levels, seed, dev):
    g = torch.Generator().manual_seed(seed)
    f1, f2 = torch.randn(B, C, H, W, generator=g).to(dev), torch.randn(B, C, H, W, generator=g).to(dev)
    pyr = [f2]
    for _ in range(levels - 1):
        pyr.append(F.avg_pool2d(pyr[-1], 2, stride=2).contiguous())
    params = [p.to(dev) for _ in range(2) for p in (torch.randn(Kc, 2, 3, 3, 3, generator=g) * 0.2, torch.randn(Kc, generator=g) * 0.1)]
    return f1, pyr, params


def one_by_one(f1, pyr, params, with_argmax):
    B, C, H, W = f1.shape
    L, Kt = len(pyr), 2 + params[0].shape[0]
    sep_u = torch.empty(B, Kt * L, W, H, W, device=f1.device)
    sep_v = torch.empty(B, Kt * L, H, H, W, device=f1.device)
    saved = []
    for l, f2 in enumerate(pyr):
        place = (sep_u, sep_v, 0) if l == 0 else None
        su, sv, *rest = ops.separation_level_forward(f1, f2, *params, with_argmax, True, 1 / math.sqrt(C), place)
        if l > 0:
            ops.upsample_displacement_into(su, sep_u, l * Kt)
            ops.upsample_displacement_into(sv, sep_v, l * Kt)
        saved.append((su, sv, *rest))
    return sep_u, sep_v, saved


# (B, C, H, W, Kc, levels)
SHAPES = [(1, 32, 8, 32, 1, 2), (1, 64, 17, 33, 2, 3), (2, 64, 24, 40, 3, 4), (1, 256, 55, 128, 4, 4), (3, 40, 47, 155, 3, 2), (1, 128, 16, 24, 4, 4),
          (2, 256, 48, 64, 2, 4), (1, 36, 33, 31, 2, 2), (1, 64, 130, 36, 1, 4), (4, 64, 61, 130, 2, 3)]


@pytest.mark.parametrize("operands", ["fp16", "tf32", "bf16"])
@pytest.mark.parametrize("with_argmax", [True, False])
@pytest.mark.parametrize("shape", SHAPES)
def test_forward(shape, with_argmax, operands, cuda_device):
    B, C, H, W, Kc, levels = shape
    if operands == "bf16" and C % 8:
        pytest.skip("needs C % 8 == 0")
    f1, pyr, params = inputs(B, C, H, W, Kc, levels, H * W + Kc, cuda_device)
    with ops.sweep_operands(operands):
        sep_u, sep_v, buffer = ops.separation_pyramid_forward(f1, pyr, *params, with_argmax, 1 / math.sqrt(C))
        ref_u, ref_v, ref = one_by_one(f1, pyr, params, with_argmax)
    assert torch.equal(sep_u, ref_u) and torch.equal(sep_v, ref_v)
    for got, want in zip(ops.separation_pyramid_saved(buffer, f1, pyr, Kc, with_argmax), ref):
        for x, y in zip(got, want):
            assert (x is None) == (y is None) and (x is None or torch.equal(x, y))


# The feature gradients are sums over up to H*W pixels that the tensor core forms 8 (TF32) or 16 products at a time, each addition to the
# FP32 accumulator cut off at 2^-23 of it: other pieces of the sum, other errors, up to H*W / 8 * 2^-23 of the result.  Beside that
# (and for the parameters alone): sums over levels and blocks in another order, 2^-24 of a few hundred terms each; and FP16 operands may take
# another power of two where a level's gradients are searched without its neighbours', for values in FP16's subnormal range (2^-25 of
# the largest).
TOL = 2e-5


def relerr(x, ref):
    return ((x.double() - ref.double()).norm() / ref.double().norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("operands", ["fp16", "tf32", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
def test_backward(shape, operands, cuda_device):
    B, C, H, W, Kc, levels = shape
    if operands == "bf16" and C % 8:
        pytest.skip("needs C % 8 == 0")
    f1, pyr, params = inputs(B, C, H, W, Kc, levels, H * W + Kc, cuda_device)
    scale1, Kt, tol = 1 / math.sqrt(C), 2 + Kc, H * W / 8 * 2 ** -23 + TOL
    gen = torch.Generator().manual_seed(3)
    gu = torch.randn(B, Kt * levels, W, H, W, generator=gen).to(cuda_device)
    gv = torch.randn(B, Kt * levels, H, H, W, generator=gen).to(cuda_device)
    with ops.sweep_operands(operands):
        sep_u, sep_v, buffer = ops.separation_pyramid_forward(f1, pyr, *params, True, scale1)
        g1, g2, *gp = ops.separation_pyramid_backward(f1, pyr, params[0], params[2], sep_u, sep_v, buffer, gu, gv, scale1)
        _, _, saved = one_by_one(f1, pyr, params, True)
        ref1, refp = 0, [0, 0, 0, 0]
        for l, (f2, (su, sv, am_u, am_v, a_u, a_v)) in enumerate(zip(pyr, saved)):
            if l == 0:
                out = ops.separation_level_backward(f1, f2, params[0], params[2], sep_u, sep_v, am_u, am_v, a_u, a_v, gu, gv, True, scale1, 0)
            else:
                gsu = ops.upsample_displacement_backward(gu, l * Kt, Kt, su.shape[2])
                gsv = ops.upsample_displacement_backward(gv, l * Kt, Kt, sv.shape[2])
                out = ops.separation_level_backward(f1, f2, params[0], params[2], su, sv, am_u, am_v, a_u, a_v, gsu, gsv, True, scale1)
            assert relerr(g2[l], out[1]) < tol
            ref1 = ref1 + out[0].double()
            refp = [r + p.double() for r, p in zip(refp, out[2:])]
        again = ops.separation_pyramid_backward(f1, pyr, params[0], params[2], sep_u, sep_v, buffer, gu, gv, scale1)
    assert relerr(g1, ref1) < tol
    # a softmax does not see its bias: those gradients are rounding
    assert relerr(gp[0], refp[0]) < TOL and relerr(gp[2], refp[2]) < TOL
    assert torch.equal(again[0], g1) and all(torch.equal(x, y) for x, y in zip(again[1], g2)) and all(torch.equal(x, y) for x, y in zip(again[2:], gp))


# One batch with an odd side at every level, one whose planes are not read 16 bytes at a time, one that ends inside an 8 x 8 region
@pytest.mark.parametrize("operands", ["fp16", "tf32"])
@pytest.mark.parametrize("shape", SHAPES + [(1, 32, 15, 23, 1, 4), (2, 32, 9, 13, 2, 3), (1, 64, 31, 60, 2, 4)])
def test_pooled_levels(shape, operands, cuda_device):
    """The pyramid made by the library is avg_pool2d's, bit for bit, and its gradient that of the chain of avg_pool2d."""
    B, C, H, W, Kc, levels = shape
    f1, pyr, params = inputs(B, C, H, W, Kc, levels, H + W, cuda_device)
    scale1, Kt = 1 / math.sqrt(C), 2 + Kc
    gen = torch.Generator().manual_seed(4)
    gu = torch.randn(B, Kt * levels, W, H, W, generator=gen).to(cuda_device)
    gv = torch.randn(B, Kt * levels, H, H, W, generator=gen).to(cuda_device)
    with ops.sweep_operands(operands):
        sep_u, sep_v, buffer = ops.separation_pyramid_forward(f1, pyr[:1], *params, True, scale1, levels)
        ref_u, ref_v, ref_buffer = ops.separation_pyramid_forward(f1, pyr, *params, True, scale1)
        assert torch.equal(sep_u, ref_u) and torch.equal(sep_v, ref_v)
        g1, (g2,), *gp = ops.separation_pyramid_backward(f1, pyr[:1], params[0], params[2], sep_u, sep_v, buffer, gu, gv, scale1, levels)
        r1, r2, *rp = ops.separation_pyramid_backward(f1, pyr, params[0], params[2], ref_u, ref_v, ref_buffer, gu, gv, scale1)
    assert torch.equal(g1, r1) and all(torch.equal(x, y) for x, y in zip(gp, rp))
    f2 = pyr[0].clone().requires_grad_(True)
    chain = [f2]
    for _ in range(levels - 1):
        chain.append(F.avg_pool2d(chain[-1], 2, stride=2))
    (ref2,) = torch.autograd.grad(chain, f2, r2)
    assert relerr(g2, ref2) < 1e-6   # the same additions, in an order of autograd's choice


def test_block_pyramid_on_demand(cuda_device):
    """The differentiable levels of a block are made when they are read, with the grad mode the block was made in."""
    import separableflowthesis_b200 as sfb
    f1, pyr, _ = inputs(1, 32, 16, 24, 2, 3, 1, cuda_device)
    f2 = pyr[0].requires_grad_(True)
    block = sfb.AlternateCorrBlockSepflow(f1, f2, None, num_levels=3)
    with torch.no_grad():
        levels = block.pyramid
    assert all(torch.equal(x, y) for x, y in zip(levels, pyr)) and levels[2].requires_grad and block.pyramid is levels
    with torch.no_grad():
        block = sfb.AlternateCorrBlockSepflow(f1, f2, None, num_levels=3)
    assert not block.pyramid[1].requires_grad
    with pytest.raises(RuntimeError):
        sfb.AlternateCorrBlockSepflow(f1, f2, None, num_levels=6)


@pytest.mark.parametrize("shape", [(1, 32, 16, 24, 2, 3), (2, 64, 17, 33, 1, 4), (2, 32, 15, 31, 2, 2), (1, 36, 40, 60, 4, 4)])
@pytest.mark.parametrize("layout", ["contiguous", "channels_last", "off a 16-byte boundary"])
def test_block_takes_its_pyramid_when_made(shape, layout, cuda_device):
    """The coarser levels are those of the maps as they are in the constructor (core/corr.py:377-382), whatever is written to them later,
    and whether or not `pyramid` is read in between; level 0 is the maps themselves."""
    import separableflowthesis_b200 as sfb
    B, C, H, W, Kc, levels = shape
    f1, pyr, params = inputs(B, C, H, W, Kc, levels, H + W, cuda_device)
    modules = []
    for i in (0, 2):
        m = torch.nn.Conv3d(2, Kc, 3, padding=1).to(cuda_device)
        with torch.no_grad():
            m.weight.copy_(params[i])
            m.bias.copy_(params[i + 1])
        modules.append(m)
    f2 = pyr[0]
    if layout == "channels_last":
        f2 = f2.contiguous(memory_format=torch.channels_last)
    elif layout != "contiguous":
        f2 = torch.empty(f2.numel() + 1, device=cuda_device)[1:].view_as(f2).copy_(f2)
    for read in (False, True):
        with torch.no_grad():
            maps = f2.clone() if layout != "off a 16-byte boundary" else torch.empty(f2.numel() + 1, device=cuda_device)[1:].view_as(f2).copy_(f2)
            block = sfb.AlternateCorrBlockSepflow(f1, maps, None, num_levels=levels)
            maps.mul_(-0.5)
            if read:
                assert all(torch.equal(x, y) for x, y in zip(block.pyramid[1:], pyr[1:])) and block.pyramid[0] is maps
            if layout == "off a 16-byte boundary":   # the library refuses such a level 0, as it always did
                with pytest.raises(RuntimeError, match="aligned"):
                    block(None, sep=True, attention_weights=modules)
                continue
            got = block(None, sep=True, attention_weights=modules)
            want = ops.separation_pyramid_forward(f1, [(-0.5 * pyr[0]).contiguous(), *pyr[1:]], *params, False, 1 / math.sqrt(C))
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("shape", [(1, 32, 16, 24, 2, 3), (2, 64, 17, 33, 1, 4)])
def test_block_gradients(shape, cuda_device):
    """One call for all levels and their averages, and the same through the levels as tensors: equal gradients; a write to the maps
    between forward and backward is noticed; the levels' gradients are avg_pool2d's, to the second derivative."""
    import separableflowthesis_b200 as sfb
    B, C, H, W, Kc, levels = shape
    f1, pyr, _ = inputs(B, C, H, W, Kc, levels, H + W, cuda_device)
    modules = [torch.nn.Conv3d(2, Kc, 3, padding=1).to(cuda_device) for _ in range(2)]
    grads = []
    for read in (False, True):
        f2 = pyr[0].clone().requires_grad_(True)
        block = sfb.AlternateCorrBlockSepflow(f1, f2, None, num_levels=levels, support_backward=True)
        if read:
            block.pyramid
        u, v = block(None, sep=True, attention_weights=modules)
        grads.append(torch.autograd.grad((u * u).sum() + v.sum(), [f2, modules[0].weight, modules[1].weight]))
    assert all(relerr(x, y) < 1e-6 for x, y in zip(*grads))
    for read in (False, True):
        f2 = pyr[0].clone().requires_grad_(True)
        block = sfb.AlternateCorrBlockSepflow(f1, f2, None, num_levels=levels, support_backward=True)
        if read:
            block.pyramid
        loss = sum(x.sum() for x in block(None, sep=True, attention_weights=modules))
        f2.data.add_(0)   # not tracked
        with torch.no_grad():
            f2.add_(0)
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            loss.backward()
    f2 = pyr[0].clone().requires_grad_(True)
    made = sfb.AlternateCorrBlockSepflow(f1, f2, None, num_levels=levels).pyramid
    chain = [f2]
    for _ in range(levels - 1):
        chain.append(F.avg_pool2d(chain[-1], 2, stride=2))
    for p in (made, chain):   # a write to a level reaches neither the others nor the maps
        p[-1].mul_(1.5)
    assert all(torch.equal(x, y) for x, y in zip(made, chain))
    inner = [torch.autograd.grad([(t * t).sum() for t in p], p[1], retain_graph=True)[0] for p in (made, chain)]
    assert torch.equal(*inner)
    first = [torch.autograd.grad([(t * t * t).sum() for t in p], f2, create_graph=True)[0] for p in (made, chain)]
    assert torch.equal(*first)
    assert torch.equal(*[torch.autograd.grad((g * g).sum(), f2)[0] for g in first])
