"""Both aggregated volumes looked up by one call, and the gradients of several lookups summed in one accumulator per volume: against
the single-volume ops and the oracle, around the edges of pixel groups, vectors of four pixels, pyramid stages and windows."""
import pytest
import torch

import separableflowthesis_b200 as sfb
from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# FP32 interpolation of two values at positions of up to D = 40 (tests/test_ops_gpu.py, LOOKUP_TOL); a gradient adds up at most
# ITERATIONS * 4 levels * 2 products more, each rounded to 2^-24 of a value no larger than the sum's terms
TOL = 5e-5
ITERATIONS = 3


def relerr(x, ref):
    return ((x.double().cpu() - ref.double().cpu()).abs().max() / ref.double().abs().max().clamp_min(1e-30)).item()


def inputs(B, dim, H, W, seed):
    g = torch.Generator().manual_seed(seed)
    vols = [torch.randn(B, dim, W, H, W, generator=g), torch.randn(B, dim, H, H, W, generator=g)]
    coords = [torch.rand(B, 2, H, W, generator=g) * (max(H, W) + 12) - 6 for _ in range(ITERATIONS)]
    coords[0].view(-1)[0], coords[1].view(-1)[-1] = 3.0, float("nan")
    return vols, coords, g


# (B, dim, H, W, levels, radius)
SHAPES = [(1, 1, 2, 3, 1, 4), (2, 1, 8, 9, 3, 4), (1, 2, 17, 21, 4, 4), (1, 2, 9, 17, 3, 4), (2, 1, 16, 16, 4, 4), (1, 1, 33, 40, 5, 4), (1, 1, 9, 11, 2, 0),
          (2, 1, 12, 20, 3, 2), (1, 2, 17, 16, 4, 6)]


@pytest.mark.parametrize("shape", SHAPES)
def test_against_single_volumes_and_oracle(shape, cuda_device):
    B, dim, H, W, levels, radius = shape
    vols, coords, g = inputs(B, dim, H, W, 7 * H + W)
    dev_vols = [v.to(cuda_device).requires_grad_(True) for v in vols]
    block = sfb.CorrBlock1D(*dev_vols, num_levels=levels, radius=radius)
    size = (B, levels * dim * (2 * radius + 1), H, W)
    gouts = [[torch.randn(size, generator=g) for _ in range(2)] for _ in coords]
    outs = [block(c.to(cuda_device)) for c in coords]
    grads = torch.autograd.grad([o for pair in outs for o in pair], dev_vols, [x.to(cuda_device) for pair in gouts for x in pair])
    for i, clamp in enumerate((True, False)):
        vol = dev_vols[i].detach()
        pyr = ops.lookup_build_pyramid(vol, levels)
        total = 0
        for c, pair, gout in zip(coords, outs, gouts):
            assert torch.equal(pair[i].nan_to_num(7.0), ops.lookup_forward(vol, pyr, c.to(cuda_device)[:, i], levels, radius, clamp).nan_to_num(7.0))
            total = total + ops.lookup_backward(tuple(vol.shape), c.to(cuda_device)[:, i], gout[i].to(cuda_device), levels, radius, clamp).double()
        # a NaN position samples nothing and gets nothing: no NaN in either
        assert torch.isfinite(total).all() and torch.isfinite(grads[i]).all()
        assert relerr(grads[i], total) < TOL
    # a NaN coordinate is the single-volume op's business; the oracle sees the lookups without it
    clean = [torch.nan_to_num(c, nan=1.5) for c in coords]
    block = sfb.CorrBlock1D(*dev_vols, num_levels=levels, radius=radius)
    outs = [block(c.to(cuda_device)) for c in clean]
    grads = torch.autograd.grad([o for pair in outs for o in pair], dev_vols, [x.to(cuda_device) for pair in gouts for x in pair])
    for i, clamp in enumerate((True, False)):
        ref = sum(orc.lookup_backward(vols[i].shape, c[:, i].double(), gout[i].double(), levels, radius, clamp) for c, gout in zip(clean, gouts))
        assert relerr(grads[i], ref) < TOL
        for c, pair in zip(clean, outs):
            assert relerr(pair[i], orc.lookup_forward(vols[i].double(), c[:, i].double(), levels, radius, clamp)) < TOL


def test_autograd_of_a_chain(cuda_device):
    """What autograd gave for independent lookups: a backward per lookup, volumes that are not reached, one volume that needs no
    gradient, lookups without grad in between, several chains."""
    vols, coords, g = inputs(2, 1, 16, 18, 5)
    coords = [torch.nan_to_num(c, nan=1.5).to(cuda_device) for c in coords]
    v1, v2 = [v.to(cuda_device).requires_grad_(True) for v in vols]
    ref = []
    for c in coords:   # every lookup by itself
        o1, o2 = sfb.CorrBlock1D(v1, v2)(c)
        ref.append((o1, o2, *torch.autograd.grad([o1.sum() + (o2 * o2).sum()], [v1, v2])))
    block = sfb.CorrBlock1D(v1, v2)
    outs = []
    for c in coords:
        outs.append(block(c))
        with torch.no_grad():
            assert not block(c)[0].requires_grad
    for (o1, o2), r in zip(outs, ref):   # one backward per lookup, none of them retaining the graph
        assert torch.equal(o1, r[0]) and torch.equal(o2, r[1])
        g1, g2 = torch.autograd.grad([o1.sum() + (o2 * o2).sum()], [v1, v2])
        assert torch.equal(g1, r[2]) and torch.equal(g2, r[3])
    outs = [block(c) for c in coords]
    loss = sum(o1.sum() + (o2 * o2).sum() for o1, o2 in outs)
    first = torch.autograd.grad(loss, [v1, v2], retain_graph=True)
    again = torch.autograd.grad(loss, [v1, v2])
    for i in range(2):
        assert torch.equal(first[i], again[i])
        assert relerr(first[i], sum(r[2 + i].double() for r in ref)) < TOL
    # only one output reaches the loss: the other volume was not used
    g1, g2 = torch.autograd.grad(block(coords[0])[0].sum(), [v1, v2], allow_unused=True)
    assert g2 is None and torch.equal(g1, ref[0][2])
    # a volume without gradient
    o1, o2 = sfb.CorrBlock1D(v1.detach(), v2)(coords[0])
    assert not o1.requires_grad and o2.requires_grad
    (g2,) = torch.autograd.grad((o2 * o2).sum(), [v2])
    assert torch.equal(g2, ref[0][3])
    # coordinates that need a gradient get none, whatever the volumes need
    for vols in ((v1.detach(), v2.detach()), (v1, v2.detach()), (v1.detach(), v2)):
        c = coords[0].clone().requires_grad_(True)
        o1, o2 = sfb.CorrBlock1D(*vols)(c)
        got = torch.autograd.grad((o1 * o1).sum() + o2.sum(), [c] + [v for v in vols if v.requires_grad], allow_unused=True)
        assert got[0] is None and all(x is not None for x in got[1:])
    # chains of two lookups
    block = sfb.CorrBlock1D(v1, v2)
    block.CHAIN = 2
    got = torch.autograd.grad(sum(o1.sum() + (o2 * o2).sum() for o1, o2 in (block(c) for c in coords)), [v1, v2])
    for i in range(2):
        assert relerr(got[i], sum(r[2 + i].double() for r in ref)) < TOL
    with pytest.raises(RuntimeError):
        block(coords[0][:, :, ::2])
    with pytest.raises(RuntimeError):
        block(coords[0].double())
