"""The host side of the lookups on both aggregated volumes: the native module refuses what the ops refuse, and a lookup that needs no gradient
goes past the autograd Function only where that Function would not have had a say."""
import pytest
import torch

import separableflowthesis_b200 as sfb
from separableflowthesis_b200 import _lib, corr, functions, ops

LEVELS, RADIUS = 2, 2


class Ops:
    @staticmethod
    def lookup_build_pyramid_pair(corr1, corr2, levels):
        return None, None

    @staticmethod
    def lookup_forward_pair(corr1, corr2, pyramid1, pyramid2, coords, levels, radius):
        size = (coords.shape[0], levels * (2 * radius + 1), *coords.shape[2:])
        return coords.new_zeros(size), coords.new_ones(size)


@pytest.fixture()
def block(monkeypatch):
    monkeypatch.setattr(functions, "MemorySaver", Ops)
    monkeypatch.setattr(corr, "_ops", Ops)
    return sfb.CorrBlock1D(torch.zeros(1, 1, 5, 4, 5), torch.zeros(1, 1, 4, 4, 5), num_levels=LEVELS, radius=RADIUS)


def test_without_gradients_the_function_is_not_entered(block, monkeypatch):
    def entered(*args):
        raise AssertionError("entered")

    monkeypatch.setattr(functions.LookupPairFunction, "forward", staticmethod(entered))
    coords = torch.zeros(1, 2, 4, 5)
    out1, out2 = block(coords)
    assert not out1.requires_grad and not out2.requires_grad
    with torch.no_grad():
        block(coords.requires_grad_(True))
    with pytest.raises(AssertionError):   # coordinates that need a gradient: the outputs have to require one
        block(coords)


def test_transforms_and_forward_mode_reach_the_function(block):
    coords = torch.zeros(3, 1, 2, 4, 5)
    with torch.no_grad(), pytest.raises(RuntimeError, match="vmap"):
        torch.func.vmap(lambda c: block(c)[0])(coords)
    with torch.autograd.forward_ad.dual_level(), torch.no_grad():
        dual = torch.autograd.forward_ad.make_dual(coords[0], torch.ones_like(coords[0]))
        entered = []
        forward = functions.LookupPairFunction.forward
        functions.LookupPairFunction.forward = staticmethod(lambda *a: entered.append(1) or forward(*a))
        try:
            block(dual)
        except RuntimeError:
            pass   # what torch says to a Function without a forward-mode derivative
        finally:
            functions.LookupPairFunction.forward = staticmethod(forward)
    assert entered


@pytest.mark.parametrize("owner, name", [(torch._C, "_are_functorch_transforms_active"), (torch.autograd.forward_ad, "_current_level")])
def test_a_torch_without_the_switches_counts_as_active(monkeypatch, owner, name):
    assert not corr._transforms_active()
    monkeypatch.delattr(owner, name)
    assert corr._transforms_active()


def test_traces_reach_the_function(block):
    """A trace would record a direct call as the allocation of its outputs, without the lookup."""
    coords = torch.zeros(1, 2, 4, 5)
    with torch.no_grad():
        traced = torch.jit.trace(lambda c: block(c), (coords,), check_trace=False)
        assert "LookupPairFunction" in str(traced.graph)
        out1, out2 = traced(coords)
    assert torch.equal(out1, torch.zeros_like(out1)) and torch.equal(out2, torch.ones_like(out2))


@pytest.mark.gpu
def test_a_trace_looks_up(cuda_device):
    g = torch.Generator().manual_seed(1)
    v1, v2 = torch.randn(1, 1, 24, 16, 24, generator=g).to(cuda_device), torch.randn(1, 1, 16, 16, 24, generator=g).to(cuda_device)
    first, then = (torch.rand(1, 2, 16, 24, generator=g).to(cuda_device) * 10 for _ in range(2))
    lookup = sfb.CorrBlock1D(v1, v2, num_levels=2, radius=2)
    with torch.no_grad():
        traced = torch.jit.trace(lambda c: lookup(c), (first,), check_trace=False)
        for got, want in zip(traced(then), lookup(then)):
            assert torch.equal(got, want)


def test_cpu_tensors_are_refused():
    v1, v2, coords = torch.zeros(1, 1, 16, 16, 16), torch.zeros(1, 1, 16, 16, 16), torch.zeros(1, 2, 16, 16)
    with pytest.raises(RuntimeError, match="CUDA"):
        ops.lookup_build_pyramid_pair(v1, v2, 2)
    with pytest.raises(RuntimeError, match="CUDA"):
        ops.lookup_forward_pair(v1, v2, v1, v2, coords, 2, 2)
    with pytest.raises(RuntimeError, match="CUDA"):
        ops.lookup_accumulate_pair(v1.shape, v2.shape, coords, None, None, None, None, 2, 2)
    with pytest.raises(RuntimeError, match="Tensor"):
        ops.lookup_forward_pair(v1, v2, v1, v2, [1.0], 2, 2)


@pytest.mark.gpu
def test_malformed_arguments_are_refused(cuda_device):
    H, W, levels, radius = 16, 24, 2, 2
    v1, v2 = torch.zeros(2, 1, W, H, W, device=cuda_device), torch.zeros(2, 1, H, H, W, device=cuda_device)
    coords = torch.zeros(2, 2, H, W, device=cuda_device)
    p1, p2 = ops.lookup_build_pyramid_pair(v1, v2, levels)
    out1, out2 = ops.lookup_forward_pair(v1, v2, p1, p2, coords, levels, radius)
    assert out1.shape == (2, levels * 5, H, W) and out1.device == cuda_device and out1.dtype == torch.float32
    for args, match in (((v1.double(), v2, p1, p2, coords), "dtype"), ((v1[:, :, :, :, ::2], v2, p1, p2, coords), "contiguous"),
                        ((v1[0], v2, p1, p2, coords), "dimensions"), ((v1, v2[:1], p1, p2, coords), "differ"),
                        ((v1, v2, p1, p2, coords.double()), "coords"), ((v1, v2, p1, p2, coords[:1]), "coords"),
                        ((v1, v2, p1, p2, coords.transpose(2, 3).contiguous().transpose(2, 3)), "contiguous")):
        with pytest.raises(RuntimeError, match=match):
            ops.lookup_forward_pair(*args, levels, radius)
    with pytest.raises(RuntimeError, match="unsupported"):
        ops.lookup_build_pyramid_pair(v1, v2, 6)
    acc = torch.zeros(ops.lookup_accumulator_size(v1.shape, levels, True), device=cuda_device)
    for gout, sums, match in ((out1[:1], acc, "shape"), (out1, acc[1:], "shape"), (out1.double(), acc, "dtype")):
        with pytest.raises(RuntimeError, match=match):
            ops.lookup_accumulate_pair(v1.shape, v2.shape, coords, gout, None, sums, None, levels, radius)
    # a slice of a larger tensor of coordinates is taken as it lies
    wide = torch.rand(2, 5, H, W, device=cuda_device) * 8
    a = ops.lookup_forward_pair(v1 + 1, v2, p1, p2, wide[:, 1:3], levels, radius)
    b = ops.lookup_forward_pair(v1 + 1, v2, p1, p2, wide[:, 1:3].contiguous(), levels, radius)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
