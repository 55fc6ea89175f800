"""CPU: the autograd side of the lookups on both aggregated volumes (LookupPairFunction, LookupVolumeFunction) with the oracle in place
of the library; the library's own ops are tested in the gpu-marked files."""
import pytest
import torch

from oracle import separation_oracle as orc
from separableflowthesis_b200 import functions


class PairOps:
    """The pair ops on CPU tensors.  An accumulator holds the gradient of its volume."""

    @staticmethod
    def lookup_build_pyramid_pair(corr1, corr2, levels):
        return None, None

    @staticmethod
    def lookup_forward_pair(corr1, corr2, pyramid1, pyramid2, coords, levels, radius):
        return (orc.lookup_forward(corr1, coords[:, 0], levels, radius, True), orc.lookup_forward(corr2, coords[:, 1], levels, radius, False))

    @staticmethod
    def lookup_accumulator_size(shape, levels, clamp_unit):
        return torch.Size(shape).numel()

    @staticmethod
    def lookup_accumulate_pair(shape1, shape2, coords, g1, g2, acc1, acc2, levels, radius):
        for g, acc, shape, axis in ((g1, acc1, shape1, 0), (g2, acc2, shape2, 1)):
            if g is not None:
                acc += orc.lookup_backward(shape, coords[:, axis], g, levels, radius, axis == 0).reshape(-1)

    @staticmethod
    def lookup_fold_gradient(acc, shape, levels, clamp_unit):
        return acc.reshape(shape)


@pytest.fixture()
def pair_ops(monkeypatch):
    monkeypatch.setattr(functions, "MemorySaver", PairOps)


LEVELS, RADIUS = 2, 2


def inputs(needs1, needs2, coords_need, seed=3):
    g = torch.Generator().manual_seed(seed)
    v1 = torch.randn(2, 1, 7, 6, 7, generator=g, dtype=torch.float64).requires_grad_(needs1)
    v2 = torch.randn(2, 1, 6, 6, 7, generator=g, dtype=torch.float64).requires_grad_(needs2)
    coords = (8 * torch.rand(2, 2, 6, 7, generator=g, dtype=torch.float64) - 1).requires_grad_(coords_need)
    return v1, v2, coords


@pytest.mark.parametrize("needs1,needs2", [(False, False), (True, False), (False, True), (True, True)])
def test_coordinates_that_need_a_gradient(needs1, needs2, pair_ops):
    """They get none, and neither do volumes that need none; a loss of either output alone can still be differentiated, as with one
    lookup per volume (LookupFunction)."""
    for part in ((0,), (1,), (0, 1)):
        v1, v2, coords = inputs(needs1, needs2, True)
        edges = [functions.LookupVolumeFunction.apply(v, LEVELS, clamp) if v.requires_grad else None for v, clamp in ((v1, True), (v2, False))]
        outs = functions.LookupPairFunction.apply(v1, v2, None, None, coords, *edges, LEVELS, RADIUS)[:2]
        assert outs[0].requires_grad and outs[1].requires_grad
        sum((outs[i] * outs[i]).sum() for i in part).backward()
        assert coords.grad is None
        for i, (v, needs) in enumerate(((v1, needs1), (v2, needs2))):
            if not needs or i not in part:
                assert v.grad is None
                continue
            want = orc.lookup_backward(v.shape, coords.detach()[:, i], 2 * outs[i].detach(), LEVELS, RADIUS, i == 0)
            assert torch.equal(v.grad, want)


def test_outputs_of_volumes_without_gradients(pair_ops):
    v1, v2, coords = inputs(False, False, False)
    out1, out2, *_ = functions.LookupPairFunction.apply(v1, v2, None, None, coords, None, None, LEVELS, RADIUS)
    assert not out1.requires_grad and not out2.requires_grad
