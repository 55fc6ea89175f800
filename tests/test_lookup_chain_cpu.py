"""CPU: the host side of the lookups on both aggregated volumes (CorrBlock1D, LookupPairFunction, LookupVolumeFunction) with the oracle in
place of the library; the library's own ops are tested in the gpu-marked files."""
import os

import numpy as np
import pytest
import torch

import separableflowthesis_b200 as sfb
from oracle import separation_oracle as orc
from separableflowthesis_b200 import corr, functions


class PairOps:
    """The pair ops on CPU tensors.  An accumulator holds the gradient of its volume."""

    log = []   # accumulations and folds

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
        PairOps.log.append(("accumulate", g1 is not None, g2 is not None))
        for g, acc, shape, axis in ((g1, acc1, shape1, 0), (g2, acc2, shape2, 1)):
            if g is not None:
                acc += orc.lookup_backward(shape, coords[:, axis], g, levels, radius, axis == 0).reshape(-1)

    @staticmethod
    def lookup_fold_gradient(acc, shape, levels, clamp_unit):
        PairOps.log.append(("fold", clamp_unit))
        return acc.reshape(shape)


@pytest.fixture()
def pair_ops(monkeypatch):
    monkeypatch.setattr(functions, "MemorySaver", PairOps)
    monkeypatch.setattr(corr, "_ops", PairOps)
    del PairOps.log[:]


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
    lookup per volume."""
    for part in ((0,), (1,), (0, 1)):
        v1, v2, coords = inputs(needs1, needs2, True)
        edges = [functions.LookupVolumeFunction.apply(v, LEVELS, clamp, []) if v.requires_grad else None for v, clamp in ((v1, True), (v2, False))]
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


def sequence(block, coords):
    return [block(c) for c in coords]


def test_chain_against_the_reference(golden_dir, pair_ops):
    """Several lookups of one block, one backward: the outputs and, for the golden upstream gradients of one lookup, the gradients of the
    reference's own class; accumulated per lookup, folded once per volume."""
    g = np.load(os.path.join(golden_dir, "lookup1d_b1_dim2_16x24.npz"))
    load = lambda name: torch.from_numpy(np.ascontiguousarray(g[name])).double()
    v1, v2, coords = load("corr1").requires_grad_(True), load("corr2").requires_grad_(True), load("coords")
    block = sfb.CorrBlock1D(v1, v2, num_levels=int(g["levels"]), radius=int(g["radius"]))
    weights = (1.0, -0.5, 3.0)
    outs = sequence(block, [coords] * 3)
    for out1, out2 in outs:
        assert (out1 - load("out1")).abs().max() < 1e-6 and (out2 - load("out2")).abs().max() < 1e-6
    sum(w * ((o1 * load("w1")).sum() + (o2 * load("w2")).sum()) for w, (o1, o2) in zip(weights, outs)).backward()
    assert (v1.grad - sum(weights) * load("g_corr1")).abs().max() < 5e-6
    assert (v2.grad - sum(weights) * load("g_corr2")).abs().max() < 5e-6
    assert PairOps.log == [("accumulate", True, True)] * 3 + PairOps.log[3:] and sorted(PairOps.log[3:]) == [("fold", False), ("fold", True)]


def test_chain_of_different_lookups(pair_ops):
    """Lookups that reach the loss with one output, with none, and lookups without grad in between."""
    v1, v2, _ = inputs(True, True, False)
    coords = [inputs(False, False, False, seed)[2] for seed in range(4)]
    block = sfb.CorrBlock1D(v1, v2, num_levels=LEVELS, radius=RADIUS)
    outs = sequence(block, coords[:2])
    with torch.no_grad():
        assert not block(coords[0])[0].requires_grad
    outs += sequence(block, coords[2:])
    (outs[0][0].sum() + (outs[2][1] ** 2).sum() + outs[3][0].sum()).backward()
    lookup = lambda v, i, g, axis: orc.lookup_backward(v.shape, coords[i][:, axis], g, LEVELS, RADIUS, axis == 0)
    ones = torch.ones_like(outs[0][0])
    assert torch.allclose(v1.grad, lookup(v1, 0, ones, 0) + lookup(v1, 3, ones, 0), atol=1e-12)
    assert torch.allclose(v2.grad, lookup(v2, 2, 2 * outs[2][1].detach(), 1), atol=1e-12)


@pytest.mark.parametrize("retain", [False, True])
def test_backward_after_every_lookup(retain, pair_ops, monkeypatch):
    """Each goes through its own lookup alone."""
    walked = []
    backward = functions.LookupPairFunction.backward

    def counted(ctx, *grads):
        walked.append(1)
        return backward(ctx, *grads)

    monkeypatch.setattr(functions.LookupPairFunction, "backward", staticmethod(counted))
    v1, v2, _ = inputs(True, True, False)
    block = sfb.CorrBlock1D(v1, v2, num_levels=LEVELS, radius=RADIUS)
    for i in range(4):
        coords = inputs(False, False, False, i)[2]
        o1, o2 = block(coords)
        g1, g2 = torch.autograd.grad([(o1 * o1).sum() + o2.sum()], [v1, v2], retain_graph=retain)
        assert torch.equal(g1, orc.lookup_backward(v1.shape, coords[:, 0], 2 * o1.detach(), LEVELS, RADIUS, True))
        assert torch.equal(g2, orc.lookup_backward(v2.shape, coords[:, 1], torch.ones_like(o2), LEVELS, RADIUS, False))
    assert len(walked) == 4
    outs = sequence(block, [coords] * 3)   # and a chain goes on where there was none
    sum(o1.sum() + o2.sum() for o1, o2 in outs).backward()
    assert len(walked) == 7


def test_volumes_and_coordinates_are_the_ops_business(monkeypatch):
    """No path around the library: what the pair ops refuse is refused."""
    v1, v2, coords = inputs(False, False, False)
    with pytest.raises(RuntimeError, match="CUDA"):
        sfb.CorrBlock1D(v1, v2)
