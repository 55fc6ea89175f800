"""The three autograd Functions of libs/MemorySaver/functions/MemorySaver.py, same names, argument
order, outputs and error behaviour, on top of the B200 ops, which make the tensors' device current themselves."""
from __future__ import annotations

import torch
from torch.autograd import Function
from torch.autograd.function import once_differentiable

from . import ops as MemorySaver


class ComputeMaxAvgFunction(Function):
    """Max and mean channels without argmax; inference only (functions/MemorySaver.py:6-38)."""

    @staticmethod
    def forward(ctx, img1_features_l0, img2_features_lk):
        assert img1_features_l0.is_contiguous() and img2_features_lk.is_contiguous()
        max_avg_output_u, max_avg_output_v = MemorySaver.max_avg_forward(img1_features_l0, img2_features_lk)
        return max_avg_output_u, max_avg_output_v

    @staticmethod
    def backward(ctx, gradOutput_u, gradOutput_v):
        raise NotImplementedError("max avg backward pass is not implemented: use max argmax avg")


class ComputeMaxArgmaxAvgFunction(Function):
    """Max (+argmax kept for backward) and mean channels (functions/MemorySaver.py:40-105)."""

    @staticmethod
    def forward(ctx, img1_features_l0, img2_features_lk):
        assert img1_features_l0.is_contiguous() and img2_features_lk.is_contiguous()
        ma_u, ma_v, am_u, am_v = MemorySaver.max_argmax_avg_forward(img1_features_l0, img2_features_lk)
        ctx.save_for_backward(img1_features_l0, img2_features_lk, am_u, am_v)
        return ma_u, ma_v

    @staticmethod
    def backward(ctx, grad_MaxAvg_u, grad_MaxAvg_v):
        img1_features_l0, img2_features_lk, am_u, am_v = ctx.saved_tensors
        grad_MaxAvg_u = grad_MaxAvg_u.contiguous()
        grad_MaxAvg_v = grad_MaxAvg_v.contiguous()
        g1, g2 = MemorySaver.max_argmax_avg_backward(img1_features_l0, img2_features_lk, am_u, am_v,
                                                     grad_MaxAvg_u, grad_MaxAvg_v)
        return g1, g2


class ComputeSelfCompressionFunction(Function):
    """Attention-weighted compression channels (functions/MemorySaver.py:107-177)."""

    @staticmethod
    def forward(ctx, img1_features_l0, img2_features_lk, attention_weights_u, attention_weights_v):
        assert img1_features_l0.is_contiguous() and img2_features_lk.is_contiguous()
        assert attention_weights_u.is_contiguous() and attention_weights_v.is_contiguous()
        c_u, c_v = MemorySaver.compression_forward(img1_features_l0, img2_features_lk,
                                                   attention_weights_u, attention_weights_v)
        ctx.save_for_backward(img1_features_l0, img2_features_lk, attention_weights_u, attention_weights_v)
        return c_u, c_v

    @staticmethod
    def backward(ctx, grad_compressed_output_u, grad_compressed_output_v):
        f1, f2, a_u, a_v = ctx.saved_tensors
        grad_compressed_output_u = grad_compressed_output_u.contiguous()
        grad_compressed_output_v = grad_compressed_output_v.contiguous()
        g1, g2, ga_u, ga_v = MemorySaver.compression_backward(f1, f2, a_u, a_v, grad_compressed_output_u,
                                                              grad_compressed_output_v)
        return g1, g2, ga_u, ga_v


# --------------------------------------------------------------------------------------------------
# Fused backward for the call site.  Not part of the reference's surface.
#
# When the max/avg node and the compression node act on the same (F1, F2) -- which is how
# AlternateCorrBlockSepflow.separate uses them (core/corr.py:425,448) -- their two feature gradients are
# summed by autograd.  The pair of Functions below produces that sum with ONE pair of gradient GEMMs:
# the compression node's backward returns only the attention gradients (they are needed at once, the
# Conv3d/softmax backward sits between the two nodes) and parks its inputs in a shared state object; the
# max/avg node's backward, which autograd always runs later because its outputs feed the attention
# weights, then computes the summed feature gradients.
class SeparationState:
    """Shared between the two fused Functions of one pyramid level."""

    def __init__(self):
        self.pending = None          # (A_u, A_v, gC_u, gC_v) parked by the compression node's backward
        self.collected = True


def _guard_pending(state):
    # runs when the backward pass that parked the tensors ends: they must have been consumed by then
    def check():
        if state.pending is not None:
            state.pending = None
            raise RuntimeError(
                "fused separation backward: the compression node deferred its feature gradients but the "
                "max/avg node's backward never ran (its outputs do not reach the loss); use "
                "AlternateCorrBlockSepflow(..., fuse_backward=False)")
    return check


class FusedMaxArgmaxAvgFunction(Function):
    @staticmethod
    def forward(ctx, img1_features_l0, img2_features_lk, state):
        assert img1_features_l0.is_contiguous() and img2_features_lk.is_contiguous()
        ma_u, ma_v, am_u, am_v = MemorySaver.max_argmax_avg_forward(img1_features_l0, img2_features_lk)
        ctx.save_for_backward(img1_features_l0, img2_features_lk, am_u, am_v)
        ctx.state = state
        return ma_u, ma_v

    @staticmethod
    def backward(ctx, grad_MaxAvg_u, grad_MaxAvg_v):
        f1, f2, am_u, am_v = ctx.saved_tensors
        grad_MaxAvg_u = grad_MaxAvg_u.contiguous()
        grad_MaxAvg_v = grad_MaxAvg_v.contiguous()
        pending, ctx.state.pending = ctx.state.pending, None
        if pending is None:
            g1, g2 = MemorySaver.max_argmax_avg_backward(f1, f2, am_u, am_v, grad_MaxAvg_u, grad_MaxAvg_v)
        else:
            a_u, a_v, gc_u, gc_v = pending
            g1, g2 = MemorySaver.separation_feature_backward(f1, f2, am_u, am_v, grad_MaxAvg_u, grad_MaxAvg_v,
                                                             a_u, a_v, gc_u, gc_v)
        return g1, g2, None


class FusedSelfCompressionFunction(Function):
    @staticmethod
    def forward(ctx, img1_features_l0, img2_features_lk, attention_weights_u, attention_weights_v, state):
        assert img1_features_l0.is_contiguous() and img2_features_lk.is_contiguous()
        assert attention_weights_u.is_contiguous() and attention_weights_v.is_contiguous()
        c_u, c_v = MemorySaver.compression_forward(img1_features_l0, img2_features_lk,
                                                   attention_weights_u, attention_weights_v)
        ctx.save_for_backward(img1_features_l0, img2_features_lk, attention_weights_u, attention_weights_v)
        ctx.state = state
        return c_u, c_v

    @staticmethod
    def backward(ctx, grad_compressed_output_u, grad_compressed_output_v):
        f1, f2, a_u, a_v = ctx.saved_tensors
        gc_u = grad_compressed_output_u.contiguous()
        gc_v = grad_compressed_output_v.contiguous()
        if not (ctx.needs_input_grad[0] or ctx.needs_input_grad[1]):
            ga_u, ga_v = MemorySaver.compression_attention_backward(f1, f2, gc_u, gc_v)
            return None, None, ga_u, ga_v, None
        if not (ctx.needs_input_grad[2] or ctx.needs_input_grad[3]):
            # the attention weights do not depend on the max/avg node: nothing guarantees that node's
            # backward runs after this one, so do not defer
            g1, g2, ga_u, ga_v = MemorySaver.compression_backward(f1, f2, a_u, a_v, gc_u, gc_v)
            return g1, g2, ga_u, ga_v, None
        ga_u, ga_v = MemorySaver.compression_attention_backward(f1, f2, gc_u, gc_v)
        ctx.state.pending = (a_u, a_v, gc_u, gc_v)
        torch.autograd.Variable._execution_engine.queue_callback(_guard_pending(ctx.state))
        return None, None, ga_u, ga_v, None


# --------------------------------------------------------------------------------------------------
# Channels-first pair for the call site: same fused backward, and every per-pixel tensor already has the
# (B, K, D, H1, W1) layout of the Conv3d attention modules, so the call site's permute copies disappear.
class SeparationMaxAvgCF(Function):
    @staticmethod
    def forward(ctx, img1_features_l0, img2_features_lk, state, with_argmax):
        assert img1_features_l0.is_contiguous() and img2_features_lk.is_contiguous()
        sep_v, sep_u, am_u, am_v = MemorySaver.max_argmax_avg_forward_cf(img1_features_l0, img2_features_lk,
                                                                         with_argmax)
        if with_argmax:
            ctx.save_for_backward(img1_features_l0, img2_features_lk, am_u, am_v)
        ctx.state = state
        ctx.with_argmax = with_argmax
        return sep_v, sep_u

    @staticmethod
    def backward(ctx, grad_sep_v, grad_sep_u):
        if not ctx.with_argmax:
            raise NotImplementedError("max avg backward pass is not implemented: use max argmax avg")
        f1, f2, am_u, am_v = ctx.saved_tensors
        pending, ctx.state.pending = ctx.state.pending, None
        if pending is None:
            raise RuntimeError("channels-first separation backward needs the compression node's backward first "
                               "(use AlternateCorrBlockSepflow(..., channels_first=False) for max/avg alone)")
        a_u, a_v, gc_u, gc_v = pending
        g1, g2 = MemorySaver.separation_feature_backward_cf(f1, f2, am_u, am_v, grad_sep_v.contiguous(),
                                                            grad_sep_u.contiguous(), a_u, a_v, gc_u, gc_v)
        return g1, g2, None, None


class SeparationCompressionCF(Function):
    @staticmethod
    def forward(ctx, img1_features_l0, img2_features_lk, a_u, a_v, state):
        assert img1_features_l0.is_contiguous() and img2_features_lk.is_contiguous()
        assert a_u.is_contiguous() and a_v.is_contiguous()
        c_u, c_v = MemorySaver.compression_forward_cf(img1_features_l0, img2_features_lk, a_u, a_v)
        ctx.save_for_backward(img1_features_l0, img2_features_lk, a_u, a_v)
        ctx.state = state
        return c_u, c_v

    @staticmethod
    def backward(ctx, grad_c_u, grad_c_v):
        f1, f2, a_u, a_v = ctx.saved_tensors
        gc_u, gc_v = grad_c_u.contiguous(), grad_c_v.contiguous()
        ga_u, ga_v = MemorySaver.compression_attention_backward_cf(f1, f2, gc_u, gc_v)
        if ctx.needs_input_grad[0] or ctx.needs_input_grad[1]:
            ctx.state.pending = (a_u, a_v, gc_u, gc_v)
            torch.autograd.Variable._execution_engine.queue_callback(_guard_pending(ctx.state))
        return None, None, ga_u, ga_v, None


# --------------------------------------------------------------------------------------------------
# One pyramid level as a single autograd node: max/avg sweep, both attention modules (Conv3d(2, Kc, 3,
# padding=1) + softmax over the displacement axis, core/corr.py:437-442) and the compression sweep, writing
# the concatenated tensors of core/corr.py:454-457 directly.  The backward is one call as well.
class SeparationLevelFunction(Function):
    @staticmethod
    def forward(ctx, img1_features_l0, img2_features_lk, weight_u, bias_u, weight_v, bias_v, with_argmax,
                fmaps=False, scale1=1.0):
        """With ``fmaps`` the features are the model's maps (B,C,H,W) and ``scale1`` multiplies image 1's."""
        assert img1_features_l0.is_contiguous() and img2_features_lk.is_contiguous()
        ctx.fmaps, ctx.scale1 = fmaps, scale1
        sep_u, sep_v, am_u, am_v, a_u, a_v = MemorySaver.separation_level_forward(
            img1_features_l0, img2_features_lk, weight_u.contiguous(), bias_u.contiguous(),
            weight_v.contiguous(), bias_v.contiguous(), with_argmax, fmaps, scale1)
        if with_argmax:
            ctx.save_for_backward(img1_features_l0, img2_features_lk, weight_u, weight_v, sep_u, sep_v, am_u, am_v,
                                  a_u, a_v)
        ctx.with_argmax = with_argmax
        return sep_u, sep_v

    @staticmethod
    @once_differentiable
    def backward(ctx, grad_sep_u, grad_sep_v):
        if not ctx.with_argmax:
            raise NotImplementedError("max avg backward pass is not implemented: use max argmax avg")
        f1, f2, weight_u, weight_v, sep_u, sep_v, am_u, am_v, a_u, a_v = ctx.saved_tensors
        g1, g2, gw_u, gb_u, gw_v, gb_v = MemorySaver.separation_level_backward(
            f1, f2, weight_u.contiguous(), weight_v.contiguous(), sep_u, sep_v, am_u, am_v, a_u, a_v,
            grad_sep_u.contiguous(), grad_sep_v.contiguous(), ctx.fmaps, ctx.scale1)
        return g1, g2, gw_u, gb_u, gw_v, gb_v, None, None, None


# --------------------------------------------------------------------------------------------------
# All pyramid levels as one autograd node (core/corr.py:416-475): the maps of up to four levels go to the library in one call, which
# runs every kernel once for all of them.  Else, or where there is no memory for what that takes at a time, the one-call forward of a
# level from the feature maps per level, whose volumes are resampled along the displacement axis and written straight into their channel slice
# of the concatenated outputs (the reference runs F.interpolate per level and torch.cat over levels).
def _levels_together(fmap1, fmap2_levels, Kc):
    H2, W2 = fmap2_levels[0].shape[2:]
    return (fmap1.is_cuda and len(fmap2_levels) <= MemorySaver.PYRAMID_MAX_LEVELS and Kc <= MemorySaver.PYRAMID_MAX_CHANNELS
            and all(f.shape[2] <= H2 and f.shape[3] <= W2 for f in fmap2_levels) and fmap1.shape[0] * (2 + Kc) <= 65535)


def _levels_forward(fmap1, fmap2_levels, params, with_argmax, scale1):
    """Level by level: sep_u, sep_v and, for a backward, (sep_u, sep_v, argmax_u, argmax_v, a_u, a_v) per level; volumes that lie in the
    outputs are None."""
    B, _, H1, W1 = fmap1.shape
    H2, W2 = fmap2_levels[0].shape[2:]     # displacement ranges of the outputs (= H1, W1 unless image-1 rows are sharded)
    L, Kt = len(fmap2_levels), 2 + params[0].shape[0]
    sep_u = torch.empty(B, Kt * L, W2, H1, W1, dtype=fmap1.dtype, device=fmap1.device)
    sep_v = torch.empty(B, Kt * L, H2, H1, W1, dtype=fmap1.dtype, device=fmap1.device)
    saved = []
    for l, fmap2 in enumerate(fmap2_levels):
        if tuple(fmap2.shape[2:]) == (H2, W2):   # displacement range of the output: written in place
            level = MemorySaver.separation_level_forward(fmap1, fmap2, *params, with_argmax, True, scale1, (sep_u, sep_v, l * Kt))
        else:
            level = MemorySaver.separation_level_forward(fmap1, fmap2, *params, with_argmax, True, scale1)
            MemorySaver.upsample_displacement_into(level[0], sep_u, l * Kt)
            MemorySaver.upsample_displacement_into(level[1], sep_v, l * Kt)
        if with_argmax:
            saved.append(tuple(level))
    return sep_u, sep_v, saved


def _levels_backward(fmap1, fmap2_levels, weight_u, weight_v, sep_u, sep_v, saved, gu, gv, scale1):
    """Gradients of fmap1, [fmap2_l], weight_u, bias_u, weight_v, bias_v from what _levels_forward saved."""
    Kt = 2 + weight_u.shape[0]
    total, g2 = None, []
    for l, (fmap2, (su, sv, am_u, am_v, a_u, a_v)) in enumerate(zip(fmap2_levels, saved)):
        if su is None:
            out = MemorySaver.separation_level_backward(fmap1, fmap2, weight_u, weight_v, sep_u, sep_v, am_u, am_v, a_u, a_v, gu, gv, True,
                                                        scale1, l * Kt)
        else:
            gsu = MemorySaver.upsample_displacement_backward(gu, l * Kt, Kt, su.shape[2])
            gsv = MemorySaver.upsample_displacement_backward(gv, l * Kt, Kt, sv.shape[2])
            out = MemorySaver.separation_level_backward(fmap1, fmap2, weight_u, weight_v, su, sv, am_u, am_v, a_u, a_v, gsu, gsv, True, scale1)
        g2.append(out.pop(1))
        if total is None:
            total = out
        else:
            for t, x in zip(total, out):
                t += x
    g1, *gparams = total
    return (g1, g2, *gparams)


def _pyramid_forward(ctx, with_argmax, scale1, weight_u, bias_u, weight_v, bias_v, fmap1, fmap2_levels, levels=None, pooled=None):
    """`pooled`: fmap2_levels is the first of so many levels, and the others are in that buffer (pool_levels)."""
    params = [t.contiguous() for t in (weight_u, bias_u, weight_v, bias_v)]
    ctx.with_argmax, ctx.scale1, ctx.levels = with_argmax, scale1, levels or len(fmap2_levels)
    ctx.together = _levels_together(fmap1, fmap2_levels, weight_u.shape[0])
    if ctx.together:
        try:
            sep_u, sep_v, saved = MemorySaver.separation_pyramid_forward(fmap1, fmap2_levels, *params, with_argmax, scale1, levels, pooled)
        except torch.OutOfMemoryError:
            ctx.together = False   # (not here, where the exception keeps the attempt's tensors)
    if not ctx.together:
        sep_u, sep_v, saved = _levels_forward(fmap1, _all_levels(fmap2_levels, ctx.levels, pooled), params, with_argmax, scale1)
    if with_argmax:
        if not ctx.together:   # volumes written in place are saved as the outputs themselves
            ctx.in_place = [t[0] is None for t in saved]
        flat = [saved] if ctx.together else [x for t in saved for x in t if x is not None]
        ctx.save_for_backward(fmap1, weight_u, weight_v, sep_u, sep_v, *fmap2_levels, *([] if pooled is None else [pooled]), *flat)
    return sep_u, sep_v


def _all_levels(fmap2_levels, levels, pooled):
    return fmap2_levels if pooled is None else [*fmap2_levels, *MemorySaver.pooled_level_views(pooled, fmap2_levels[0].shape, levels)]


def _pyramid_backward(ctx, grad_sep_u, grad_sep_v, is_pooled=False):
    """(g1, [g2_l], parameters'); `is_pooled`: the one gradient of the first level, with what its averages contribute."""
    if not ctx.with_argmax:
        raise NotImplementedError("max avg backward pass is not implemented: use max argmax avg")
    L = ctx.levels
    fmap1, weight_u, weight_v, sep_u, sep_v, *rest = ctx.saved_tensors
    given = 1 if is_pooled else L
    fmap2_levels, pooled, saved = rest[:given], rest[given] if is_pooled else None, rest[given + is_pooled:]
    wu, wv = weight_u.contiguous(), weight_v.contiguous()
    gu, gv = grad_sep_u.contiguous(), grad_sep_v.contiguous()
    if ctx.together:
        try:
            return MemorySaver.separation_pyramid_backward(fmap1, fmap2_levels, wu, wv, sep_u, sep_v, saved[0], gu, gv, ctx.scale1, L, pooled)
        except torch.OutOfMemoryError:
            pass
    fmap2_levels = _all_levels(fmap2_levels, L, pooled)
    if ctx.together:
        saved = MemorySaver.separation_pyramid_saved(saved[0], fmap1, fmap2_levels, weight_u.shape[0], True)
    else:
        flat = iter(saved)
        saved = [tuple(None if in_place and i < 2 else next(flat) for i in range(6)) for in_place in ctx.in_place]
    g1, g2, *gparams = _levels_backward(fmap1, fmap2_levels, wu, wv, sep_u, sep_v, saved, gu, gv, ctx.scale1)
    if is_pooled:
        for l in range(L - 1, 0, -1):
            g2[l - 1] += torch.ops.aten.avg_pool2d_backward(g2[l], fmap2_levels[l - 1], [2, 2], [2, 2], [0, 0], False, True, None)
        del g2[1:]
    return (g1, g2, *gparams)


class SeparationPyramidFunction(Function):
    @staticmethod
    def forward(ctx, with_argmax, scale1, weight_u, bias_u, weight_v, bias_v, fmap1, *fmap2_levels):
        assert fmap1.is_contiguous() and all(f.is_contiguous() for f in fmap2_levels)
        return _pyramid_forward(ctx, with_argmax, scale1, weight_u, bias_u, weight_v, bias_v, fmap1, fmap2_levels)

    @staticmethod
    @once_differentiable
    def backward(ctx, grad_sep_u, grad_sep_v):
        g1, g2, *gparams = _pyramid_backward(ctx, grad_sep_u, grad_sep_v)
        return (None, None, *gparams, g1, *g2)


class SeparationPooledPyramidFunction(Function):
    """The same for the levels that ``pool_levels`` made of the first one, whose gradient has what they contribute: ``apply(with_argmax,
    scale1, levels, weight_u, bias_u, weight_v, bias_v, fmap1, fmap2, pooled)`` on CUDA maps, 2 to 4 levels with the first."""

    @staticmethod
    def forward(ctx, with_argmax, scale1, levels, weight_u, bias_u, weight_v, bias_v, fmap1, fmap2, pooled):
        return _pyramid_forward(ctx, with_argmax, scale1, weight_u, bias_u, weight_v, bias_v, fmap1, [fmap2], levels, pooled)

    @staticmethod
    @once_differentiable
    def backward(ctx, grad_sep_u, grad_sep_v):
        g1, (g2,), *gparams = _pyramid_backward(ctx, grad_sep_u, grad_sep_v, is_pooled=True)
        return (None, None, None, *gparams, g1, g2, None)


class PooledLevelFunction(Function):
    """A level that ``pool_levels`` made of the one before, as a differentiable tensor: ``apply(finer, (level,))`` returns level, with the
    gradient of avg_pool2d."""

    @staticmethod
    def forward(ctx, finer, level):
        ctx.save_for_backward(finer)
        return level[0]

    @staticmethod
    def backward(ctx, grad):
        (finer,) = ctx.saved_tensors
        return torch.ops.aten.avg_pool2d_backward(grad, finer, [2, 2], [2, 2], [0, 0], False, True, None), None


# --------------------------------------------------------------------------------------------------
# Lookups on the two aggregated 3D volumes (CorrBlock1D, core/corr.py:576-594).  The volumes' pyramids are passed in so that they are
# built once, not once per refinement iteration.  No gradient for the coordinates: the model detaches them (core/sepflow.py:192).
#
# A refinement looks up a dozen times on the same two volumes.  Gradients of the volumes themselves, one per lookup, would each be
# written whole and then added up by autograd.  Instead every lookup takes an edge to its volume (a tensor that stands for
# the volume's accumulator and holds nothing) and hands it on to the next: in the backward the accumulator comes down that
# chain, each lookup adds its windows to it, and the volume's node folds it into the gradient, once.
class LookupVolumeFunction(Function):
    """Start of a volume's chain: ``apply(corr, levels, clamp_unit, passed)`` -> edge.  A backward that has come down the chain appends to
    the list ``passed``: a lookup after it begins a chain of its own, and does not take later backwards through the earlier lookups."""

    @staticmethod
    def forward(ctx, corr, levels, clamp_unit, passed):
        ctx.cfg = (tuple(corr.shape), levels, clamp_unit)
        ctx.passed = passed
        ctx.set_materialize_grads(False)
        return torch.empty_strided((MemorySaver.lookup_accumulator_size(corr.shape, levels, clamp_unit),), (0,), dtype=corr.dtype,
                                   device=corr.device)

    @staticmethod
    @once_differentiable
    def backward(ctx, acc):
        if not ctx.passed:
            ctx.passed.append(True)
        if acc is None:
            return None, None, None, None
        shape, levels, clamp_unit = ctx.cfg
        return MemorySaver.lookup_fold_gradient(acc.contiguous(), shape, levels, clamp_unit), None, None, None


class LookupPairFunction(Function):
    """Lookup on both volumes: ``apply(corr1, corr2, pyramid1, pyramid2, coords, edge1, edge2, levels, radius)`` -> (out1, out2,
    edge1, edge2).  An edge is None where the volume needs no gradient."""

    @staticmethod
    def forward(ctx, corr1, corr2, pyramid1, pyramid2, coords, edge1, edge2, levels, radius):
        out1, out2 = MemorySaver.lookup_forward_pair(corr1, corr2, pyramid1, pyramid2, coords, levels, radius)
        ctx.cfg = (tuple(corr1.shape), tuple(corr2.shape), levels, radius)
        ctx.set_materialize_grads(False)
        if edge1 is not None or edge2 is not None:
            ctx.save_for_backward(coords)
            # (with coordinates that need a gradient, and get none, both outputs stay differentiable, whatever the volumes need)
            if not ctx.needs_input_grad[4]:
                ctx.mark_non_differentiable(*[out for out, edge in ((out1, edge1), (out2, edge2)) if edge is None])
        return out1, out2, edge1, edge2

    @staticmethod
    @once_differentiable
    def backward(ctx, g1, g2, acc1, acc2):
        # An accumulator belongs to this chain alone (its edges go from lookup to lookup), so it is added to in place.  A lookup
        # whose outputs are not part of the loss hands it on; its saved tensors may be gone by then.
        shape1, shape2, levels, radius = ctx.cfg
        if not ctx.needs_input_grad[5]:
            g1 = None
        if not ctx.needs_input_grad[6]:
            g2 = None
        if g1 is not None or g2 is not None:
            (coords,) = ctx.saved_tensors
            if g1 is not None:
                g1 = g1.contiguous()
                acc1 = _lookup_accumulator(acc1, shape1, levels, True, g1)
            if g2 is not None:
                g2 = g2.contiguous()
                acc2 = _lookup_accumulator(acc2, shape2, levels, False, g2)
            MemorySaver.lookup_accumulate_pair(shape1, shape2, coords, g1, g2, acc1, acc2, levels, radius)
        return None, None, None, None, None, acc1, acc2, None, None


def _lookup_accumulator(acc, shape, levels, clamp_unit, like):
    if acc is not None:
        return acc.contiguous()
    return like.new_zeros(MemorySaver.lookup_accumulator_size(shape, levels, clamp_unit))


class Lookup4dFunction(Function):
    """Lookup on the 4D correlation volume without storing it.  ``apply(coords, radius, scale, F1, *F2_levels)`` with
    channels-last features -> (B, levels*(2r+1)^2, H1, W1); gradients for the features only (the model detaches
    the coordinates, core/sepflow.py:193)."""

    @staticmethod
    def forward(ctx, coords, radius, scale, F1, *F2_levels):
        out = MemorySaver.lookup4d_forward(F1, list(F2_levels), coords, radius, scale)
        ctx.save_for_backward(coords, F1, *F2_levels)
        ctx.cfg = (radius, scale)
        return out

    @staticmethod
    @once_differentiable
    def backward(ctx, grad_out):
        coords, F1, *F2_levels = ctx.saved_tensors
        radius, scale = ctx.cfg
        gF1, gF2 = MemorySaver.lookup4d_backward(F1, F2_levels, coords, grad_out.contiguous(), radius, scale)
        return (None, None, None, gF1, *gF2)
