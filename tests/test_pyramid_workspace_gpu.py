"""The workspace of a pyramid's backward: regions used twice, and the gradient of the volume stored for all samples, for some at a time
(batches that the chunk does not divide among them) or not at all, whatever room the buffer has."""
import ctypes
import math

import pytest
import torch
import torch.nn.functional as F

from separableflowthesis_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def level_sizes(H, W, levels):
    return [(ctypes.c_int32 * levels)(*[n >> l for l in range(levels)]) for n in (H, W)]


# (B, C, H, W, Kc, levels): 5 and 19 samples in chunks of any size, levels with an odd side; one sample beyond 4096 pixels
@pytest.mark.parametrize("operands", ["fp16", "bf16", "tf32"])
@pytest.mark.parametrize("shape", [(5, 64, 24, 40, 2, 4), (19, 32, 16, 33, 1, 2), (3, 32, 66, 64, 1, 2), (3, 32, 66, 64, 3, 4)])
def test_room_for_the_gradient_of_the_volume(shape, operands, cuda_device, monkeypatch):
    B, C, H, W, Kc, levels = shape
    g = torch.Generator().manual_seed(B)
    randn = lambda *s: torch.randn(*s, generator=g).to(cuda_device)
    f1, pyr, Kt, scale1 = randn(B, C, H, W), [randn(B, C, H, W)], 2 + Kc, 1 / math.sqrt(C)
    for _ in range(levels - 1):
        pyr.append(F.avg_pool2d(pyr[-1], 2, stride=2).contiguous())
    params = [randn(Kc, 2, 3, 3, 3) * 0.2, randn(Kc) * 0.1, randn(Kc, 2, 3, 3, 3) * 0.2, randn(Kc) * 0.1]
    gu, gv = randn(B, Kt * levels, W, H, W), randn(B, Kt * levels, H, H, W)
    lib = _lib.load()
    dims = _lib.SfbShape(B, H, W, H, W, C, Kc)
    sizes = level_sizes(H, W, levels)
    size = lambda backward: lib.sfb_separation_pyramid_workspace_bytes(ctypes.byref(dims), *sizes, levels, backward)
    sample = sum(-(-(H >> l) // 4) * -(-(W >> l) // 16) * (-(-(H * W) // 128) * 128) * 128 for l in range(levels))   # bytes of a sample's G
    with ops.sweep_operands(operands):
        full, least = size(1), size(2)
        assert (full == least) == (operands == "tf32")
        sep_u, sep_v, buffer = ops.separation_pyramid_forward(f1, pyr, *params, True, scale1)

        def backward(nbytes):
            """Gradients with a buffer of exactly that size, filled with NaN, and the launches of the gradient GEMMs and their folds."""
            monkeypatch.setattr(ops, "_workspace", lambda n, dev, stream: torch.full((nbytes // 4,), math.nan, device=dev).view(torch.uint8))
            _lib.kernel_timing(True)
            out = ops.separation_pyramid_backward(f1, pyr, params[0], params[2], sep_u, sep_v, buffer, gu, gv, scale1)
            report = {name: n for name, _, n in _lib.kernel_timing_report()}
            _lib.kernel_timing(False)
            return [out[0], *out[1], *out[2:]], report["grad_gemm_kernel<fused,image1-major>"]

        want, launches = backward(full)
        assert launches <= 2
        relerr = lambda x, ref: ((x.double() - ref.double()).norm() / ref.double().norm().clamp_min(1e-30)).item()
        seen = {launches}
        for nbytes in sorted({least} | {n // 256 * 256 for n in range(least, full, sample)}):
            got, launches = backward(nbytes)
            seen.add(launches)
            for i, (x, ref) in enumerate(zip(got, want)):
                if i in (levels + 2, levels + 4):   # a softmax does not see its bias: those gradients are rounding
                    assert torch.isfinite(x).all()
                    continue
                # sums of up to H*W products in other pieces (tests/test_pyramid_levels_gpu.py)
                assert relerr(x, ref) < H * W / 8 * 2 ** -23 + 2e-5, (nbytes, i)
        assert operands == "tf32" or len(seen) > 1   # some buffers took chunks
        with pytest.raises(RuntimeError, match="needed"):
            backward(least - 256)
