"""The gradient GEMMs at the edges of their K blocks (4 x 16 image-2 pixels, 32 image-1 pixels) and row tiles, whole and in
pieces.  Features, weights and gradients are small whole numbers, and the mean-gradients multiples of the row length that its FP32
reciprocal takes back to whole numbers, so dLoss/dS and every product and sum are exact whatever their order: results are compared
bit for bit."""
import pytest
import torch

from separableflowthesis_b200 import _lib, ops

pytestmark = pytest.mark.gpu

# (B, H1, W1, H2, W2, C, Kc) and whether the image-1-major and the image-2-major form are cut into pieces
SHAPES = [
    ((1, 2, 16, 1, 1, 8, 1), (False, False)),         # a single image-2 pixel, one block of image-1 pixels
    ((1, 3, 11, 3, 15, 8, 2), (False, False)),        # one pixel more than a block; rows and columns short of one
    ((1, 4, 32, 4, 16, 40, 3), (False, False)),       # whole tiles and blocks
    ((2, 3, 43, 5, 17, 24, 4), (False, False)),       # one row and column more
    ((1, 7, 40, 8, 64, 136, 6), (False, False)),      # two passes over channels, the second added to the first
    ((149, 1, 3, 9, 16, 16, 1), (False, False)),      # a tail of one tile behind a wave, too short to be cut
    ((149, 1, 3, 16, 64, 16, 1), (True, False)),      # and long enough
    ((1, 9, 31, 23, 33, 256, 2), (True, False)),      # several blocks both ways
    ((1, 43, 61, 5, 17, 24, 6), (False, True)),       # pieces of a second pass, folded into what the first has written
    ((149, 25, 41, 3, 15, 16, 2), (False, True)),     # a tail of one image-2 tile behind a wave
    ((1, 37, 53, 21, 37, 40, 6), (True, True)),       # both, two passes, odd sizes
]


def launches(call):
    """What the call returns, and the launches of every kind of gradient GEMM in it (two when its tiles are cut: the pieces are
    folded by a kernel of their own)."""
    _lib.kernel_timing(True)
    out = call()
    report = {name: n for name, _, n in _lib.kernel_timing_report() if name.startswith("grad_gemm")}
    _lib.kernel_timing(False)
    return out, report


def mean_gradients(D, ints, *shape):
    """Whole multiples k * D with k * D * fl(1 / D) == k in FP32 (1 / 15, say, is rounded so that only some k come back)."""
    k = ints(-3, 3, *shape)
    return torch.where(k * D * (torch.ones(()) / D) == k, k * D, 0.)


@pytest.mark.parametrize("operands", ["fp16", "tf32", "bf16"])
@pytest.mark.parametrize("shape,cut", SHAPES)
def test_exact(shape, cut, operands, cuda_device):
    B, H1, W1, H2, W2, C, Kc = shape
    g = torch.Generator().manual_seed(6)
    ints = lambda lo, hi, *s: torch.randint(lo, hi + 1, s, generator=g).float()
    F1, F2 = ints(-2, 2, B, H1, W1, C), ints(-2, 2, B, H2, W2, C)
    A_u, A_v = ints(0, 2, B, H1, W1, Kc, W2), ints(0, 2, B, H1, W1, Kc, H2)
    gC_u, gC_v = ints(-2, 2, B, H1, W1, Kc, H2), ints(-2, 2, B, H1, W1, Kc, W2)
    gM_u, gM_v = ints(-3, 3, B, H1, W1, 2, H2), ints(-3, 3, B, H1, W1, 2, W2)
    gM_u[..., 1, :], gM_v[..., 1, :] = mean_gradients(W2, ints, B, H1, W1, H2), mean_gradients(H2, ints, B, H1, W1, W2)
    AM_u = torch.randint(0, W2, (B, H1, W1, 1, H2), generator=g, dtype=torch.int32)
    AM_v = torch.randint(0, H2, (B, H1, W1, 1, W2), generator=g, dtype=torch.int32)
    G_max = torch.round(gM_u[..., 1, :, None] / W2) + torch.round(gM_v[..., 1, None, :] / H2)
    G_max.scatter_add_(4, AM_u[..., 0, :, None].long(), gM_u[..., 0, :, None])
    G_max.scatter_add_(3, AM_v[..., 0, None, :].long(), gM_v[..., 0, None, :])
    G_sum = torch.einsum("bijku,bijkv->bijuv", gC_u, A_u) + torch.einsum("bijku,bijkv->bijuv", A_v, gC_v)
    dev = {k: v.to(cuda_device) for k, v in dict(F1=F1, F2=F2, A_u=A_u, A_v=A_v, gC_u=gC_u, gC_v=gC_v, gM_u=gM_u, gM_v=gM_v,
                                                 AM_u=AM_u, AM_v=AM_v).items()}
    d = lambda *names: [dev[n] for n in names]
    passes = (Kc + 3) // 4
    with ops.sweep_operands(operands):
        for name, G, n, call in (
                ("maxavg", G_max, 1, lambda: ops.max_argmax_avg_backward(*d("F1", "F2", "AM_u", "AM_v", "gM_u", "gM_v"))),
                ("compress", G_sum, passes, lambda: ops.compression_backward(*d("F1", "F2", "A_u", "A_v", "gC_u", "gC_v"))[:2]),
                ("fused", G_max + G_sum, 1, lambda: ops.separation_feature_backward(
                    *d("F1", "F2", "AM_u", "AM_v", "gM_u", "gM_v", "A_u", "A_v", "gC_u", "gC_v")))):
            (gF1, gF2), report = launches(call)
            for form in (0, 1):
                assert report[f"grad_gemm_kernel<{name},image{form + 1}-major>"] == n * (2 if cut[form] else 1), (name, report)
            assert torch.equal(gF1.cpu(), torch.einsum("bijuv,buvc->bijc", G, F2)), name
            assert torch.equal(gF2.cpu(), torch.einsum("bijuv,bijc->buvc", G, F1)), name


@pytest.mark.parametrize("operands", ["fp16", "tf32"])
@pytest.mark.parametrize("shape,cut", [SHAPES[3], SHAPES[-3], SHAPES[-1]])
def test_layouts_agree(shape, cut, operands, cuda_device):
    """The gradients of the model's channels-first maps, whose pieces are folded four pixels at a time (odd sizes: unaligned, and
    fewer than four at the end of a row), are those of pixel-major features, bit for bit."""
    B, H1, W1, H2, W2, C, Kc = shape
    g = torch.Generator().manual_seed(11)
    randn = lambda *s: torch.randn(*s, generator=g).to(cuda_device)
    F1, F2 = randn(B, H1, W1, C) / C ** 0.5, randn(B, H2, W2, C)
    maps = [t.permute(0, 3, 1, 2).contiguous() for t in (F1, F2)]
    w_u, w_v = (randn(Kc, 2, 3, 3, 3) * 0.3 for _ in range(2))
    with ops.sweep_operands(operands):
        level = ops.separation_level_forward(F1, F2, w_u, randn(Kc), w_v, randn(Kc))
        rest = (w_u, w_v, *level, randn(*level[0].shape), randn(*level[1].shape))
        pixels, report = launches(lambda: ops.separation_level_backward(F1, F2, *rest))
        channels = ops.separation_level_backward(*maps, *rest, fmaps=True)
    for form in (0, 1):
        assert report[f"grad_gemm_kernel<fused,image{form + 1}-major>"] == (2 if cut[form] else 1), report
    for p, c in zip(pixels[:2], channels[:2]):
        assert torch.equal(p, c.permute(0, 2, 3, 1))


@pytest.mark.parametrize("operands", ["fp16", "bf16", "tf32"])
@pytest.mark.parametrize("H,W", [(55, 128), (135, 240)])
def test_repeated_calls_agree(H, W, operands, cuda_device):
    """Many K blocks through every ring of stages, with the values of one op and of both: the same bits every time."""
    g = torch.Generator(device=cuda_device).manual_seed(5)
    randn = lambda *s: torch.randn(*s, generator=g, device=cuda_device)
    F1, F2 = randn(1, H, W, 256) / 16, randn(1, H, W, 256)
    A_u, A_v = (randn(1, H, W, 4, D).softmax(-1) for D in (W, H))
    gC_u, gC_v, gM_u, gM_v = (randn(1, H, W, K, D) for K in (4, 2) for D in (H, W))
    AM_u, AM_v = (torch.randint(0, n, (1, H, W, 1, D), generator=g, device=cuda_device, dtype=torch.int32) for n, D in ((W, H), (H, W)))

    def run():
        return (list(ops.compression_backward(F1, F2, A_u, A_v, gC_u, gC_v))
                + list(ops.max_argmax_avg_backward(F1, F2, AM_u, AM_v, gM_u, gM_v))
                + list(ops.separation_feature_backward(F1, F2, AM_u, AM_v, gM_u, gM_v, A_u, A_v, gC_u, gC_v)))

    with ops.sweep_operands(operands):
        first = run()
        for _ in range(6):
            for x, y in zip(first, run()):
                assert torch.equal(x, y)
