"""The gradient GEMMs at the edges of their K blocks (4 x 16 image-2 pixels, 32 image-1 pixels) and row tiles, whole and in
pieces.  Features, weights and gradients are small whole numbers (no mean-gradients, whose 1/W2 is not), so dLoss/dS and every
product and sum are exact whatever their order: results are compared bit for bit."""
import pytest
import torch

from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# (B, H1, W1, H2, W2, C, Kc)
SHAPES = [
    (1, 2, 16, 1, 1, 8, 1),        # a single image-2 pixel, one block of image-1 pixels
    (1, 3, 11, 3, 15, 8, 2),       # one pixel more than a block; rows and columns short of one
    (1, 4, 32, 4, 16, 40, 3),      # whole tiles and blocks
    (2, 3, 43, 5, 17, 24, 4),      # one row and column more
    (1, 9, 31, 23, 33, 256, 2),    # several blocks both ways, cut into pieces
    (1, 7, 40, 8, 64, 136, 6),     # two passes over channels, the second added to the first
    (149, 1, 3, 9, 16, 16, 1),     # a tail of one tile behind a wave
]


@pytest.mark.parametrize("operands", ["fp16", "tf32", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
def test_exact(shape, operands, cuda_device):
    B, H1, W1, H2, W2, C, Kc = shape
    g = torch.Generator().manual_seed(6)
    ints = lambda lo, hi, *s: torch.randint(lo, hi + 1, s, generator=g).float()
    F1, F2 = ints(-2, 2, B, H1, W1, C), ints(-2, 2, B, H2, W2, C)
    A_u, A_v = ints(0, 2, B, H1, W1, Kc, W2), ints(0, 2, B, H1, W1, Kc, H2)
    gC_u, gC_v = ints(-2, 2, B, H1, W1, Kc, H2), ints(-2, 2, B, H1, W1, Kc, W2)
    gM_u, gM_v = ints(-3, 3, B, H1, W1, 2, H2), ints(-3, 3, B, H1, W1, 2, W2)
    gM_u[..., 1, :] = gM_v[..., 1, :] = 0
    AM_u = torch.randint(0, W2, (B, H1, W1, 1, H2), generator=g, dtype=torch.int32)
    AM_v = torch.randint(0, H2, (B, H1, W1, 1, W2), generator=g, dtype=torch.int32)
    G_max = torch.zeros(B, H1, W1, H2, W2)
    G_max.scatter_add_(4, AM_u[..., 0, :, None].long(), gM_u[..., 0, :, None])
    G_max.scatter_add_(3, AM_v[..., 0, None, :].long(), gM_v[..., 0, None, :])
    G_sum = torch.einsum("bijku,bijkv->bijuv", gC_u, A_u) + torch.einsum("bijku,bijkv->bijuv", A_v, gC_v)
    dev = {k: v.to(cuda_device) for k, v in dict(F1=F1, F2=F2, A_u=A_u, A_v=A_v, gC_u=gC_u, gC_v=gC_v, gM_u=gM_u, gM_v=gM_v,
                                                 AM_u=AM_u, AM_v=AM_v).items()}
    d = lambda *names: [dev[n] for n in names]
    with ops.sweep_operands(operands):
        got = {"max": ops.max_argmax_avg_backward(*d("F1", "F2", "AM_u", "AM_v", "gM_u", "gM_v")),
               "sum": ops.compression_backward(*d("F1", "F2", "A_u", "A_v", "gC_u", "gC_v"))[:2],
               "both": ops.separation_feature_backward(*d("F1", "F2", "AM_u", "AM_v", "gM_u", "gM_v", "A_u", "A_v", "gC_u", "gC_v"))}
    for name, G in (("max", G_max), ("sum", G_sum), ("both", G_max + G_sum)):
        assert torch.equal(got[name][0].cpu(), torch.einsum("bijuv,buvc->bijc", G, F2)), name
        assert torch.equal(got[name][1].cpu(), torch.einsum("bijuv,bijc->buvc", G, F1)), name


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
