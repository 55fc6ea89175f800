"""The tiled attention kernels of the level calls at the edges of their tiles (32 columns, 4 rows to a thread, 16 and 8 rows to a
tile), with planes fetched by TMA (image-1 widths that are a multiple of 4) and by copies (other widths), in one piece and in
several, and with more channels than a launch takes."""
import pytest
import torch

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# As in test_attention_walks_gpu.py: FP32 sums of 54 products, then a softmax.
TOL = 2e-5
# Gradients come from volumes of FP16 operands (10 mantissa bits, the library's 1e-3).
GRAD_TOL = 1e-3

SIZES = [(1, 1, 5, 7), (3, 5, 9, 4), (4, 4, 8, 8), (5, 33, 7, 17), (7, 31, 20, 3), (8, 32, 3, 40), (9, 36, 33, 6), (15, 29, 6, 18),
         (16, 64, 17, 16), (17, 65, 5, 65), (33, 100, 12, 130), (47, 35, 70, 9)]


def relerr(a, b):
    return ((a.double().cpu() - b).norm() / b.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("Kc", [1, 2, 3, 4, 5, 7])
def test_tile_edges(size, Kc, cuda_device):
    H1, W1, H2, W2 = size
    B = 2
    g = torch.Generator().manual_seed(31 * Kc + H1 + W1)
    F1, F2 = torch.randn(B, H1, W1, 16, generator=g) / 4, torch.randn(B, H2, W2, 16, generator=g)
    params = [torch.randn(Kc, 2, 3, 3, 3, generator=g) * 0.3, torch.randn(Kc, generator=g),
              torch.randn(Kc, 2, 3, 3, 3, generator=g) * 0.3, torch.randn(Kc, generator=g)]
    w_u, b_u, w_v, b_v = [p.to(cuda_device) for p in params]
    F1d, F2d = F1.to(cuda_device), F2.to(cuda_device)
    level = ops.separation_level_forward(F1d, F2d, w_u, b_u, w_v, b_v)
    sep_u, sep_v, am_u, am_v, a_u, a_v = level
    for sep, a, w, b in ((sep_u, a_u, params[0], params[1]), (sep_v, a_v, params[2], params[3])):
        ref = orc.attention_forward(sep[:, :2].double().cpu(), w.double(), b.double())
        assert relerr(a, ref) < TOL
        # every pixel of its own: the norm of a whole tensor would not show one row or column of a tile
        error = (a.double().cpu() - ref).abs().amax(dim=(1, 2)) / ref.abs().amax(dim=(1, 2))
        assert error.max().item() < 10 * TOL
    g_u, g_v = torch.randn(sep_u.shape, generator=g), torch.randn(sep_v.shape, generator=g)
    out = ops.separation_level_backward(F1d, F2d, w_u, w_v, *level, g_u.to(cuda_device), g_v.to(cuda_device))
    ref = orc.separation_level_backward(F1.double(), F2.double(), params[0].double(), params[2].double(), sep_u.double().cpu(),
                                        sep_v.double().cpu(), am_u.cpu(), am_v.cpu(), a_u.double().cpu(), a_v.double().cpu(),
                                        g_u.double(), g_v.double())
    for i in (0, 1, 2, 4):   # features (through the input gradients) and filters
        assert relerr(out[i], ref[i]) < GRAD_TOL, i
    pixels = (out[0].double().cpu() - ref[0]).norm(dim=-1).max() / ref[0].norm(dim=-1).max()
    assert pixels.item() < 4 * GRAD_TOL
    for x, y in zip(out, ops.separation_level_backward(F1d, F2d, w_u, w_v, *level, g_u.to(cuda_device), g_v.to(cuda_device))):
        assert torch.equal(x, y)


@pytest.mark.parametrize("Kc", [1, 2, 3, 4])
def test_copies_and_tma_agree(Kc, cuda_device):
    """The same pixels in an image whose width TMA takes and in one of another width, with a zero column of image 1 beside them
    (its max/mean channels are zero as the padding is): the same sums in the same order."""
    H1, W1, H2, W2 = 21, 36, 19, 23
    g = torch.Generator().manual_seed(Kc)
    F1, F2 = torch.randn(1, H1, W1, 16, generator=g), torch.randn(1, H2, W2, 16, generator=g)
    wide = torch.cat([F1, torch.zeros(1, H1, 1, 16)], dim=2).contiguous()
    params = [(torch.randn(*s, generator=g) * 0.3).to(cuda_device) for s in ((Kc, 2, 3, 3, 3), (Kc,), (Kc, 2, 3, 3, 3), (Kc,))]
    tma = ops.separation_level_forward(F1.to(cuda_device), F2.to(cuda_device), *params)
    copies = ops.separation_level_forward(wide.to(cuda_device), F2.to(cuda_device), *params)
    for i in (4, 5):
        assert torch.equal(tma[i], copies[i][..., :W1])
