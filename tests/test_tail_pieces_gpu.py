"""Contractions whose last wave of tiles is cut into pieces (column blocks of the sweeps, K ranges of the gradient GEMMs)
and put together by a kernel behind them: one tile, a full wave of 148 tiles and one or two more, few column
blocks, ragged edges, several samples, more channels than one sweep takes.  Against the float64 oracle, and bit for bit
against a second run: the pieces are added in a fixed order."""
import pytest
import torch

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu

# operands rounded to 10 mantissa bits, FP32 accumulation: as tests/test_ops_gpu.py
TOL = 1e-3

# (B, H1, W1, H2, W2, C, Kc)
SHAPES = [
    (1, 1, 5, 5, 97, 16, 1),        # one tile of few pixels, four column blocks
    (1, 9, 31, 33, 65, 40, 3),      # three tiles, ragged rows and columns
    (3, 20, 27, 18, 50, 64, 6),     # several samples, two compression sweeps
    (1, 1, 148 * 128, 3, 17, 8, 2),        # exactly one wave: no tail
    (1, 1, 148 * 128 + 1, 17, 49, 8, 2),   # a tail of one pixel
    (2, 75, 128, 6, 70, 32, 4),     # a tail of two tiles that belong to the second sample
    (1, 16, 16, 131, 33, 256, 2),   # widest features, image 2 higher than wide
]


def relerr(x, ref):
    x, ref = x.detach().double().cpu(), ref.detach().double().cpu()
    return ((x - ref).abs().max() / max(x.abs().max().item(), ref.abs().max().item(), 1e-30)).item()


@pytest.mark.parametrize("operands", ["fp16", "tf32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_pieces(shape, operands, cuda_device):
    B, H1, W1, H2, W2, C, Kc = shape
    g = torch.Generator().manual_seed(31)
    F1 = torch.randn(B, H1, W1, C, generator=g) / C ** 0.5
    F2 = torch.randn(B, H2, W2, C, generator=g)
    A_u = torch.randn(B, H1, W1, Kc, W2, generator=g).softmax(-1)
    A_v = torch.randn(B, H1, W1, Kc, H2, generator=g).softmax(-1)
    up = [torch.randn(B, H1, W1, k, D, generator=g) for k, D in ((2, H2), (2, W2), (Kc, H2), (Kc, W2))]
    dev = [t.to(cuda_device) for t in (F1, F2, A_u, A_v, *up)]
    f1, f2, a_u, a_v, gm_u, gm_v, gc_u, gc_v = dev

    def run():
        fw = ops.max_argmax_avg_forward(f1, f2)
        return (list(fw) + list(ops.compression_forward(f1, f2, a_u, a_v))
                + list(ops.max_argmax_avg_backward(f1, f2, fw[2], fw[3], gm_u, gm_v))
                + list(ops.compression_backward(f1, f2, a_u, a_v, gc_u, gc_v)))

    with ops.sweep_operands(operands):
        out, again = run(), run()
    for x, y in zip(out, again):
        assert torch.equal(x, y)
    d = [t.double() for t in (F1, F2, A_u, A_v, *up)]
    ref = list(orc.max_argmax_avg_forward(d[0], d[1]))[:2]
    for x, r in zip(out[:2], ref):
        for ch in (0, 1):
            assert relerr(x[..., ch, :], r[..., ch, :]) < TOL
    # the arg-max points at an entry within tolerance of the maximum
    S = orc.corr_volume(d[0], d[1])
    scale = S.abs().max()
    picked_u = S.gather(4, out[2].cpu()[..., 0, :].long().unsqueeze(-1)).squeeze(-1)
    picked_v = S.gather(3, out[3].cpu()[..., 0, :].long().unsqueeze(-2)).squeeze(-2)
    assert (ref[0][..., 0, :] - picked_u).abs().max() / scale < TOL
    assert (ref[1][..., 0, :] - picked_v).abs().max() / scale < TOL
    for x, r in zip(out[4:6], orc.compression_forward(*d[:4])):
        assert relerr(x, r) < TOL
    am = [t.cpu() for t in out[2:4]]
    for x, r in zip(out[6:8], orc.max_argmax_avg_backward(d[0], d[1], am[0], am[1], d[4], d[5])):
        assert relerr(x, r) < TOL
    for x, r in zip(out[8:12], orc.compression_backward(*d[:4], d[6], d[7])):
        assert relerr(x, r) < TOL


def test_ties_across_pieces(cuda_device):
    """Equal columns that fall into different pieces: the lowest one wins, as within a piece."""
    g = torch.Generator().manual_seed(5)
    F1 = torch.randn(1, 6, 9, 32, generator=g) / 8
    F2 = torch.randn(1, 20, 112, 32, generator=g)
    for v in (35, 70, 111):
        F2[:, :, v] = F2[:, :, 3]
    _, _, AM_u, _ = ops.max_argmax_avg_forward(F1.to(cuda_device), F2.to(cuda_device))
    assert not any((AM_u == v).any() for v in (35, 70, 111)) and (AM_u == 3).any()
