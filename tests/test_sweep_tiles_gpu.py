"""The correlation sweeps at the edges of their tiles (8 x 32, and 16 x 16 over narrow images), of the two warpgroups that share
one and of the column blocks, and with every number of channels a sweep takes.  Features are small whole numbers and weights multiples of 1/8, so every product
and sum is exact in FP32 whatever its order: results are compared bit for bit, ties included (the lowest index wins)."""
import pytest
import torch

from separableflowthesis_b200 import _lib, ops

pytestmark = pytest.mark.gpu

# (B, H1, W1, H2, W2, Kc)
SHAPES = [(1, 3, 43, h2, w2, kc) for kc, (h2, w2) in enumerate([(4, 16), (5, 31), (8, 32), (9, 33)], 1)] + [
    (2, 1, 128, 3, 17, 4),      # fewer rows than one warpgroup takes
    (1, 8, 17, 12, 64, 1),      # rows of the second warpgroup only in the first tile
    (1, 5, 26, 33, 97, 3),      # a channel without a neighbour, several blocks both ways
    (1, 9, 31, 23, 48, 6),      # two sweeps, half a column block left over
    (150, 1, 5, 9, 33, 2),      # more tiles than SMs
    (149, 1, 5, 17, 97, 3),     # a tail of one tile behind a wave, in four pieces
    (150, 1, 5, 33, 97, 6),     # of two tiles, of samples 148 and 149, two sweeps
]
# image 2 so narrow, or so little wider than a block, that it is swept in tiles of 16 x 16
NARROW = [
    (1, 3, 43, 9, 16, 2),       # one row of the second warpgroup
    (2, 1, 128, 17, 15, 4),     # a row more than a tile
    (1, 5, 26, 40, 1, 3),       # a single column
    (1, 8, 17, 32, 48, 1),      # whole tiles in three blocks
    (1, 9, 31, 48, 47, 6),      # three blocks, two sweeps
    (150, 1, 5, 25, 8, 2),      # more tiles than SMs
    (150, 1, 5, 48, 48, 2),     # a tail of two, in three pieces; the sums on wide tiles in two
]


def features(shape, seed=3):
    B, H1, W1, H2, W2, _ = shape
    g = torch.Generator().manual_seed(seed)
    return (torch.randint(-2, 3, (B, H1, W1, 16), generator=g).float(), torch.randint(-2, 3, (B, H2, W2, 16), generator=g).float())


def first_max(S, dim):
    """Largest entries that are numbers and the lowest index of each."""
    S = S.nan_to_num(nan=-float("inf"))
    m = S.amax(dim)
    n = S.shape[dim]
    index = torch.arange(n).view([-1 if d == dim else 1 for d in range(S.dim())])
    return m, torch.where(S == m.unsqueeze(dim), index, n).amin(dim)


@pytest.mark.parametrize("operands", ["fp16", "tf32"])
@pytest.mark.parametrize("shape", SHAPES + NARROW)
def test_exact(shape, operands, cuda_device):
    F1, F2 = features(shape)
    B, H1, W1, H2, W2, Kc = shape
    g = torch.Generator().manual_seed(4)
    A_u, A_v = (torch.randint(0, 8, (B, H1, W1, Kc, D), generator=g).float() / 8 for D in (W2, H2))
    dev = [t.to(cuda_device) for t in (F1, F2, A_u, A_v)]
    with ops.sweep_operands(operands):
        MA_u, MA_v, AM_u, AM_v = [t.cpu() for t in ops.max_argmax_avg_forward(*dev[:2])]
        M_u, M_v = [t.cpu() for t in ops.max_avg_forward(*dev[:2])]
        C_u, C_v = [t.cpu() for t in ops.compression_forward(*dev)]
    S = torch.einsum("bijc,buvc->bijuv", F1, F2)
    assert torch.equal(ops.corr_volume(*dev[:2]).cpu().view_as(S), S)
    for dim, value, plain, arg in ((4, MA_u, M_u, AM_u), (3, MA_v, M_v, AM_v)):
        m, index = first_max(S, dim)
        assert torch.equal(value[..., 0, :], m) and torch.equal(plain[..., 0, :], m)
        assert torch.equal(arg[..., 0, :].long(), index)
    assert torch.equal(C_u, torch.einsum("bijuv,bijkv->bijku", S, A_u))
    assert torch.equal(C_v, torch.einsum("bijuv,bijku->bijkv", S, A_v))


@pytest.mark.parametrize("shape", [SHAPES[3], SHAPES[6], NARROW[1], NARROW[4]])
def test_entries_that_are_not_numbers_are_passed_over(shape, cuda_device):
    """Also where they fill the rows of a column block; a pixel with no number has the maxima NaN over rows and -inf over
    columns, both at index 0."""
    F1, F2 = features(shape)
    F2[0, 0, :32] = float("nan")
    F2[0, 1, min(3, F2.shape[2] - 1)] = F2[0, 4, 0] = F2[0, -1, -1] = float("nan")
    with ops.sweep_operands("tf32"):
        F1[0, 0, 1] = float("nan")
        MA_u, MA_v, AM_u, AM_v = [t.cpu() for t in ops.max_argmax_avg_forward(F1.to(cuda_device), F2.to(cuda_device))]
    S = torch.einsum("bijc,buvc->bijuv", F1, F2)
    for dim, value, arg, none in ((4, MA_u, AM_u, float("nan")), (3, MA_v, AM_v, -float("inf"))):
        m, index = first_max(S, dim)
        empty = S.isnan().all(dim)
        m, index = torch.where(empty, none, m), torch.where(empty, 0, index)
        assert torch.equal(value[..., 0, :].nan_to_num(nan=7e7), m.nan_to_num(nan=7e7))
        assert torch.equal(arg[..., 0, :].long(), index)


@pytest.mark.parametrize("H2,W2", [(32, 48), (17, 16), (8, 64)])
def test_a_level_sweeps_its_maxima_and_its_sums_each_in_their_tiles(H2, W2, cuda_device):
    """Narrow tiles for the maxima only, for both, for neither.  A sum over n columns of whole numbers times weights that add up to
    one, in FP32, is within n 2^-24 of the largest entry."""
    F1, F2 = features((1, 8, 20, H2, W2, 3))
    g = torch.Generator().manual_seed(8)
    params = [t.to(cuda_device) for t in (torch.randn(3, 2, 3, 3, 3, generator=g) * 0.3, torch.randn(3, generator=g)) * 2]
    sep_u, sep_v, _, _, a_u, a_v = [t.cpu() for t in ops.separation_level_forward(F1.to(cuda_device), F2.to(cuda_device), *params)]
    S = torch.einsum("bijc,buvc->buvij", F1, F2)
    assert torch.equal(sep_v[:, 0], S.amax(2)) and torch.equal(sep_u[:, 0], S.amax(1))
    bound = max(H2, W2) * 2 ** -24 * S.abs().max().item()
    S, a_u, a_v = S.double(), a_u.double(), a_v.double()
    assert (sep_v[:, 2:] - torch.einsum("buvij,bkvij->bkuij", S, a_u)).abs().max() <= bound
    assert (sep_u[:, 2:] - torch.einsum("buvij,bkuij->bkvij", S, a_v)).abs().max() <= bound


@pytest.mark.parametrize("shape", [SHAPES[-2], SHAPES[-1], NARROW[-1]])
def test_the_tails_behind_a_wave_are_cut(shape, cuda_device):
    """What test_exact says of these shapes: the pieces are folded by a launch of their own."""
    F1, F2 = [t.to(cuda_device) for t in features(shape)]
    B, H1, W1, H2, W2, Kc = shape
    A_u, A_v = (torch.ones(B, H1, W1, Kc, D, device=cuda_device) for D in (W2, H2))
    _lib.kernel_timing(True)
    ops.max_argmax_avg_forward(F1, F2)
    ops.compression_forward(F1, F2, A_u, A_v)
    report = {name: n for name, _, n in _lib.kernel_timing_report()}
    _lib.kernel_timing(False)
    assert report["sweep_kernel<maxavg>"] == 2 and report["sweep_kernel<compress>"] == 2 * ((Kc + 3) // 4)
