"""Row sums of the compression sweeps by TMA (16-bit operands, planes of a multiple of 4 pixels) and by red.global (other planes):
the same sums in the same order, over the edges of tiles (8 rows, 32 columns), one and several row and column blocks, every number
of channels of a launch and more than one launch, whole tiles and pieces."""
import pytest
import torch

from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(5, 32, 3, 40), (4, 4, 8, 33), (7, 20, 9, 32), (12, 36, 17, 70), (3, 44, 40, 100), (9, 28, 24, 16)])
@pytest.mark.parametrize("Kc", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("operands", ["fp16", "bf16"])
def test_the_same_sums_with_and_without_tma(size, Kc, operands, cuda_device):
    """An image 1 whose planes TMA takes, and the same with a zero column beside it, whose planes it does not take.  (The column's own
    max/mean channels are zero, as the padding of the attention modules is.)"""
    H1, W1, H2, W2 = size
    B = 2
    assert H1 * W1 % 4 == 0
    g = torch.Generator().manual_seed(Kc + H2)
    F1, F2 = torch.randn(B, H1, W1, 32, generator=g), torch.randn(B, H2, W2, 32, generator=g)
    rows = 1 if H1 % 4 == 0 else 0   # planes of a multiple of 4 rows: a zero row as well, so that they are not
    wide = torch.zeros(B, H1 + rows, W1 + 1, 32)
    wide[:, :H1, :W1] = F1
    assert wide.shape[1] * wide.shape[2] % 4 != 0
    params = [(torch.randn(*s, generator=g) * 0.3).to(cuda_device) for s in ((Kc, 2, 3, 3, 3), (Kc,), (Kc, 2, 3, 3, 3), (Kc,))]
    with ops.sweep_operands(operands):
        tma = ops.separation_level_forward(F1.to(cuda_device), F2.to(cuda_device), *params)
        plain = ops.separation_level_forward(wide.to(cuda_device), F2.to(cuda_device), *params)
        for i in (0, 1, 4, 5):
            assert torch.equal(tma[i], plain[i][..., :H1, :W1]), i
        again = ops.separation_level_forward(F1.to(cuda_device), F2.to(cuda_device), *params)
        for p, q in zip(tma, again):
            assert torch.equal(p, q)
        # the attention gradients are the same kernel with the upstream gradients as weights
        gu, gv = torch.randn(tma[0].shape, generator=g).to(cuda_device), torch.randn(tma[1].shape, generator=g).to(cuda_device)
        pad = lambda t: torch.nn.functional.pad(t, (0, 1, 0, rows))
        b_tma = ops.compression_attention_backward_cf(F1.to(cuda_device), F2.to(cuda_device), gv[:, 2:].contiguous(), gu[:, 2:].contiguous())
        b_plain = ops.compression_attention_backward_cf(wide.to(cuda_device), F2.to(cuda_device), pad(gv[:, 2:]).contiguous(),
                                                        pad(gu[:, 2:]).contiguous())
        for p, q in zip(b_tma, b_plain):
            assert torch.equal(p, q[..., :H1, :W1])


def level(f1, f2, params, scale1):
    return ops.separation_level_forward(f1, f2, *params, True, True, scale1)


# 1 to 4 rows in the last of several row blocks: with one or two channels a group of warps has none of them
@pytest.mark.parametrize("W2", [40, 70])
@pytest.mark.parametrize("H2", [9, 11, 12, 17, 18, 19, 20])
@pytest.mark.parametrize("Kc", [1, 2, 5])
def test_a_last_row_block_of_one_group(H2, W2, Kc, cuda_device):
    g = torch.Generator().manual_seed(H2 * W2 + Kc)
    B, H1, W1, C = 2, 10, 36, 32
    f1, f2 = torch.randn(B, C, H1, W1, generator=g).to(cuda_device), torch.randn(B, C, H2, W2, generator=g).to(cuda_device)
    wide = torch.nn.functional.pad(f1, (0, 1)).contiguous()   # planes of 370 pixels
    params = [(torch.randn(*s, generator=g) * 0.3).to(cuda_device) for s in ((Kc, 2, 3, 3, 3), (Kc,), (Kc, 2, 3, 3, 3), (Kc,))]
    tma, plain = level(f1, f2, params, 1.0), level(wide, f2, params, 1.0)
    for i in (0, 1, 4, 5):
        assert torch.equal(tma[i], plain[i][..., :W1]), i


def test_a_pyramid_with_such_a_level(cuda_device):
    """47 x 156 with four levels: 11 x 39 at the third, in one launch with the others."""
    g = torch.Generator().manual_seed(5)
    B, C, H, W, Kc, levels = 2, 64, 47, 156, 2, 4
    f1, f2 = torch.randn(B, C, H, W, generator=g).to(cuda_device), torch.randn(B, C, H, W, generator=g).to(cuda_device)
    params = [(torch.randn(*s, generator=g) * 0.3).to(cuda_device) for s in ((Kc, 2, 3, 3, 3), (Kc,), (Kc, 2, 3, 3, 3), (Kc,))]
    pyr = [f2]
    for _ in range(levels - 1):
        pyr.append(torch.nn.functional.avg_pool2d(pyr[-1], 2, stride=2).contiguous())
    sep_u, sep_v, buffer = ops.separation_pyramid_forward(f1, pyr, *params, True, 0.125)
    wide = torch.nn.functional.pad(f1, (0, 1)).contiguous()   # planes of 47 * 157 pixels
    saved = ops.separation_pyramid_saved(buffer, f1, pyr, Kc, True)
    for l in range(levels):
        plain = level(wide, pyr[l], params, 0.125)
        su, sv = (sep_u[:, :2 + Kc], sep_v[:, :2 + Kc]) if l == 0 else saved[l][:2]
        assert torch.equal(su, plain[0][..., :W]) and torch.equal(sv, plain[1][..., :W]), l
