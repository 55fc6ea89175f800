"""Changes of layout: between the reference's and the library's, in patches of 32 pixels (small launches) and of 128, a batch
whose tensors take the long ones against its samples alone, which take the short ones; channel-major copies."""
import pytest
import torch

from oracle import separation_oracle as orc
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H1,W1", [(9, 14), (8, 16), (11, 3), (25, 31)])
@pytest.mark.parametrize("H2,W2", [(31, 33), (32, 64), (65, 5)])
def test_batch_and_its_samples(H1, W1, H2, W2, cuda_device):
    K = 3
    # patches of 128 pixels x 32 displacements: at least four per SM in the batch, fewer in a sample
    per_sample = -(-H1 * W1 // 128) * (-(-H2 // 32) + -(-W2 // 32)) * 2
    assert per_sample * K < 4 * 148
    B = -(-4 * 148 // per_sample)
    g = torch.Generator(device=cuda_device).manual_seed(H1 * W2)
    randn = lambda *s: torch.randn(*s, generator=g, device=cuda_device)
    F1, F2 = randn(B, H1, W1, 16), randn(B, H2, W2, 16)
    a_u, a_v = randn(B, H1, W1, K, W2).softmax(-1), randn(B, H1, W1, K, H2).softmax(-1)
    with ops.sweep_operands("bf16"):   # no scales, which are of a call's whole tensors
        batch = [*ops.max_argmax_avg_forward(F1, F2), *ops.compression_forward(F1, F2, a_u, a_v)]
        for b in {0, B // 2, B - 1}:
            f1, f2, w_u, w_v = [t[b:b + 1].clone() for t in (F1, F2, a_u, a_v)]
            alone = [*ops.max_argmax_avg_forward(f1, f2), *ops.compression_forward(f1, f2, w_u, w_v)]
            for x, y in zip(batch, alone):
                assert torch.equal(x[b:b + 1], y)


# as GRAD_TOL of tests/test_attention_tiles_gpu.py; 7 mantissa bits for bfloat16
@pytest.mark.parametrize("operands,tol", [("fp16", 1e-3), ("bf16", 1e-2), ("tf32", 1e-3)])
@pytest.mark.parametrize("W2", [2, 15, 16, 17, 63, 64, 65, 80, 130])
def test_channel_major_copies(W2, operands, tol, cuda_device):
    """Feature gradients, whose products read channel-major copies made of 64 pixels x 32 channels at a time."""
    B, H1, W1, H2, C, K = 2, 5, 13, 6, 48, 2
    g = torch.Generator().manual_seed(W2)
    F1, F2 = torch.randn(B, H1, W1, C, generator=g) / 7, torch.randn(B, H2, W2, C, generator=g)
    a_u, a_v = torch.randn(B, H1, W1, K, W2, generator=g).softmax(-1), torch.randn(B, H1, W1, K, H2, generator=g).softmax(-1)
    args = (F1, F2, a_u, a_v, torch.randn(B, H1, W1, K, H2, generator=g), torch.randn(B, H1, W1, K, W2, generator=g))
    with ops.sweep_operands(operands):
        out = ops.compression_backward(*[t.to(cuda_device) for t in args])
    for x, ref in zip(out[:2], orc.compression_backward(*[t.double() for t in args])):
        assert (x.double().cpu() - ref).norm() < tol * ref.norm()
