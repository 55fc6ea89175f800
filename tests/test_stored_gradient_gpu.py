"""The gradient GEMMs that hand G = dLoss/dS over through memory: with room for all samples, for some at a time, and for none (G is then
generated twice).  Small whole numbers, exact whatever the order of the sums, compared bit for bit."""
import pytest
import torch

from separableflowthesis_b200 import _lib, ops

pytestmark = pytest.mark.gpu


# (B, H1, W1, H2, W2, C, Kc): tiles of 256 image-2 pixels (four blocks of 4 x 16) and of 128 image-1 pixels, one short, whole, one over
@pytest.mark.parametrize("shape", [(150, 1, 3, 16, 33, 8, 1), (75, 8, 17, 17, 31, 40, 6), (2, 8, 16, 64, 80, 64, 2), (3, 3, 43, 65, 65, 136, 3),
                                   (3, 11, 47, 67, 63, 256, 4)])
@pytest.mark.parametrize("operands", ["fp16", "bf16"])
def test_exact(shape, operands, cuda_device, monkeypatch):
    B, H1, W1, H2, W2, C, Kc = shape
    g = torch.Generator().manual_seed(8)
    ints = lambda lo, hi, *s: torch.randint(lo, hi + 1, s, generator=g).float()
    F1, F2 = ints(-2, 2, B, H1, W1, C), ints(-2, 2, B, H2, W2, C)
    A_u, A_v = ints(0, 2, B, H1, W1, Kc, W2), ints(0, 2, B, H1, W1, Kc, H2)
    gC_u, gC_v = ints(-2, 2, B, H1, W1, Kc, H2), ints(-2, 2, B, H1, W1, Kc, W2)
    G = torch.einsum("bijku,bijkv->bijuv", gC_u, A_u) + torch.einsum("bijku,bijkv->bijuv", A_v, gC_v)
    want = torch.einsum("bijuv,buvc->bijc", G, F2), torch.einsum("bijuv,bijc->buvc", G, F1)
    args = [t.to(cuda_device) for t in (F1, F2, A_u, A_v, gC_u, gC_v)]
    sample = -(-H2 // 4) * -(-W2 // 16) * (-(-(H1 * W1) // 128) * 128) * 128   # bytes of a sample's G
    passes = -(-Kc // 4)
    for missing in (0, 1, B - 1, B):   # samples that the buffer has no room for
        monkeypatch.setattr(ops, "_workspace", lambda n, dev, stream: torch.empty(n - missing * sample, dtype=torch.uint8, device=dev))
        _lib.kernel_timing(True)
        with ops.sweep_operands(operands):
            gF1, gF2 = ops.compression_backward(*args)[:2]
        report = {name: n for name, _, n in _lib.kernel_timing_report()}
        _lib.kernel_timing(False)
        chunks = -(-B // (B - missing)) if missing < B else 1
        for form in (1, 2):   # (a chunk's tiles may be cut into pieces, which a launch of their own folds)
            assert passes * chunks <= report[f"grad_gemm_kernel<compress,image{form}-major>"] <= 2 * passes * chunks, (missing, report)
        assert torch.equal(gF1.cpu(), want[0]) and torch.equal(gF2.cpu(), want[1]), missing
