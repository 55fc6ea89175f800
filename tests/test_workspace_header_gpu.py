"""Calls clear the header of the workspace that they are given: status word, counters and scale slots may hold anything."""
import pytest
import torch

from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("operands", ["fp16", "bf16", "tf32"])
@pytest.mark.parametrize("byte", [0x00, 0x7f, 0xff])
def test_header_is_cleared(operands, byte, cuda_device, monkeypatch):
    g = torch.Generator().manual_seed(5)
    randn = lambda *s: torch.randn(*s, generator=g).to(cuda_device)
    F1, F2 = randn(2, 9, 12, 32), randn(2, 7, 36, 32)
    a_u, a_v = randn(2, 9, 12, 2, 36).softmax(-1), randn(2, 9, 12, 2, 7).softmax(-1)

    def calls():
        return [*ops.max_argmax_avg_forward(F1, F2), *ops.compression_forward(F1, F2, a_u, a_v)]

    with ops.sweep_operands(operands):
        want = calls()
        monkeypatch.setattr(ops, "_workspace", lambda n, dev, stream: torch.full((n,), byte, dtype=torch.uint8, device=dev))
        for x, y in zip(calls(), want):
            assert torch.equal(x, y)
