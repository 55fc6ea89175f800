"""Calls for whose workspace there is no memory: they do with less where they can, level by level in the end, and give the same results.
The shortage is made by the allocation of the workspace, which refuses sizes from a limit on."""
import math

import pytest
import torch

import separableflowthesis_b200 as sfb
from separableflowthesis_b200 import _lib, ops

pytestmark = pytest.mark.gpu


class Shortage:
    def __init__(self, monkeypatch):
        self.limit, self.asked, self.given = math.inf, [], []
        allocate = ops._workspace

        def refuse(n, device, stream):
            self.asked.append(n)
            if n > self.limit:
                raise torch.OutOfMemoryError("made by the test")
            self.given.append(n)
            return allocate(n, device, stream)

        monkeypatch.setattr(ops, "_workspace", refuse)

    def start(self, limit):
        self.limit, self.asked, self.given = limit, [], []
        ops.release_workspaces()


@pytest.fixture()
def shortage(monkeypatch):
    yield Shortage(monkeypatch)
    ops.release_workspaces()


def relerr(x, ref):
    return ((x.double() - ref.double()).norm() / ref.double().norm().clamp_min(1e-30)).item()


def test_gradients_of_one_level(shortage, cuda_device):
    """G of every sample, or generated twice; whole numbers, exact either way."""
    B, H, W, C, Kc = 3, 65, 64, 64, 2
    g = torch.Generator().manual_seed(1)
    ints = lambda lo, hi, *s: torch.randint(lo, hi + 1, s, generator=g).float().to(cuda_device)
    args = [ints(-2, 2, B, H, W, C), ints(-2, 2, B, H, W, C), ints(0, 2, B, H, W, Kc, W), ints(0, 2, B, H, W, Kc, H), ints(-2, 2, B, H, W, Kc, H),
            ints(-2, 2, B, H, W, Kc, W)]
    want = ops.compression_backward(*args)
    (full,) = shortage.asked
    for _ in range(2):   # the second call does not ask for what there was no memory for
        got = ops.compression_backward(*args)
        assert all(torch.equal(x, y) for x, y in zip(got, want))
        if shortage.limit == math.inf:
            shortage.start(full - 1)
            got = ops.compression_backward(*args)
            assert shortage.asked[0] == full and len(shortage.asked) == 2 and shortage.asked[1] < full
            shortage.asked.clear()
        else:
            assert len(shortage.asked) == 1 and shortage.asked[0] < full
    ops.release_workspaces()
    shortage.asked.clear()
    ops.compression_backward(*args)
    assert shortage.asked[0] == full
    shortage.start(1000)
    for _ in range(2):
        with pytest.raises(torch.OutOfMemoryError):
            ops.compression_backward(*args)


# fmap levels averaged by the block, or read by the caller before the call
@pytest.mark.parametrize("operands", ["fp16", "tf32"])
@pytest.mark.parametrize("read", [False, True])
@pytest.mark.parametrize("shape", [(5, 64, 24, 40, 2, 4), (3, 32, 66, 65, 1, 3)])
def test_pyramid(shape, read, operands, shortage, cuda_device, monkeypatch):
    B, C, H, W, Kc, levels = shape
    g = torch.Generator().manual_seed(2)
    f1, f2 = [torch.randn(B, C, H, W, generator=g).to(cuda_device).requires_grad_(True) for _ in range(2)]
    modules = [torch.nn.Conv3d(2, Kc, 3, padding=1).to(cuda_device) for _ in range(2)]
    leaves = [f1, f2, modules[0].weight, modules[1].weight]
    upstream = [torch.randn(B, (2 + Kc) * levels, D, H, W, generator=g).to(cuda_device) for D in (W, H)]

    together = ops.separation_pyramid_forward

    def no_memory(*args):
        raise torch.OutOfMemoryError("made by the test")

    def step(short_forward, backward_limit):
        shortage.start(math.inf)
        monkeypatch.setattr(ops, "separation_pyramid_forward", no_memory if short_forward else together)
        block = sfb.AlternateCorrBlockSepflow(f1, f2, None, num_levels=levels, support_backward=True)
        if read:
            block.pyramid
        outs = block(None, sep=True, attention_weights=modules)
        shortage.start(backward_limit)
        _lib.kernel_timing(True)
        grads = torch.autograd.grad(outs, leaves, upstream)
        gemms = {name: n for name, _, n in _lib.kernel_timing_report()}["grad_gemm_kernel<fused,image1-major>"]
        _lib.kernel_timing(False)
        return outs, grads, list(shortage.asked), gemms

    with ops.sweep_operands(operands):
        outs, want, (full,), gemms = step(False, math.inf)
        assert gemms <= 2
        # what the call for all levels needs at least, and what its levels take one by one
        sizes = step(False, full - 1)[2]
        if operands == "fp16":
            assert len(sizes) == 2 and sizes[1] < full
        least = sizes[1] if operands == "fp16" else full
        for short_forward, limit in ((False, full - 1), (False, least - 1), (True, math.inf), (True, least - 1)):
            got_outs, got, asked, gemms = step(short_forward, limit)
            assert all(torch.equal(x, y) for x, y in zip(got_outs, outs))
            if short_forward or limit < least:
                assert gemms >= levels and len(asked) >= levels
            for x, ref in zip(got, want):   # sums in other pieces (tests/test_pyramid_levels_gpu.py)
                assert relerr(x, ref) < H * W / 8 * 2 ** -23 + 2e-5, (short_forward, limit)
        with pytest.raises(torch.OutOfMemoryError):
            step(False, 1000)


def test_native_module(cuda_device):
    """The MemorySaver module asks torch's allocator itself, which is given room for the smaller buffer alone."""
    from separableflowthesis_b200 import build
    module = build.load_pybind_module()
    B, H, W, C, Kc = 3, 65, 64, 64, 2
    g = torch.Generator().manual_seed(1)
    ints = lambda lo, hi, *s: torch.randint(lo, hi + 1, s, generator=g).float().to(cuda_device)
    args = [ints(-2, 2, B, H, W, C), ints(-2, 2, B, H, W, C), ints(0, 2, B, H, W, Kc, W), ints(0, 2, B, H, W, Kc, H), ints(-2, 2, B, H, W, Kc, H),
            ints(-2, 2, B, H, W, Kc, W)]
    want = ops.compression_backward(*args)
    shape = _lib.SfbShape(B, H, W, H, W, C, Kc)
    full, least = [f(_lib.OP_COMPRESSION_BACKWARD, shape) for f in (_lib.load().sfb_workspace_bytes, _lib.load().sfb_workspace_least_bytes)]
    assert least + 2 ** 26 < full
    ops.release_workspaces()
    stream = torch.cuda.Stream()   # whose buffer the module does not have yet
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total, before = torch.cuda.get_device_properties(cuda_device).total_memory, torch.cuda.memory_reserved()
    try:
        torch.cuda.set_per_process_memory_fraction((before + full) / total)   # the outputs want some of it, too
        with torch.cuda.stream(stream):
            for _ in range(2):
                got = module.compression_backward(*args)
                assert all(torch.equal(x, y) for x, y in zip(got, want))
        torch.cuda.synchronize()
        assert least <= torch.cuda.memory_reserved() - before < full
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
