"""The sweeps and gradient GEMMs with the tiles of their last wave cut into pieces against the same calls with whole tiles.
The library cuts only when the workspace has room for the pieces' scratch, so a buffer that lacks the last bytes of
``sfb_workspace_bytes`` makes the same call run whole tiles; where there is no such scratch, it is refused."""
import ctypes

import pytest
import torch

from separableflowthesis_b200 import _lib, ops

pytestmark = pytest.mark.gpu

# (B, H1, W1, H2, W2, C, Kc), all of them cut
SHAPES = [
    (1, 1, 5, 5, 97, 16, 1),              # one tile of few pixels, four column blocks
    (1, 9, 31, 33, 65, 40, 3),            # three tiles, ragged rows and columns
    (3, 20, 27, 18, 50, 64, 6),           # several samples, two compression sweeps
    (1, 1, 148 * 128 + 1, 17, 49, 8, 2),  # a wave of whole tiles and a tail of one pixel
    (2, 75, 128, 6, 70, 32, 4),           # a tail of two tiles that belong to the second sample
    (1, 16, 16, 131, 33, 256, 2),         # widest features, image 2 higher than wide
    (1, 55, 128, 55, 128, 16, 4),         # several column blocks in every piece
    (3, 47, 156, 47, 156, 8, 3),          # pieces of unequal size behind a wave of whole tiles
]

OPS = {
    # name: (op of sfb_workspace_bytes, entry point)
    "max/avg": (_lib.OP_MAX_AVG_FORWARD, "sfb_max_argmax_avg_forward"),
    "compression": (_lib.OP_COMPRESSION_FORWARD, "sfb_compression_forward"),
    "attention gradients": (_lib.OP_COMPRESSION_FORWARD, "sfb_compression_attention_backward"),
    "max/avg gradients": (_lib.OP_MAX_ARGMAX_AVG_BACKWARD, "sfb_max_argmax_avg_backward"),
    "feature gradients": (_lib.OP_SEPARATION_BACKWARD, "sfb_separation_feature_backward"),
}


def call_with_buffer(name, shape, tensors, missing):
    """One call with a workspace of sfb_workspace_bytes - missing bytes; returns the status."""
    lib = _lib.load()
    op, entry = OPS[name]
    s = _lib.SfbShape(*shape)
    size = lib.sfb_workspace_bytes(op, ctypes.byref(s)) - missing
    ws = torch.zeros(size + 256, dtype=torch.uint8, device=tensors[0].device)
    stream = torch.cuda.current_stream().cuda_stream
    rc = getattr(lib, entry)(*[ctypes.c_void_p(t.data_ptr()) for t in tensors], ctypes.byref(s), ctypes.c_void_p(ws.data_ptr()),
                             ctypes.c_size_t(size), ctypes.c_void_p(stream))
    torch.cuda.synchronize()
    return rc


def call_op(name, shape, missing, data):
    """Outputs of one op, or None when the buffer is refused as too small: without scratch for pieces in the op's workspace,
    that is, where no tile of the shape is cut."""
    B, H1, W1, H2, W2, C, Kc = shape
    dev, d = data["f"][0].device, data
    new = lambda *s, dtype=torch.float32: torch.full(s, 7, dtype=dtype, device=dev)
    maxavg = [new(B, H1, W1, 2, H2), new(B, H1, W1, 2, W2)]
    if name == "max/avg":
        out = maxavg + [new(B, H1, W1, 1, H2, dtype=torch.int32), new(B, H1, W1, 1, W2, dtype=torch.int32)]
        ins = d["f"]
    elif name == "compression":
        out, ins = [new(B, H1, W1, Kc, H2), new(B, H1, W1, Kc, W2)], d["f"] + d["a"]
    elif name == "attention gradients":
        out, ins = [new(B, H1, W1, Kc, W2), new(B, H1, W1, Kc, H2)], d["f"] + d["gc"]
    else:
        out = [new(B, H1, W1, C), new(B, H2, W2, C)]
        ins = d["f"] + d["am"] + d["gm"] + ([] if name == "max/avg gradients" else d["a"] + d["gc"])
    rc = call_with_buffer(name, shape, ins + out, missing)
    if rc == _lib.SFB_ERR_WORKSPACE_TOO_SMALL:
        return None
    assert rc == _lib.SFB_OK, _lib.load().sfb_last_error()
    return out


def make_data(shape, dev):
    B, H1, W1, H2, W2, C, Kc = shape
    g = torch.Generator().manual_seed(41)
    randn = lambda *s: torch.randn(*s, generator=g).to(dev)
    return {"f": [randn(B, H1, W1, C) / C ** 0.5, randn(B, H2, W2, C)],
            "a": [randn(B, H1, W1, Kc, D).softmax(-1) for D in (W2, H2)],
            "gc": [randn(B, H1, W1, Kc, D) for D in (H2, W2)],
            "gm": [randn(B, H1, W1, 2, D) for D in (H2, W2)],
            "am": [torch.randint(0, n, (B, H1, W1, 1, D), generator=g, dtype=torch.int32).to(dev)
                   for n, D in ((W2, H2), (H2, W2))]}


@pytest.mark.parametrize("operands", ["fp16", "tf32", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("name", list(OPS))
def test_pieces_give_what_whole_tiles_give(name, shape, operands, cuda_device):
    """Maxima, arg-maxima, means and the sums of the compression (its attention gradients are the same sums) bit for bit;
    gradients, whose pieces accumulate apart, up to the order of an FP32 sum."""
    with ops.sweep_operands(operands):
        data = make_data(shape, cuda_device)
        cut, whole = call_op(name, shape, 0, data), call_op(name, shape, 256, data)
    assert whole is not None, "this shape is meant to be cut"
    for x, y in zip(cut, whole):
        if name in ("max/avg gradients", "feature gradients"):
            # n products added in FP32 in two orders.  Each addition rounds its running sum by at most 2^-24 of it, and
            # a running sum of terms of random sign stays near the largest result: sqrt(n) independent roundings of
            # 2^-24 of that, the eightfold for the largest of some 10^6 values.
            n = max(shape[1] * shape[2], shape[3] * shape[4])
            assert (x - y).abs().max() <= 8 * n ** 0.5 * 2.0 ** -24 * y.abs().max()
        else:
            assert torch.equal(x, y)


@pytest.mark.parametrize("operands", ["fp16", "tf32", "bf16"])
@pytest.mark.parametrize("shape", [SHAPES[1], SHAPES[5], SHAPES[6], SHAPES[7]])
def test_not_a_number_in_a_later_piece(shape, operands, cuda_device):
    """A NaN feature hides from the maxima what it hides in a whole tile and no more: not the rest of its piece."""
    data = make_data(shape, cuda_device)
    for u, v in ((3, 0), (5, 16), (8, 48), (11, 64), (20, 96), (31, 112), (40, 71)):   # first columns of blocks, one inside
        data["f"][1][-1, min(u, shape[3] - 1), min(v, shape[4] - 1)] = float("nan")
    data["f"][0][-1, shape[1] // 2, 4] = float("nan")   # and a pixel whose every entry is NaN
    with ops.sweep_operands(operands):
        cut, whole = call_op("max/avg", shape, 0, data), call_op("max/avg", shape, 256, data)
    assert whole is not None
    for x, y in zip(cut, whole):
        assert torch.equal(x.isnan(), y.isnan()) and torch.equal(x.nan_to_num(), y.nan_to_num())


def test_a_sample_gives_the_same_in_any_batch(cuda_device):
    """The number of pieces follows the number of tiles, hence the batch; the results of a sample do not (TF32 operands:
    FP16 ones are scaled by the whole batch's magnitude)."""
    B, H1, W1, H2, W2, C, Kc = shape = (5, 37, 128, 30, 90, 32, 3)
    data = make_data(shape, cuda_device)
    with ops.sweep_operands("tf32"):
        full = ops.max_argmax_avg_forward(*data["f"]) + ops.compression_forward(*data["f"], *data["a"])
        for b in range(B):
            f1, f2, a_u, a_v = (t[b:b + 1].contiguous() for t in data["f"] + data["a"])
            for x, y in zip(full, ops.max_argmax_avg_forward(f1, f2) + ops.compression_forward(f1, f2, a_u, a_v)):
                assert torch.equal(x[b:b + 1], y)
