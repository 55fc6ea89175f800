"""Kernels that are on the device before the one before them has ended: calls back to back, on one stream and on several, and replayed from a
CUDA graph, give the bits of calls with the device idle between them."""
import pytest
import torch

import separableflowthesis_b200 as sfb
from separableflowthesis_b200 import ops

pytestmark = pytest.mark.gpu


def problem(shape, seed, device):
    B, H1, W1, H2, W2, C, K = shape
    g = torch.Generator(device=device).manual_seed(seed)
    randn = lambda *s: torch.randn(*s, generator=g, device=device)
    F1, F2 = randn(B, H1, W1, C) / C ** 0.5, randn(B, H2, W2, C)
    params = [randn(K, 2, 3, 3, 3) * 0.3, randn(K), randn(K, 2, 3, 3, 3) * 0.3, randn(K)]
    g_u, g_v = randn(B, 2 + K, W2, H1, W1), randn(B, 2 + K, H2, H1, W1)
    a_u, a_v = randn(B, H1, W1, K, W2).softmax(-1), randn(B, H1, W1, K, H2).softmax(-1)
    return F1, F2, params, g_u, g_v, a_u, a_v


def steps(p):
    """One step after the other as they depend on each other: results of a step."""
    F1, F2, params, g_u, g_v, a_u, a_v = p
    level = ops.separation_level_forward(F1, F2, *params)
    yield list(level)
    yield list(ops.separation_level_backward(F1, F2, params[0], params[2], *level, g_u, g_v))
    yield list(ops.max_argmax_avg_forward(F1, F2))
    yield list(ops.compression_forward(F1, F2, a_u, a_v))


# a few tiles and cut ones; more than a wave; widths that TMA takes and one that it does not
SHAPES = [(1, 9, 20, 11, 35, 64, 2), (2, 30, 40, 30, 40, 128, 4), (3, 47, 65, 20, 33, 64, 3)]


@pytest.mark.parametrize("shape", SHAPES)
def test_back_to_back_and_apart(shape, cuda_device):
    problems = [problem(shape, seed, cuda_device) for seed in range(3)]
    apart = []
    for p in problems:
        apart.append([])
        for result in steps(p):
            torch.cuda.synchronize()
            apart[-1] += [t.clone() for t in result]
            torch.cuda.synchronize()
    for _ in range(4):
        together = [[t for result in steps(p) for t in result] for p in problems]
        torch.cuda.synchronize()
        for a, b in zip(apart, together):
            assert all(torch.equal(x, y) for x, y in zip(a, b))


def test_on_several_streams(cuda_device):
    problems = [problem(SHAPES[1], seed, cuda_device) for seed in range(3)]
    want = [[t.clone() for result in steps(p) for t in result] for p in problems]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in problems]
    for _ in range(3):
        got = []
        for s, p in zip(streams, problems):
            with torch.cuda.stream(s):
                got.append([t for result in steps(p) for t in result])
        torch.cuda.synchronize()
        for a, b in zip(want, got):
            assert all(torch.equal(x, y) for x, y in zip(a, b))


def test_replayed_from_a_graph(cuda_device, monkeypatch):
    monkeypatch.setenv("SFB_CHECK_DEVICE_STATUS", "0")   # (reads the status word after every call)
    F1, F2, _, _, _, a_u, a_v = problem(SHAPES[1], 5, cuda_device)
    vol1, vol2 = torch.randn(1, 1, 40, 30, 40, device=cuda_device), torch.randn(1, 1, 30, 30, 40, device=cuda_device)
    coords = 20 * torch.rand(1, 2, 30, 40, device=cuda_device)

    def calls():
        block = sfb.CorrBlock1D(vol1, vol2)
        return (*ops.max_argmax_avg_forward(F1, F2), *ops.compression_forward(F1, F2, a_u, a_v), *block(coords), *block(coords + 1))

    side = torch.cuda.Stream()
    with torch.no_grad(), torch.cuda.stream(side):
        calls()   # workspaces of this stream
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(graph, stream=side):
        captured = calls()
    for seed in range(3):
        g = torch.Generator(device=cuda_device).manual_seed(seed)
        F1.copy_(torch.randn(F1.shape, generator=g, device=cuda_device))
        vol1.copy_(torch.randn(vol1.shape, generator=g, device=cuda_device))
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in captured]
        with torch.no_grad():
            want = calls()
        assert all(torch.equal(x, y) for x, y in zip(got, want))
