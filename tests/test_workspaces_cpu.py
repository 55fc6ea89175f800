"""CPU: which sizes of workspace are asked for where memory is short (separableflowthesis_b200/ops.py)."""
import pytest
import torch

from separableflowthesis_b200 import ops

DEV = torch.device("cuda", 0)   # (never allocated on: torch.empty is replaced)


@pytest.fixture()
def memory(monkeypatch):
    """Allocations of up to `limit` bytes beside those alive succeed."""
    class Memory:
        limit, asked = 0, []

        def empty(self, n, dtype, device):
            self.asked.append(n)
            if n + sum(ws.numel() for ws in ops._workspaces.values()) > self.limit:
                raise torch.OutOfMemoryError("made by the test")
            return torch.zeros(n, dtype=dtype)

    memory = Memory()
    memory.asked = []
    monkeypatch.setattr(ops.torch, "empty", memory.empty)
    monkeypatch.setattr(ops, "_workspaces", {})
    monkeypatch.setattr(ops, "_too_large", {})
    return memory


def test_less_where_there_is_no_memory(memory):
    memory.limit = 500
    take = lambda n, least, must=True: ops._workspace_or_less(n, lambda: least, DEV, 0, must).numel()
    assert take(800, 300) == 300 and memory.asked == [800, 300]
    assert take(800, 300) == 300 and memory.asked == [800, 300]          # neither is asked for again
    assert take(450, 300) == 450 and memory.asked == [800, 300, 450, 450]   # the smaller buffer went first
    with pytest.raises(torch.OutOfMemoryError):
        take(900, 700)
    assert memory.asked[4:] == [700, 700]   # beside the 450 and without it; 900 is more than what failed before
    del memory.asked[:]
    with pytest.raises(torch.OutOfMemoryError):
        take(900, 700, must=False)
    assert memory.asked == []
    assert ops._workspace_or_less(200, lambda: 100, DEV, 7).numel() == 200   # another stream
    memory.limit = 5000
    assert ops.release_workspaces() > 0
    assert take(900, 700, must=False) == 900 and memory.asked[-1] == 900
    memory.limit = 0
    assert take(900, 100) == 900 and take(850, 100) == 900   # what is there is used


def test_a_buffer_that_is_there_is_used_whatever_failed(memory):
    memory.limit = 500
    with pytest.raises(torch.OutOfMemoryError):
        ops._workspace_or_less(600, lambda: 550, DEV, 0)
    memory.limit = 700
    assert ops._workspace_or_less(600, lambda: 560, DEV, 0).numel() == 560
    memory.limit = 0
    assert ops._workspace_or_less(555, lambda: 100, DEV, 0, must=False).numel() == 560
