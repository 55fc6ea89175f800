"""CPU: the order in which the compression sweeps move their row sums.  A warp has two buffers, which its tiles take in turn; the copy of a
buffer to memory is a bulk group, and before a buffer is used again, and a row added to again, the groups of two tiles ago have to be complete.
The kernel waits by counting groups, so every tile has to commit one.  On a GPU a missing wait hides behind the time that a tile takes; here
the waits are checked against a model of the groups, and the model's rule is read from the source."""
import os
import re

import pytest

from separableflowthesis_b200 import build

ROWS, COLUMNS = 8, 32   # of a tile


def source(name):
    return re.sub(r"//.*", "", open(os.path.join(build.CSRC, name)).read())


def body_of(text, start):
    text = text[text.index(start):]
    return text[:text.index("\n}")]


def enclosing(text, at):
    """Headers of the blocks that are open at a place, outermost first."""
    open_blocks = []
    for i, ch in enumerate(text[:at]):
        if ch == "{":
            open_blocks.append(text[text.rfind("\n", 0, i) + 1:i].strip())
        elif ch == "}":
            open_blocks.pop()
    return open_blocks


def epilogue():
    return body_of(source("sweep.cu"), "__device__ void epilogue_compress(")


def commits_in_every_tile():
    text = epilogue()
    commits = [m.start() for m in re.finditer(r"\bbulk_commit\(\);", text)]
    if len(commits) != 1:
        return False
    inside = enclosing(text, commits[0])
    tile = max(i for i, header in enumerate(inside) if header.startswith("for (int ub = 0; ub < sc.n_ub;"))
    return inside[tile + 1:] == ["if constexpr (TMA_ROWS)"]


def test_copies_leave_the_group_to_the_kernel():
    text = source("sm100_primitives.cuh")
    for name in ("tma_store_4d", "tma_add_4d"):
        assert "commit_group" not in body_of(text, f"void {name}("), name
    assert "commit_group" in text[text.index("void bulk_commit()"):].split("\n")[0]


def test_every_tile_is_a_group():
    assert commits_in_every_tile()


def test_the_waits_are_the_modelled_ones():
    text = re.sub(r"\s+", " ", epilogue())
    assert "if (e.lane == 0) { if (sc.n_ub > 1) bulk_wait<1>(); else bulk_wait<0>(); } __syncwarp();" in text
    assert "row_buffer + (t & 1) * " in text and "if (TMA_ROWS && e.lane == 0) bulk_wait_all();" in text


def walk(H2, column_blocks, channels, group, in_every_tile):
    """The first tile of a warp's walk that uses a buffer, or adds to a row, of a copy that may be under way; or None."""
    split = channels <= 2
    rows = ROWS // 2 if split else ROWS
    row0 = group * rows if split else 0
    n_ub = -(-H2 // ROWS)
    groups = []   # committed and perhaps under way: (buffer, first row) of the copy in it, or None
    t = 0
    for vb in range(column_blocks):
        for ub in range(n_ub):
            leave = 1 if n_ub > 1 else 0
            groups = groups[len(groups) - leave:] if leave else []
            u0, buffer = ub * ROWS + row0, t % 2
            under_way = [g for g in groups if g is not None]
            if any(g[0] == buffer for g in under_way):
                return vb, ub
            if min(rows, H2 - u0) > 0:
                if any(g[1] == u0 for g in under_way):
                    return vb, ub
                groups.append((buffer, u0))
            elif in_every_tile:
                groups.append(None)
            t += 1
    return None


@pytest.mark.parametrize("channels", [1, 2, 3, 4])
def test_no_access_overtakes_a_copy(channels):
    for H2 in range(1, 66):
        for column_blocks in range(1, 6):
            for group in (0, 1):
                assert walk(H2, column_blocks, channels, group, commits_in_every_tile()) is None, (H2, column_blocks, group)


def test_the_model_sees_a_tile_without_a_group():
    for H2 in (9, 12, 17, 20, 67):
        assert walk(H2, 2, 2, 1, False) is not None, H2
    assert walk(16, 3, 2, 1, False) is None and walk(12, 3, 4, 1, False) is None and walk(12, 3, 2, 0, False) is None
