"""CPU: a ring stage that a TMA load fills is handed back behind a cross-proxy fence.  The next load is a write of the async proxy;
an arrive orders only the generic proxy's accesses, so reads that merely come before it in program order may still be under way
when that load's data lands.  What the kernels do about it can be read in their source; values that got mixed up would show on a
GPU only now and then."""
import os
import re

import pytest

from separableflowthesis_b200 import build

SOURCES = ["grad_gemm.cu", "attention.cu"]


@pytest.mark.parametrize("name", SOURCES)
def test_stages_filled_by_tma_are_handed_back_behind_a_fence(name):
    text = open(os.path.join(build.CSRC, name)).read()
    text = re.sub(r"//.*", "", text)
    filled = set(re.findall(r"tma_load_\dd\([^;]*?&sm\.(\w*)full\[", text, flags=re.S))
    assert filled
    arrives = [m for m in re.finditer(r"(mbar_arrive|hand_back_stage)\(&sm\.(\w*)empty\[", text) if m.group(2) in filled]
    assert arrives
    for m in arrives:
        if m.group(1) == "hand_back_stage":
            continue
        # a plain arrive: the fence comes after the last read of a stage
        reads = [r.end() for r in re.finditer(r"load_shared\(|= sm\.\w+\[", text[:m.start()])]
        assert "fence_proxy_async_smem();" in text[reads[-1]:m.start()], text[m.start():m.start() + 60]


def test_a_hand_back_fences_in_every_lane_before_one_arrives():
    text = open(os.path.join(build.CSRC, "sm100_primitives.cuh")).read()
    body = text[text.index("void hand_back_stage("):]
    body = body[:body.index("\n}")]
    fence, together, arrive = (body.index(s) for s in ("fence_proxy_async_smem();", "__syncwarp();", "if (lane == 0) mbar_arrive("))
    assert fence < together < arrive
