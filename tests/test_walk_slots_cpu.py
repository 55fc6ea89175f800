"""CPU: the walks of the tiled attention kernels are cut for as many blocks as fit on the SMs at a time.  How many do is a matter of the compiled
kernels' registers, so the number is asked for (or held by the launch bounds), of the kernel that is launched; a number written down
beside them holds for one compiler and one form."""
import os
import re

from separableflowthesis_b200 import build


def source():
    return re.sub(r"//.*", "", open(os.path.join(build.CSRC, "attention.cu")).read())


def body(text, start):
    text = text[text.index(start):]
    return text[:text.index("\n}")]


def test_logits_and_input_gradients_ask_for_their_kernels():
    text = source()
    for walks, launcher, kernel in (("logits_walks", "launch_attention_forward", "attention_logits_tiled_kernel"),
                                    ("input_grad_walks", "launch_attention_backward", "attention_input_grad_tiled_kernel")):
        asked = re.findall(r"blocks_per_sm<(\w+)<KC, (?:false, )?(FEED_\w+)>>\(\)", body(text, f"static Walks {walks}("))
        assert sorted(asked) == [(kernel, "FEED_COPIES"), (kernel, "FEED_TMA")]
        assert f"= {walks}(job, count, tiled, tma);" in body(text, f"cudaError_t {launcher}(")
    callers = [m for m in re.finditer(r"\bstencil_walks\(job, count, tiled, (\w+), ", text)]
    assert [m.group(1) for m in callers] == ["per_sm", "per_sm"]
    assert "cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, KERNEL, AT_THREADS, 0)" in body(text, "static int blocks_per_sm()")


def test_the_weight_gradients_hold_to_theirs():
    text = source()
    assert re.search(r"__launch_bounds__\(wg_threads\(FEED\), WG_PER_SM\)\s*attention_weight_grad_tiled_kernel\(", text)
    assert "tiled_walk(blocks * chunks, D, count, WG_PER_SM * SM_COUNT, " in body(text, "static WeightWalks weight_walks(")
