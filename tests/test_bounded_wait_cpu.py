"""CPU: what the kernels with bounded waits have to do so that every wait stays bounded, read from their source."""
import os
import re

from separableflowthesis_b200 import build


def kernels_with_barriers():
    for name in build.SOURCES:
        text = re.sub(r"//.*", "", open(os.path.join(build.CSRC, name)).read())
        for part in re.split(r"(?m)^(?=__global__|template)", text):
            if part.startswith("__global__") and "mbar_init(" in part:
                # up to the end of the function: the first line that is a closing brace
                yield re.search(r"(\w+)\(", part.split(")", 1)[1]).group(1), part[:part.index("\n}")]


def test_the_kernels_are_found():
    names = [name for name, _ in kernels_with_barriers()]
    assert len(names) == 5 and "sweep_kernel" in names and "grad_gemm_kernel" in names, names


def test_a_cta_leaves_early_as_a_whole():
    """The status word can be written by another CTA between the reads of two warps.  A warp that left alone would be missing
    from the barriers, from the barriers' initialisation or from the hand-over of registers, for which no limit exists."""
    for name, body in kernels_with_barriers():
        first = body[body.index("{") + 1:].strip()
        assert re.match(r"if \(!cta_has_work\((a\.)?status\)\) return;", first), name
        assert "volatile int*>(status)" not in body and "volatile int*>(a.status)" not in body, name
    text = open(os.path.join(build.CSRC, "sm100_primitives.cuh")).read()
    helper = text[text.index("bool cta_has_work("):]
    assert "__syncthreads_or(" in helper[:helper.index("\n}")]


def test_a_register_split_is_checked_against_the_compiled_kernel():
    """setmaxnreg.inc waits for registers of the CTA's launch; a kernel compiled for fewer than the split adds up to must be
    refused by the host."""
    sources = [re.sub(r"//.*", "", open(os.path.join(build.CSRC, name)).read()) for name in build.SOURCES]
    split = [text for text in sources if "set_max_registers<" in text]
    assert len(split) == 1
    host = split[0][split[0].index("static cudaError_t launch_one("):]
    host = host[:host.index("\n}")]
    order = [host.index(s) for s in ("cudaFuncGetAttributes(&built, kern)", "register_split_fits(built.numRegs)", "launch_next(kern,")]
    assert order == sorted(order)
    assert len(re.findall(r"launch_\w+\(kern\b", split[0])) == 1 and host.count("auto kern = sweep_kernel<") == split[0].count("= sweep_kernel<") == 1


def test_a_cta_that_gives_up_lets_its_copies_land():
    """Shared memory may go to another CTA when the last warp leaves.  Either all roles meet at the end and wait there, or every
    wait that fails is followed by the pause."""
    for name, body in kernels_with_barriers():
        waits = list(re.finditer(r"mbar_wait\([^;{]*;", body)) + list(re.finditer(r"if \(!mbar_wait\([^{]*", body))
        if not waits:   # the roles are functions of their own: they meet
            assert re.search(r"__syncthreads\(\);\s*if \(wait_ctl_aborted\(&sm\.ctl\)\) \{\s*let_copies_land\(\);", body), name
        for m in waits:
            assert "let_copies_land();" in body[m.start():m.start() + 400], name
