"""CPU: what the launches that overlap the end of the kernel before them rest on, read from the source.  A kernel may be on the device before its
predecessor has ended; it has to wait for it before anything else, and in every kernel: the end of a kernel stands for the end of all before
it only if it has waited itself."""
import os
import re

from separableflowthesis_b200 import build


def source(name):
    return re.sub(r"//.*", "", open(os.path.join(build.CSRC, name)).read())


def kernels(text):
    for m in re.finditer(r"__global__", text):
        # the first name( that is not an attribute, its parameter list, its body
        at = m.end()
        while True:
            name = re.compile(r"(\w+)\s*\(").search(text, at)
            depth, end = 1, name.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[end], 0)
                end += 1
            if name.group(1) != "__launch_bounds__":
                break
            at = end
        yield name.group(1), text[text.index("{", end) + 1:].lstrip()


def test_every_kernel_waits_first():
    found = [(name, body) for f in build.SOURCES for name, body in kernels(source(f))]
    assert len(found) >= 39
    for name, body in found:
        assert body.startswith("follow_previous_kernel();") or re.match(r"if \(!cta_has_work\((a\.)?status\)\) return;", body), name


def test_the_wait_comes_before_the_next_launch_is_allowed():
    text = source("sm100_primitives.cuh")
    body = text[text.index("void follow_previous_kernel()"):]
    body = body[:body.index("\n}")]
    assert body.index("griddepcontrol.wait") < body.index("griddepcontrol.launch_dependents")
    helper = text[text.index("bool cta_has_work("):]
    helper = helper[helper.index("{") + 1:].lstrip()
    assert helper.startswith("follow_previous_kernel();")


def test_kernels_are_launched_in_one_way():
    for f in build.SOURCES:
        assert "<<<" not in source(f), f
