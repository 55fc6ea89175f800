"""CPU: the result of a kernel launcher cannot be dropped.  A launcher takes the runtime's error with it when it reports it,
so a step of several launches that ignores one of them would go on with stale data and report success; with the build's
flags such code does not compile."""
import os
import re
import subprocess

from separableflowthesis_b200 import build

SNIPPET = """
#include "kernels.h"
cudaError_t step(cudaStream_t st) {{
  {drop}sfb::launch_lookup_pyramid(sfb::LookupDims{{}}, nullptr, nullptr, st);
  return cudaGetLastError();
}}
"""


def compiles(tmp_path, drop):
    src = tmp_path / "step.cu"
    src.write_text(SNIPPET.format(drop=drop))
    flags = [f for f in build.NVCC_FLAGS if f != "-shared"]
    res = subprocess.run([build._nvcc(), *flags, "-I", build.CSRC, "-c", str(src), "-o", str(tmp_path / "step.o")],
                         capture_output=True, text=True)
    return res.returncode == 0, res.stderr


def test_a_dropped_result_is_an_error(tmp_path):
    ok, err = compiles(tmp_path, "const cudaError_t first = ")
    assert ok, err
    ok, err = compiles(tmp_path, "")
    assert not ok and "launch_lookup_pyramid" in err


def test_every_launcher_is_covered():
    text = open(os.path.join(build.CSRC, "kernels.h")).read()
    launchers = re.findall(r"^(\S*\s?)cudaError_t (launch_\w+)\(", text, flags=re.M)
    assert len(launchers) > 10
    assert all("[[nodiscard]]" in before for before, _ in launchers), launchers
