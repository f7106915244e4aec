"""The no-allocation solve's host code: its objects call no C++ allocator, so that a
call neither takes host memory nor throws through the C entry.  (The names that an
object refers to, as nm lists them; no GPU needed.)"""
import os
import subprocess

import pytest

from frehdc_b200 import build


@pytest.mark.parametrize("source", ["noalloc.cu", "cg_res.cu"])
def test_no_cpp_allocation(source):
    build.build_library()
    names = subprocess.run(["nm", "-u", os.path.join(build.BUILD, source + ".o")], check=True,
                           stdout=subprocess.PIPE, text=True).stdout.split()
    assert "cudaLaunchKernelExC" in names or "cudaLaunchCooperativeKernel" in names
    assert [n for n in names if n.startswith(("_Znw", "_Zna", "_ZdlPv", "_ZdaPv"))
            or "_M_" in n or n.startswith("__cxa_throw")] == []
