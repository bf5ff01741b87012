"""The kernel's warps share out registers at its start; taking more than the launch gave would wait for ever,
outside every bounded wait. The host refuses a kernel that was built with too few."""
import os
import subprocess

from tests.helpers import ROOT

CHECK = """
#include "stage_table.h"
using mononn::register_split_fits;
static_assert(register_split_fits(168), "what 384 threads can have");
static_assert(!register_split_fits(160) && !register_split_fits(167) && !register_split_fits(0), "too few");
"""


def test_a_kernel_with_too_few_registers_is_refused(tmp_path):
    src = tmp_path / "check.cc"
    src.write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-I", os.path.join(ROOT, "mononn_b200", "csrc"), str(src)],
                   check=True)
    for name in ("runtime.cu", "noalloc.cu"):  # both places that launch it
        with open(os.path.join(ROOT, "mononn_b200", "csrc", name)) as f:
            assert "register_split_fits(fa.numRegs)" in f.read()
