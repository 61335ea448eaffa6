"""Every kernel in the library is one that some call launches."""
import re
import shutil
import subprocess

import pytest


def test_no_megakernel_that_no_call_launches(built):
    from sol_b200 import build
    if not shutil.which("nm"):
        pytest.skip("nm not found")
    names = subprocess.run(["nm", str(build.LIB)], check=True, capture_output=True, text=True).stdout
    # pt_megakernel<counting, split, blocks, basic shading>: split samples without counters run on the lean kernel,
    # and the counting kernels always have full shading.
    kernels = set(re.findall(r"13pt_megakernelILb(\d)ELb(\d)ELi\d+ELb(\d)E", names))
    assert kernels == {("0", "0", "0"), ("0", "0", "1"), ("1", "0", "0"), ("1", "1", "0")}
