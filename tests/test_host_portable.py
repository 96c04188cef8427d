"""The host module asks for no instruction set that the compiler of another host (Arm beside a GB200) does not know."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "r2omni_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_no_x86_targets_off_x86():
    with open(os.path.join(CSRC, "host_ext.cpp")) as f:
        own = re.sub(r"^\s*#\s*include.*$", "", f.read(), flags=re.M)   # the module's own code: other hosts' headers are not here
    out = subprocess.run(["g++", "-E", "-P", "-U__x86_64__", "-U__x86_64", "-D__aarch64__=1", "-x", "c++", "-"], input=own, capture_output=True,
                         text=True, check=True).stdout
    assert "off_ramp" in out
    assert not re.search(r"target_clones|__target__|\btarget\s*\(|optimize\s*\(|immintrin|__builtin_ia32", out)
