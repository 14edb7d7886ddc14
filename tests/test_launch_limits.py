"""The limit on a kernel's dynamic shared memory is an attribute of the kernel on one device.  A
process-wide flag that it has been set leaves a second device without it, and its launches fail
there; read from the sources, since that needs two GPUs to see."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "msbg-flip_b200",
                    "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


@pytest.mark.parametrize("name", FILES)
def test_no_process_wide_flag_guards_a_limit(name):
    with open(os.path.join(CSRC, name)) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    if "cudaFuncSetAttribute" in src:
        # (a mask with a bit per device, as in mcf.cu, is fine)
        assert not re.search(r"static\s+(std::atomic<bool>|bool|std::once_flag)\b", src)
