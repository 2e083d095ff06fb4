"""Kernels launched dependently (launch_dependent) are resident while the launch
before them in the stream still writes what they read after their wait.  The
read-only load path is defined only for data that nobody writes while the kernel
is resident, and its loads may be moved above the wait: in these kernels it may
serve the tables that no step writes, nothing else."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cupf_b200", "csrc")
KERNELS = [("dense.cuh", "dense_update_kernel"), ("apt_step.cuh", "apt_step_kernel"),
           ("apt_step.cuh", "step_item"), ("ek2d.cuh", "ek2d_march_kernel"),
           ("ek2d.cuh", "ek2d_march32_kernel")]
# orientation table and heights: written by host copies only
CONSTANT = {"a.orient", "a.z"}


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def definition(text, name):
    """Signature and body of function `name`."""
    start = re.search(r"\b%s\s*\(" % name, text).start()
    at = text.index("{", start)
    depth, end = 0, at
    for end in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        if depth == 0:
            break
    return text[start:at], text[at:end + 1]


@pytest.mark.parametrize("name,kernel", KERNELS)
def test_read_only_loads_of_constant_tables_only(name, kernel):
    signature, body = definition(source(name), kernel)
    read = set(re.findall(r"__ldg\s*\(\s*&?\s*([\w.]+)", body))
    assert read <= CONSTANT, read - CONSTANT
    assert "__restrict__" not in signature + body


def test_every_dependently_launched_kernel_is_checked():
    launched = set()
    for f in os.listdir(CSRC):
        launched |= set(re.findall(r"launch_dependent\([^;]*?(\w+_kernel)\b", source(f)))
    assert launched and launched <= {k for _, k in KERNELS}
