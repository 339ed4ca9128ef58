"""Orders inside the kernels that no run shows reliably, read from their sources."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "speed3r_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def kernels_with_tensor_memory():
    found = []
    for path in SOURCES:
        if os.path.basename(path) == "common.cuh":
            continue
        for m in re.finditer(r"\btmem_alloc\(", code(path)):
            found.append(pytest.param(path, m.start(), id=os.path.basename(path)))
    return found


@pytest.mark.parametrize("path, at", kernels_with_tensor_memory())
def test_next_kernel_starts_after_tensor_memory_is_allocated(path, at):
    """A CTA of the next kernel that allocates first waits for this kernel's end with the columns this CTA waits for.  The
    trigger comes after a barrier behind the allocation."""
    src = code(path)
    start = src.rfind("\n}", 0, at)                    # the function before
    body = src[start:src.find("\n}", at)]
    at -= start
    launch = body.find("griddep_launch()")
    barrier = body.find("__syncthreads()", at)
    assert 0 <= barrier < launch, "griddep_launch() before the barrier behind tcgen05.alloc"
