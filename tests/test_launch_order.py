"""The order in which the kernels that allocate tensor memory wait for the kernel before them, allocate and let the next one begin. Another
order can only be seen by a kernel of another library that allocates, too, and would end in a wait without a limit: it is checked in the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "triton-flash-attention-with-flexible-masks_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


@pytest.mark.parametrize("name,overlaps", [("fwd.cu", False), ("bwd_dkdv.cu", False), ("bwd_dq.cu", True)])
def test_tensor_memory_is_allocated_between_the_wait_and_the_next_launch(name, overlaps):
    code = _code(name)
    assert code.count("tmem_alloc(") == 1
    alloc = code.index("tmem_alloc(")
    barrier = code.index("__syncthreads();", alloc)
    start = code.rindex("__global__", 0, alloc)
    go = [m.start() for m in re.finditer(r"\b(launch_dependents|follow_stream)\(\);", code) if m.start() > start]
    assert go and go[0] > barrier  # every thread is behind the barrier that the allocating warp has passed
    if overlaps:  # launched behind dK/dV only, whose blocks hold theirs: it waits before it ends
        assert code.index("wait_prerequisites();") > code.index("tmem_dealloc(")
    else:
        assert start < code.index("wait_prerequisites();") < alloc


def test_no_other_kernel_allocates_tensor_memory():
    for name in sorted(os.listdir(CSRC)):
        if name not in ("fwd.cu", "bwd_dkdv.cu", "bwd_dq.cu", "ptx.cuh"):
            assert "tmem_alloc(" not in _code(name), name


@pytest.mark.parametrize("name", sorted(n for n in os.listdir(CSRC) if n.endswith((".cu", ".cuh"))))
def test_no_loads_that_ask_for_read_only_memory(name):
    """A kernel begins while the one before it still writes what it is going to read."""
    assert not re.search(r"__ldg\b|__restrict__|ld\.global(\.\w+)*\.nc\b", _code(name))
