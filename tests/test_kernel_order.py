"""Orders inside the kernels that no run can be asked to show, read from the source: what a missing one leads to is a GPU that waits
for good, or a value that is wrong once in a long time."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "test_operator_b200", "csrc", "smla_kernels.cuh")


def _kernels():
    """Name -> body, comments taken out."""
    with open(SOURCE) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    bodies = {}
    for piece in text.split("__global__")[1:]:
        name = re.search(r"(smla_\w+_kernel)\s*\(", piece).group(1)
        depth, start = 0, piece.index("{", piece.index(name))
        for i in range(start, len(piece)):
            depth += {"{": 1, "}": -1}.get(piece[i], 0)
            if depth == 0:
                break
        bodies[name] = piece[start:i]
    return bodies


WITH_TENSOR_MEMORY = ["smla_recompute_pair_kernel", "smla_fwd_kernel", "smla_dkv_pair_kernel", "smla_dq_kernel"]


def test_the_kernels_are_found():
    bodies = _kernels()
    assert sorted(n for n, b in bodies.items() if "tmem_alloc" in b) == sorted(WITH_TENSOR_MEMORY)


@pytest.mark.parametrize("name", WITH_TENSOR_MEMORY)
def test_no_trigger_before_the_tensor_memory_is_allocated(name):
    """A block that lets the next kernel's blocks onto its SM before it has its tensor memory may find it taken by one that waits for
    this kernel to end."""
    body = _kernels()[name]
    alloc = re.search(r"\btmem_alloc\w*\(", body).start()
    allocated = body.index("__syncthreads()", alloc)
    assert all(m.start() > allocated for m in re.finditer(r"\bpdl_trigger\(\)", body))
