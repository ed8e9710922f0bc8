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


def test_p_of_the_odd_cta_is_released_to_the_issuer():
    """What the odd CTA's softmax warps have written (P by plain stores, the rescaled O into tensor memory) reaches the UMMAs that the
    even CTA issues through one forwarding thread: ordered behind the tensor-memory accesses, fenced to the async proxy, and released at
    cluster scope."""
    body = _kernels()["smla_fwd_kernel"]
    waits = [m.end() for m in re.finditer(r"mbar_wait\(bar_pfull,[^;]*;", body)]
    calls = [re.findall(r"\b(\w+)\(", body[at:])[:4] for at in waits]
    assert ["tc_fence_after_sync", "fence_proxy_async_smem", "tc_fence_before_sync", "mbar_arrive_cluster_release"] in calls
    assert len(waits) == 2 and not re.search(r"mbar_arrive_cluster_relaxed\([^;]*pfull", body)
    with open(os.path.join(os.path.dirname(SOURCE), "sm100_ptx.cuh")) as f:
        ptx = f.read()
    assert "mbarrier.arrive.release.cluster" in ptx.split("void mbar_arrive_cluster_release")[1].split("}")[0]
