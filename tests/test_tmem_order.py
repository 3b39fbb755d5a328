"""A kernel that allocates tensor memory lets its successor in (programmatic dependent launch) only when every CTA holds what it
allocates: a successor's CTA on the same SM would otherwise take the columns, wait for this grid to end, and never see it end.
Read off the sources, since the fault would be a hang."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "distributed-llm-inferencing_b200", "csrc")


def _kernels():
    """(file, text of a kernel from its __global__ to the next one or the host side) of every kernel that allocates."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for body in text.split("__global__")[1:]:
            if re.search(r"\btmem_alloc\w*\(", body):
                yield os.path.basename(path), body


KERNELS = list(_kernels())


def test_the_kernels_are_found():
    assert {name for name, _ in KERNELS} >= {"attn_prefill_tc.cu", "gemm_pair.cu", "gemm_rows.cu", "gemm_tcgen05.cu"}


@pytest.mark.parametrize("name,body", KERNELS, ids=[name for name, _ in KERNELS])
def test_the_trigger_follows_the_allocation(name, body):
    alloc = re.search(r"\btmem_alloc\w*\(", body).start()
    barrier = re.search(r"\b(__syncthreads|pair_barrier)\(\)", body[alloc:])
    assert barrier, "the block has to learn where its columns are"
    for trigger in re.finditer(r"\bpdl_trigger\(\)", body):
        assert trigger.start() > alloc + barrier.end()
