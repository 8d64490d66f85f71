"""Order of a kernel's steps that programmatic dependent launch relies on, read from the sources (csrc/pdl.cuh)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nnabla_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def kernels():
    """(file, text) of every kernel's definition, comments taken out."""
    for path in SOURCES:
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for part in re.split(r"\b__global__\b", text)[1:]:
            yield os.path.basename(path), part


ALLOCATING = [(f, t) for f, t in kernels() if re.search(r"tmem_alloc\w*\s*\(", t)]


def test_the_sources_are_found():
    assert {f for f, _ in ALLOCATING} >= {"conv_codes.cuh", "conv_planes.cuh", "conv_wgrad.cuh", "gemm.cuh", "gemm2.cuh",
                                          "narrow_conv.cu"}


@pytest.mark.parametrize("name,text", ALLOCATING, ids=[f for f, _ in ALLOCATING])
def test_the_successor_is_let_in_behind_the_allocation_of_tensor_memory(name, text):
    """A block whose allocation has to wait for another stream's kernel must not have let its own successor in: the
    successor's blocks allocate too, and hold what they got until this kernel has completed."""
    allocated = re.search(r"tmem_alloc\w*\s*\(", text).end()
    for trigger in re.finditer(r"\bpdl_trigger\(\)", text):
        assert trigger.start() > allocated
        assert re.search(r"__syncthreads\(\)|cluster_sync\(", text[allocated:trigger.start()]), name
