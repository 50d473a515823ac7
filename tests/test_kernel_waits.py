"""How the kernels wait for the grids before them on the stream, as the sources have it: a load of what such a grid writes
must depend on the wait by its address, for a memory clobber holds back neither read-only loads nor __ldcg."""
import os
import re

import pytest

from rode_b200 import build

SOURCES = sorted(f for f in os.listdir(build.CSRC) if f.endswith((".cu", ".cuh")))


def _code(name):
    with open(os.path.join(build.CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", [s for s in SOURCES if s != "rode_common.cuh"])
def test_waits_go_through_the_shared_helpers(name):
    code = _code(name)
    assert "griddepcontrol" not in code
    kernels = re.split(r"(?=__global__)", code)[1:]
    for kernel in kernels:
        for wait in re.finditer(r"(\w+) = after_chain\((\w+)\)", kernel):
            new, old = wait.groups()
            body = kernel[wait.end():]
            body = body[:body.find("\n}")]
            assert new == old or not re.search(rf"\b{old}\b", body), f"{old} is read behind the wait through its old name"


def test_what_is_waited_for_is_read_through_the_result_of_the_wait():
    """The partial rows by their pointer, the list of SDDMM's pieces by the index."""
    assert "after_chain(partial)" in _code("rode_spmm.cu")
    pieces = re.split(r"(?=__global__)", _code("rode_sddmm.cu"))
    pieces = next(k for k in pieces if "sddmm_pieces(OrderHead" in k)
    assert "b2 = after_chain(blockIdx.x)" in pieces and "chain_wait()" not in pieces
