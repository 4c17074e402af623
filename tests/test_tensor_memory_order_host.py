"""Kernels that allocate tensor memory let their successor start only behind the allocation.

A programmatic successor's CTA that starts earlier may take columns on this CTA's SM and hold them until this grid has ended, while this CTA waits for them
without a limit.  Read from the sources: on a GPU the wrong order would hang."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "megatron_mixtera_b200" / "csrc"
ALLOCATION = re.compile(r"\btmem_alloc(_pair)?\(tmem_slot")


def kernels(text):
    """(name, body) of every __global__ function with a body."""
    for m in re.finditer(r"__global__\b", text):
        brace, paren = text.find("{", m.end()), text.find(";", m.end())
        if brace < 0 or (0 <= paren < brace):
            continue
        depth, end = 0, brace
        for end in range(brace, len(text)):
            depth += (text[end] == "{") - (text[end] == "}")
            if depth == 0:
                break
        name = re.search(r"(\w+_kernel)\s*\(", text[m.end():brace])
        if name is None:
            continue
        yield name[1], text[brace:end]


FOUND = [(f.name, name, body) for f in sorted(CSRC.glob("*.cu")) for name, body in kernels(re.sub(r"//.*", "", f.read_text())) if ALLOCATION.search(body)]


def test_the_kernels_with_tensor_memory_are_found():
    assert {"paged_prompt_kernel", "latent_prompt_umma_kernel", "gemm_pair_kernel", "gemm_bf16_kernel"} <= {name for _, name, _ in FOUND}
    assert sum(len(ALLOCATION.findall(f.read_text())) for f in CSRC.glob("*.cu")) == len(FOUND)


@pytest.mark.parametrize("name,body", [pytest.param(name, body, id=f"{file}:{name}") for file, name, body in FOUND])
def test_successors_start_behind_the_allocation(name, body):
    allocated = ALLOCATION.search(body).end()
    barrier, release = body.find("__syncthreads()", allocated), body.find("pdl_launch_dependents()")
    assert release < 0 or allocated < barrier < release, name
