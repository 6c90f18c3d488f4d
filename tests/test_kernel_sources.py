"""Rules of the kernel sources that no run can show without hanging a GPU."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "bionemo_inference_runtime_b200" / "csrc"


def _kernels():
    """(name, body) of every __global__ function, up to the line of its closing brace."""
    for path in sorted(CSRC.glob("*.cu")):
        for part in re.split(r"\n__global__ ", path.read_text())[1:]:
            name = re.search(r"(\w+)\(", re.sub(r"__launch_bounds__\([^)]*\)", "", part)).group(1)
            yield f"{path.stem}:{name}", part.split("\n}\n")[0]


TENSOR_MEMORY = [(name, body) for name, body in _kernels() if "tmem_alloc(" in body]


def test_all_tensor_memory_kernels_are_seen():
    assert len(TENSOR_MEMORY) == 8


@pytest.mark.parametrize("body", [b for _, b in TENSOR_MEMORY], ids=[n for n, _ in TENSOR_MEMORY])
def test_next_kernel_starts_after_the_allocation_of_tensor_memory(body):
    """Otherwise a block of the next kernel can take the columns and wait for the block that waits for them."""
    alloc, trigger = body.index("tmem_alloc("), [m.start() for m in re.finditer(r"pdl_trigger\(\)", body)]
    barrier = body.index("__syncthreads()", alloc)
    assert trigger and all(t > barrier for t in trigger)
