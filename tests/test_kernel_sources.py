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
    assert len(trigger) == 1 and trigger[0] > alloc
    between = body[alloc:trigger[0]]  # the next statement of the allocating warp, or behind the block's barrier
    assert re.fullmatch(r"tmem_alloc\(.*\);\s*", between) or "__syncthreads()" in between
