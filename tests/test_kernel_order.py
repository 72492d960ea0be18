"""The order of steps in kernels that hold tensor memory, read from their sources: a wrong one could only be seen as a GPU that hangs."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tinyinfer_b200" / "csrc"


def holders():
    return sorted(p.name for p in CSRC.glob("*.cu") if re.search(r"tmem_alloc\(&|tcgen05\.alloc", p.read_text()))


@pytest.mark.parametrize("name", holders())
def test_next_grid_begins_when_this_one_has_its_tensor_memory(name):
    """A block of the next grid keeps the columns that it takes until this grid has ended: let go earlier, it could take those that a
    block of this one still waits for."""
    text = (CSRC / name).read_text()
    alloc = re.search(r"tmem_alloc\(&|tcgen05\.alloc", text).start()
    kernel = text.rindex("__global__", 0, alloc)
    barrier = text.index("__syncthreads();", alloc)
    assert "ti_grid_launch_dependents" not in text[kernel:barrier]
    assert "ti_grid_launch_dependents();" in text[barrier:text.index("\n}\n", barrier)]
