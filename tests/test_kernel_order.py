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


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu") if re.search(r"tma_load_2d(_pair)?\(|bulk_load\(dst", p.read_text())))
def test_copies_land_whichever_wait_ran_out(name):
    """A wait of any role may run out while the producer has no wait left to notice it: the abort is looked at behind the block's
    last barrier, and shared and tensor memory are given up only then."""
    text = (CSRC / name).read_text()
    assert "1000000ull" not in text
    if name == "attention_mma.cu":                       # no such barrier: every role that a wait ends stays for them itself
        waits = re.findall(r"if \(!mbar_wait\(.*\)\) (.*)", text)
        assert waits == ["{ ok = false; break; }", "{ land_copies(abort_flag); return; }"] and "if (!ok) land_copies(abort_flag);" in text
        return
    assert text.count("land_copies(abort_flag);") == 1
    land = text.index("land_copies(abort_flag);")
    assert text.rindex("mbar_wait", 0, land) < text.rindex("sync", 0, land)             # every role's waits, the barrier, the look
    freed = re.search(r"tmem_dealloc\(|tcgen05\.dealloc", text)
    assert freed is None or land < freed.start()
