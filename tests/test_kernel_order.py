"""The order of steps in kernels that hold tensor memory, read from their sources: a wrong one could only be seen as a GPU that hangs."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tinyinfer_b200" / "csrc"


def holders():
    return sorted(p.name for p in CSRC.glob("*.cu") if re.search(r"tmem_alloc\(&|tcgen05\.alloc", p.read_text()))


@pytest.mark.parametrize("name", holders())
def test_blocks_that_may_share_an_sm_find_their_tensor_memory(name):
    """Every kernel's columns and shared memory are held to the rule that keeps an allocation from waiting for a later grid's block, and
    the rule itself leaves no such meeting: an SM has 228 KB, a block 1 KB more than it asks for, and 512 columns."""
    assert "static_assert(tmem_shares_sm(" in (CSRC / name).read_text()
    header = (CSRC / "sm100_ptx.cuh").read_text()
    least = int(re.search(r"TMEM_SHARED_LEAST = (\d+) \* 1024", header).group(1))
    assert "TMEM_SHARED_ALONE = 228 * 1024 - TMEM_SHARED_LEAST;" in header
    assert "shared >= TMEM_SHARED_ALONE || (columns <= 128 && shared >= TMEM_SHARED_LEAST)" in header
    alone = 228 - least
    assert 3 * (least + 1) > 228 and (alone + 1) + (least + 1) > 228 and 2 * 128 <= 512


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu") if re.search(r"tma_load_2d(_pair)?\(|bulk_load\(dst", p.read_text())))
def test_copies_land_whichever_wait_ran_out(name):
    """A wait of any role may run out while the producer has no wait left to notice it: the abort is looked at behind the block's
    last barrier, and shared and tensor memory are given up only then."""
    text = (CSRC / name).read_text()
    assert "1000000ull" not in text
    if name == "attention_mma.cu":                       # no barrier ends the roles: every one that a wait ends stays itself
        waits = re.findall(r"if \(!mbar_wait\(.*\)\) (.*)", text)
        assert waits == ["{ ok = false; break; }", "{ land_copies(abort_flag); return; }"] and "if (!ok) land_copies(abort_flag);" in text
        return
    assert text.count("land_copies(abort_flag);") == 1
    land = text.index("land_copies(abort_flag);")
    if "if (!ok) land_copies(abort_flag);" in text:      # the warp that issues the MMAs, which waits for every copy
        role = text[text.rindex("elect_one()", 0, land):land]
        assert "mbar_wait_warp(" in role and not re.search(r"\bmbar_wait\(", role)
        assert role.count("if (!mbar_wait_warp(") == role.count("{ ok = false; break; }")      # no wait that does not end it
        return
    assert text.rindex("mbar_wait", 0, land) < text.rindex("sync", 0, land)             # every role's waits, the barrier, the look
    freed = re.search(r"tmem_dealloc\(|tcgen05\.dealloc", text)
    assert freed is None or land < freed.start()


def test_a_wait_s_number_names_its_kernel():
    """What a status word tells of a wait that ran out is its number alone."""
    whose = {}
    for path in sorted(CSRC.glob("*.cu")):
        for code in re.findall(r"(?:abort_flag, [pa]\.status|atomicExch\(p\.status), (\d\d)\)", path.read_text()):
            whose.setdefault(code, set()).add(path.name)
    assert len(whose) > 40 and all(len(files) == 1 for files in whose.values()), whose
