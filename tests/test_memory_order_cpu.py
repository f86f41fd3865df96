"""Places whose memory order no run can show to be wrong, checked in the source."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "heddle_b200" / "csrc"


def test_h2o_halves_are_read_behind_a_warp_barrier():
    """One lane learns that the other group's half of a sum is there; the others may read it behind a barrier only, since the shuffle that
    tells them orders no memory."""
    code = re.sub(r"//[^\n]*", "", (CSRC / "h2o_sm100.cu").read_text())
    told = code.index("atomicXor(&s.part_first")
    read = code.index("s.part[slot][grp ^ 1]", told)
    assert "__syncwarp()" in code[code.index("__shfl_sync", told):read]
