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


def test_residual_copies_are_waited_for():
    """Pair GEMM: between the copy of a residual into the CTA's shared memory and the wait for it there is no way out, also where another
    wait gives up."""
    code = re.sub(r"//[^\n]*", "", (CSRC / "gemm_sm100.cuh").read_text())
    copied = code.index("tma_load_3d(my_slabs")
    waited = code.index("mbar_wait_warp(&s.res_full", copied)
    assert not re.search(r"\b(break|return|continue)\b", code[copied:waited])
