"""What the device code may not do because its kernels start before the kernels whose results they read are complete."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "heddle_b200" / "csrc"


def test_no_read_only_loads():
    """The read-only path is for memory that nobody writes while the kernel lives.  A kernel that starts early lives while its inputs are
    written, and such a load is free to move in front of grid_wait()."""
    found = []
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        code = re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)
        found += [(path.name, m) for m in re.findall(r"__ldg\s*\(|ld\.global\S*\.nc|__restrict__|__restrict\b", code)]
    assert not found
