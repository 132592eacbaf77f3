"""Properties of the kernels that no run can show, read from their source: a
run only shows what today's compiler and today's waits do."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "taichi_dem_julia_port_gb300" / "csrc"


def code(name):
    """A source file without its comments."""
    src = re.sub(r"/\*.*?\*/", "", (CSRC / name).read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", src)


def test_no_vote_rests_on_the_active_mask():
    """__activemask() names the lanes that happen to run together, not those
    that will reach a point: bits of a shared word, or a vote, taken from it
    can lose the other lanes' share.  Kernels name their lanes by a ballot of
    the whole warp instead."""
    for f in sorted(CSRC.glob("*.cu*")):
        assert "__activemask" not in code(f.name), f.name


def test_device_waits_last_as_long_as_ever():
    """A wait for blocks that still work must not give up on them: 2^24 polls
    (about 4 s) for the grid barrier and the scan's look-back."""
    src = code("dem_kernels.cu")
    limit = re.search(r"kSpinLimit = 1ull << (\d+);", src)
    assert limit and int(limit.group(1)) >= 24
    assert len(re.findall(r"spin_limit = kSpinLimit", src)) == 1  # the grid barrier's default
    assert len(re.findall(r"d\.ctr, kSpinLimit\)", src)) == 2  # both scan sites
