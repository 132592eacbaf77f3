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


def kernels(src):
    """Name and body of every __global__ function."""
    for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\s*\([^{;]*\)\s*\{", src):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[at], 0)
            at += 1
        yield m.group(1), src[m.end():at]


def test_no_barrier_after_one_that_gave_up():
    """A grid barrier that gave up leaves arrivals in its word, which would
    release the next one early: kernels that meet at one first look for a
    pending timeout and return."""
    meet = r"grid_sync\(|search_phases<"
    found = {}
    for name, body in kernels(code("dem_kernels.cu")):
        first = re.search(meet, body)
        if first and name != "k_selftest_barrier":  # which has a counter of its own
            found[name] = "kErrTimeout) return;" in body[:first.start()]
    assert set(found) == {"k_search", "k_steps"}
    assert all(found.values()), found
