"""The step kernel's lanes exchange the operands of their exit solves through
slots that belong to the warp, numbered within the group that makes the pass.
That is sound only if one group per warp makes the pass at a time, so the group
has to come from a vote of the whole warp; the mask of lanes that happen to be
active together, which may be any part of the warp, is not one."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "modpath-rw_gb300" / "csrc"


def test_no_kernel_takes_a_group_of_lanes_from_the_active_mask():
    for f in sorted(CSRC.glob("*.cu*")):
        assert "__activemask" not in f.read_text(), f.name


def test_the_pass_runs_with_the_lanes_a_whole_warp_voted_for():
    src = (CSRC / "step.cu").read_text()
    vote = re.search(r"(\w+) = __ballot_sync\(FULL, tracks && V\.passes < kMaxStepsPerVisit\);", src)
    calls = re.findall(r"= rw_pass<R, EXP, AXI>\((\w+),", src)
    assert vote and calls == [vote.group(1)]
    # the lanes over the cap, which the vote leaves out, do not make the pass
    assert re.search(r"if \(\+\+V\.passes > kMaxStepsPerVisit\) \{\s*r = PASS_UNDEFINED;\s*\} else \{\s*r = rw_pass", src)
