"""A step's kernels run on several streams and any of them may set the run's
status while another starts.  Where threads meet at a barrier, a shuffle or a
block scan they must go on or leave together, so no function that has such a
meeting point may let each thread read the status for itself."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pot_b200", "csrc")
MEETING = re.compile(r"__syncthreads|__syncwarp|_sync\(|group_block_scan|tile_scan|block_sum3|warp_phi|inject<")
OWN_READ = re.compile(r"if \([^\n]*rec->status (?:!=|==) POT_OK")


def functions(text):
    """(first line, body) of the file's top-level functions."""
    for m in re.finditer(r"^\{\n(.*?)^\}", text, re.M | re.S):
        head = text[:m.start()].rstrip().rsplit("\n\n", 1)[-1]
        yield head.splitlines()[-1], m.group(1)


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_one_status_reading_per_meeting(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    bad = [head for head, body in functions(text) if MEETING.search(body) and OWN_READ.search(body)]
    assert not bad, bad


def test_readings_are_found():
    """The scan sees the functions it is meant for."""
    bodies = [b for p in glob.glob(os.path.join(CSRC, "*.cu")) for _, b in functions(open(p).read())]
    assert sum("block_status(rec)" in b for b in bodies) >= 5
    assert sum("warp_status(rec)" in b for b in bodies) >= 6
