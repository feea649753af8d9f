"""A lane that issues copies or MMAs must have observed the barriers that guard them itself.  Kernels issue from the lane that
elect.sync chooses, which need not be lane 0, so no role may wait with lane 0 alone and then issue from an elected lane."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wuda_b200", "csrc")
FILES = sorted(f for f in glob.glob(os.path.join(CSRC, "*.cu*")) if not f.endswith("ptx.cuh"))


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_no_role_waits_by_lane_0_and_issues_by_election(path):
    with open(path) as f:
        roles = re.split(r"// -{20,}", f.read())       # each warp role of a kernel is headed by such a line
    assert [r.split("\n")[0].strip() for r in roles if "mbar_wait_lane0(" in r and "elect_one()" in r] == []
