"""What the kernels' sources must hold to and no run can show: a wait that runs out is not made to happen on a GPU."""
import glob
import os
import re

import velox_b200.csrc

HERE = os.path.dirname(os.path.abspath(velox_b200.csrc.__file__))


def test_waits_of_whole_warps_have_one_answer():
    """Where a warp goes on as a whole (`tc_elect` names all its lanes), a bounded wait must not run out for some lanes only:
    a lane waits by itself only where it alone runs the code."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(HERE, "*.cu"))):
        with open(path) as f:
            lines = f.read().splitlines()
        if not any("tc_elect()" in line for line in lines):
            continue
        seen += 1
        for i, line in enumerate(lines):
            if not re.search(r"\bmbarrier\.(try|test)_wait|_mbar_(wait|try)\(", line):
                continue
            alone = any(re.search(r"if \(lane == 0\) \{", before) for before in lines[max(0, i - 3):i])
            assert alone, "%s:%d: a wait of single lanes in a role of the whole warp: %s" % (os.path.basename(path), i + 1, line.strip())
    assert seen >= 5
