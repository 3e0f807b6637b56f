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


def test_the_turned_products_rule_ends_where_the_wrappers_stop_asking():
    """Both sides of every line of the rule (`vx_gemm_turned_wins`), and no product that it wants beyond the rows up to which it is asked."""
    from velox_b200.csrc import ops
    wins = ops.library().vx_gemm_turned_wins
    yes = [(9, 6144, 2560, 0), (32, 6144, 2560, 0), (64, 2560, 9728, 0), (224, 4096, 12288, 0), (257, 4096, 12288, 0), (320, 2560, 9728, 0),
           (256, 1024, 3072, 0), (320, 1024, 3072, 0), (65, 2048, 6144, 0), (192, 2048, 6144, 0), (32, 6144, 1024, 1), (65, 6144, 1024, 1), (256, 6144, 1024, 1), (400, 6144, 1024, 1),
           (224, 12288, 2048, 1), (257, 12288, 2048, 1), (640, 12288, 2048, 1), (33, 19456, 2560, 1), (256, 19456, 2560, 1), (800, 19456, 2560, 1)]
    no = [(8, 6144, 2560, 0), (33, 6144, 2560, 0), (33, 2048, 6144, 0), (193, 2048, 6144, 0), (225, 4096, 12288, 0), (256, 2560, 9728, 0), (321, 2560, 9728, 0), (100, 4096, 4096, 0),
          (9, 32784, 2048, 0), (9, 6144, 2564, 0), (9, 6152, 2560, 0), (33, 6144, 1024, 1), (401, 6144, 1024, 1), (64, 12288, 2048, 1), (225, 12288, 2048, 1),
          (641, 12288, 2048, 1), (801, 19456, 2560, 1)]
    for case in yes:
        assert wins(*case) == 1, case
    for case in no:
        assert wins(*case) == 0, case
    for n, k in [(1024, 8192), (2560, 9728), (6144, 1024), (12288, 2048), (16384, 4096), (24576, 4096)]:
        assert not any(wins(m, n, k, 0) for m in range(ops.TURNED_MAX_ROWS + 1, 2000))
        assert not any(wins(m, n, k, 1) for m in range(ops.TURNED_GATED_MAX_ROWS + 1, 2000))
