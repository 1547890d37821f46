"""Every warp-aligned cluster barrier of the kernels converges its warp right before the
instruction: the aligned forms are undefined for a warp whose lanes arrive apart (a loop over
i = lane; i < M, a branch on one lane), and a cluster that waits for such an arrival may never
go on."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inq-wannier-fork_b200", "csrc")


def test_aligned_cluster_barriers_follow_a_syncwarp():
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        lines = open(path).read().splitlines()
        for n, line in enumerate(lines):
            if re.search(r"asm\b.*barrier\.cluster\.[a-z.]*aligned", line):
                seen += 1
                assert lines[n - 1].strip() == "__syncwarp();", f"{os.path.basename(path)}:{n + 1}"
    assert seen > 0
