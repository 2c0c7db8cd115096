"""Rules of the kernel sources that no run can show."""
import glob
import os

from conftest import PKG


def test_aligned_cluster_barriers_follow_a_warp_barrier():
    """barrier.cluster .aligned is defined for converged warps only: the statement
    before it has to be __syncwarp()."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(PKG, "csrc", "*.cu*"))):
        lines = open(path).read().split("\n")
        for i, line in enumerate(lines):
            if "barrier.cluster" in line and ".aligned" in line and "asm" in line:
                seen += 1
                assert lines[i - 1].strip().startswith("__syncwarp();"), (path, i + 1)
    assert seen
