"""The turn between two steps of the step kernel, on its source: every lane of warp 0 reads the
step's masks from shared memory and lane 0 overwrites them.  The warp's votes between the two
order no memory accesses, so a warp barrier has to stand there."""
import os

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hpc-ca-phospattern_b200", "csrc")


def test_masks_are_read_before_they_are_overwritten():
    src = open(os.path.join(CSRC, "csp_march.cuh")).read()
    turn = src[src.index("k_march(const __grid_constant__ MarchArgs A)"):]
    read = turn.index("const unsigned done = S.step.updated;")
    write = turn.index("S.step.cur ^= done;")
    assert read < write
    assert "__syncwarp();" in turn[read:write]
