"""What ptxas says about the stage kernel of 2D blocks: Rusanov, Linde and HLLD
spill no registers to local memory.  A limit below what Linde needs (148) costs
more than the CTA that it makes room for; Roe, which needs 210, runs faster
with 128 and five CTAs per SM."""
import os
import re
import subprocess

from batsrus_b200 import build


def test_2d_stage_kernel_does_not_spill(tmp_path):
    src = "bx_stage_flat.cu"
    cmd = [build.NVCC] + build.ARCH + build.COMMON + dict(build.UNITS)[src] + \
        ["-Xptxas", "-v", "-c", os.path.join(build.CSRC, src), "-o", str(tmp_path / "flat.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    spills = {}
    for name, st, ld in re.findall(r"Function properties for (\S+)\s+\d+ bytes stack frame, (\d+) bytes spill stores, "
                                   r"(\d+) bytes spill loads", r.stderr):
        spills[int(re.search(r"stage_flat_kernelILi(\d)E", name).group(1))] = (int(st), int(ld))
    assert set(spills) == {0, 1, 2, 3}, r.stderr  # one kernel per flux: Rusanov, Linde, HLLD, Roe
    assert all(spills[q] == (0, 0) for q in (0, 1, 2)), r.stderr
