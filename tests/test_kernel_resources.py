"""What ptxas says about the stage kernel of 2D blocks: no flux spills registers
to local memory.  A limit of registers below what a flux needs (127 for Rusanov,
146 for Linde, 116 for HLLD and 206 for Roe) costs more than the CTAs that
it makes room for."""
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
    spills = re.findall(r"(\d+) bytes spill stores, (\d+) bytes spill loads", r.stderr)
    assert len(spills) == 4, r.stderr  # one kernel per flux
    assert all(s == ("0", "0") for s in spills), r.stderr
