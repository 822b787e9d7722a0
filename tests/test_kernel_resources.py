"""What ptxas says about the stage kernel of 2D blocks: with the registers that
they are launched for, Rusanov, Linde (four CTAs per SM) and HLLD spill none to
local memory.  (Linde with five CTAs and Roe do, and gain by the fifth.)"""
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
        flux, ctas = re.search(r"stage_flat_kernelILi(\d)ELi(\d)E", name).groups()
        spills["Rusanov Linde HLLD Roe".split()[int(flux)], int(ctas)] = (int(st), int(ld))
    assert set(spills) == {("Rusanov", 5), ("Linde", 4), ("Linde", 5), ("HLLD", 5), ("Roe", 5)}, r.stderr
    assert all(spills[q] == (0, 0) for q in (("Rusanov", 5), ("Linde", 4), ("HLLD", 5))), r.stderr
