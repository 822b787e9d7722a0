"""Both sides of a resolution change use the same flux code.  A uniform flow on
a refined grid has equal fluxes on every face, so the flux differences vanish
exactly where a coarse block's face holds the sum of four finer faces of the
same function (areas are powers of two apart, and four equal numbers add up
without rounding): after some steps every cell still holds the same bits.
A coarse side computed by other arithmetic than the finer blocks' own leaves
a remainder of a unit in the last place next to the refined patch."""
import numpy as np
import pytest

from batsrus_b200 import configs, initial
from batsrus_b200.explicit import ExplicitSolver
from batsrus_b200.grid import BlockGrid
from batsrus_b200.param import Scheme

pytestmark = pytest.mark.gpu

STATES = [(0.7, 0.31, -0.23, 0.17, 0.43, 0.29, -0.37, 0.6), (1.3, -0.9, 0.77, 0.1, -0.21, 0.83, 0.39, 0.27),
          (0.11, 0.05, 0.6, -1.7, 0.51, -0.13, 0.07, 1.9)]


@pytest.mark.parametrize("flux,limiter", [("Rusanov", "mc"), ("Linde", "mc3"), ("HLLD", "minmod"), ("Roe", "mc")])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("grid", ["8_mostly", "8_patch", "8_large", "4_patch"])
def test_uniform_flow_stays_uniform(grid, precision, flux, limiter):
    """8^3 blocks, most of them at a resolution change, or one refined block
    in 5^3 or 10^3; one refined block in 5^3 blocks of 4^3"""
    if grid == "8_mostly":
        g = configs.amr_blast(nRoot=2, maxLevel=2, with_state=False)[0]
    else:
        c, r = int(grid[0]), 10 if grid == "8_large" else 5
        g = BlockGrid.adaptive(3, (c,) * 3, (r,) * 3, (-0.5,) * 3, (0.5,) * 3, ("periodic",) * 6, 1,
                               lambda lv, i, j, k: (i, j, k) == (2, 1, 3))
    assert len(set(g.iLevelCoord[:, 0])) > 1
    s = Scheme(nOrder=2, nStage=2, typeFlux=flux, typeLimiter=limiter, limiterBeta=1.2, cfl=0.8, gamma=5.0 / 3.0,
               useDivbSource=True, useHalfStep=True, precision=precision)
    x = ExplicitSolver(g, s)
    for q in STATES:
        x.set_state(initial.uniform(g, q))
        x.set_time(0.0, 0)
        x.advance(5)
        a = x.get_state()[g.interior_slices()].reshape(-1, 8)
        assert np.isfinite(a).all()
        assert (a == a[0]).all(), [int((a[:, v] != a[0, v]).sum()) for v in range(8)]
    x.close()
