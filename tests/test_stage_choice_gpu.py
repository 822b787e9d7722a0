"""Which kernel the stages of 8^3 blocks run.  In FP64 the kernel of 128-cell
units and the kernel of whole blocks agree to rounding and differ in their last
bits, so the bits tell which one ran."""
import numpy as np
import pytest

from batsrus_b200 import capi, configs, initial
from batsrus_b200.explicit import ExplicitSolver
from batsrus_b200.grid import BlockGrid
from batsrus_b200.param import Scheme

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def fresh_knobs():
    capi.tune_reset()
    yield
    capi.tune_reset()


def run(g, s, st, variant=None, steps=4):
    if variant is not None:
        capi.tune_set("stage_variant", variant)
    x = ExplicitSolver(g, s)
    x.set_state(st)
    x.advance(steps)
    a = x.get_state()[g.interior_slices()]
    x.close()
    capi.tune_reset()
    return a


@pytest.mark.parametrize("flux", ["Rusanov", "Linde", "HLLD"])
def test_variant_3_is_the_whole_block_kernel(flux):
    """stage_variant 3 can be chosen on a uniform grid and is not variant 0
    under another number"""
    g, s, st, _ = configs.uniform_3d_case(3, flux, "mc", 1.5, state="blast")
    a, b = run(g, s, st, 0), run(g, s, st, 3)
    assert not np.array_equal(a, b)
    assert np.abs(a - b).max() <= 4e-13 * np.abs(b).max()


@pytest.mark.parametrize("flux", ["Rusanov", "Linde", "HLLD"])
@pytest.mark.parametrize("name", ["mostly", "patch"])
def test_refined_grids_choose_their_kernel(flux, name):
    """FP64: whole blocks where most blocks (two thirds of 120) are at a
    resolution change, units where few (14 of 132) are.  (In FP32-bulk the two
    kernels give the same bits.)"""
    if name == "mostly":
        g = configs.amr_blast(nRoot=2, maxLevel=2, with_state=False)[0]
    else:
        g = BlockGrid.adaptive(3, (8,) * 3, (5,) * 3, (-0.5,) * 3, (0.5,) * 3, ("periodic",) * 6, 1,
                               lambda lv, i, j, k: (i, j, k) == (2, 1, 3))
    s = Scheme(nOrder=2, nStage=2, typeFlux=flux, typeLimiter="mc", limiterBeta=1.5, cfl=0.8, gamma=5.0 / 3.0,
               useDivbSource=True, useHalfStep=True)
    st = initial.orszag_tang_3d(g)
    a, b = run(g, s, st), run(g, s, st, 3)
    assert np.array_equal(a, b) == (name == "mostly")
    assert np.abs(a - b).max() <= 4e-13 * np.abs(b).max()
