"""The block ILU sweeps where one warp takes a block: block counts that no
number of warps per CTA divides, every number of warps, both precisions, the
same bits each time; and cells without a coupling: what stands in an unused
cell reaches no other cell."""
import numpy as np
import pytest

from batsrus_b200 import capi
from batsrus_b200.explicit import ExplicitSolver
from batsrus_b200.heat import HeatSolver
from batsrus_b200.heat_params import HeatParams, global_to_blocks, heat_dipole
from batsrus_b200.param import Scheme

pytestmark = pytest.mark.gpu


def system(nRoot, sweeps):
    capi.tune_reset()
    g, Te, b, used, dx = heat_dipole(nRoot=nRoot, seed=9)
    n = 8 * nRoot
    f = [global_to_blocks(a.reshape((n, n, n) + a.shape[1:]), nRoot) for a in (Te, b, used)]
    x = ExplicitSolver(g, Scheme())
    return x, HeatSolver(x, HeatParams(typePrecond="BILU", precondPrecision=sweeps), *f), f[2].astype(bool)


@pytest.mark.parametrize("sweeps", ["fp64", "fp32"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_unused_cells_reach_no_other_cell(sweeps, bad):
    x, h, used = system(2, sweeps)
    assert 0 < (~used).sum() < used.size
    r = np.random.default_rng(5).normal(size=h.shape)
    r[~used] = 0.0
    z = h.precond(r)
    r[~used] = bad
    y = h.precond(r)
    assert np.isfinite(z[used]).all()
    assert np.array_equal(y[used], z[used])
    x.close()


@pytest.mark.parametrize("sweeps", ["fp64", "fp32"])
@pytest.mark.parametrize("nRoot", [1, 3])
def test_any_number_of_warps_gives_the_same_bits(nRoot, sweeps):
    """1 and 27 blocks: the last CTA of 2 and 4 warps has warps without a block"""
    x, h, used = system(nRoot, sweeps)
    r = np.random.default_rng(3).normal(size=h.shape)
    out = {}
    for w in capi.tune_info()["heat_ilu_warps"]["candidates"]:
        capi.tune_set("heat_ilu_warps", w)
        out[w] = h.precond(r)
    capi.tune_reset()
    assert set(out) == {1, 2, 4}
    assert all(np.array_equal(z, out[1]) for z in out.values())
    x.close()
