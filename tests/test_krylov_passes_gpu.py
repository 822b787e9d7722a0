"""Gram-Schmidt in two passes per Arnoldi column (krylov_gs_steps = 64) against
one step per pass, on vector lengths below, at and beside the tile of the
passes and on bases up to the longest restart: the solves agree to the rounding
that the heat solve's multi-step test allows (1e-9 of the change of Te; the
inner products differ by their summation order only)."""
import numpy as np
import pytest

from batsrus_b200 import capi
from batsrus_b200.explicit import ExplicitSolver
from batsrus_b200.heat import HeatSolver
from batsrus_b200.heat_params import HeatParams, global_to_blocks, heat_dipole
from batsrus_b200.param import Scheme

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nRoot,m,precond", [(1, 5, "NONE"), (2, 30, "BILU"), (3, 64, "NONE"), (5, 17, "NONE")])
def test_two_pass_columns_agree_with_single_steps(nRoot, m, precond):
    capi.tune_reset()
    g, Te, b, used, dx = heat_dipole(nRoot=nRoot, seed=5)
    n = 8 * nRoot
    f = [global_to_blocks(a.reshape((n, n, n) + a.shape[1:]), nRoot) for a in (Te, b, used)]
    x = ExplicitSolver(g, Scheme())
    res = {}
    for steps in (1, 64):
        capi.tune_set("krylov_gs_steps", steps)
        h = HeatSolver(x, HeatParams(typePrecond=precond, nKrylovVector=m), *f)
        s = h.advance_semi_impl()
        res[steps] = (s["nMatvec"], h.te())
    assert abs(res[1][0] - res[64][0]) <= 1
    dT = np.abs(res[1][1] - f[0]).max()
    assert np.abs(res[1][1] - res[64][1]).max() <= 1e-9 * dT
    x.close()
    capi.tune_reset()
