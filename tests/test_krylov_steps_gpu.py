"""krylov_gs_steps = 0, the default, is what the knob table reports, and leaves
the choice to each solver: all Gram-Schmidt steps of a column in two passes
for heat conduction, three steps per pass for the implicit step.  Any other
value holds for both."""
import numpy as np
import pytest

from batsrus_b200 import capi, configs
from batsrus_b200.explicit import ExplicitSolver
from batsrus_b200.heat import HeatSolver
from batsrus_b200.heat_params import HeatParams, global_to_blocks, heat_dipole
from batsrus_b200.implicit import ImplicitSolver
from batsrus_b200.param import Scheme


def test_the_table_reports_the_value_in_use():
    capi.tune_reset()
    k = capi.tune_info()["krylov_gs_steps"]
    assert k["value"] == 0 and k["tuned"] == 0 and k["candidates"] == [0, 1, 2, 3, 4, 64]
    capi.tune_set("krylov_gs_steps", 64)
    capi.tune_set("krylov_gs_steps", 0)
    assert capi.tune_info()["krylov_gs_steps"]["value"] == 0
    capi.tune_reset()


@pytest.mark.gpu
def test_the_default_is_each_solvers_own():
    res = {}
    for steps in (0, 3, 64):
        capi.tune_reset()
        capi.tune_set("krylov_gs_steps", steps)
        g, Te, b, used, dx = heat_dipole(nRoot=3, seed=5)
        f = [global_to_blocks(a.reshape((24,) * 3 + a.shape[1:]), 3) for a in (Te, b, used)]
        x = ExplicitSolver(g, Scheme())
        h = HeatSolver(x, HeatParams(typePrecond="BILU"), *f)
        h.advance_semi_impl()
        heat = h.te()
        x.close()
        g, s, p, st = configs.jfnk_ot(nRoot=2, precond="BILU")
        x = ExplicitSolver(g, s)
        x.set_state(st)
        im = ImplicitSolver(x, p)
        for _ in range(3):
            im.advance_part_impl()
        res[steps] = (heat, x.get_state())
        x.close()
    capi.tune_reset()
    assert np.array_equal(res[0][0], res[64][0]) and not np.array_equal(res[0][0], res[3][0])
    assert np.array_equal(res[0][1], res[3][1]) and not np.array_equal(res[0][1], res[64][1])
