"""The explicit stage kernel in units of 128 cells (quarters of 8^3 blocks,
pairs of 4^3 blocks) against the oracle where its units can go wrong: one
block (its own periodic neighbour), odd block counts (the last pair of 4^3
blocks holds one), float sides, more units than CTAs of one wave, block time
steps put together from the quarters.  FP64 within 1e-12 per step (the
limit of the parity tests; a step's rounding is a few 1e-16), FP32-bulk
within 1e-6 relative L1 (the mode's bound)."""
import numpy as np
import pytest

from batsrus_b200 import configs
from batsrus_b200.explicit import ExplicitSolver
from oracle import Oracle
from test_parity_gpu import rel_err

pytestmark = pytest.mark.gpu

CASES = [
    # cells per block side, root blocks, boundary, flux, limiter, state
    (8, (1, 1, 1), "periodic", "Linde", "mc3", "ot"),
    (8, (3, 1, 2), "float", "HLLD", "mc", "blast"),
    (8, (5, 3, 1), "periodic", "Rusanov", "minmod", "ot"),
    (8, (7, 6, 5), "float", "Linde", "mc", "blast"),
    (4, (1, 1, 1), "periodic", "Linde", "mc3", "ot"),
    (4, (3, 3, 3), "float", "HLLD", "mc", "blast"),
    (4, (5, 1, 1), "periodic", "Roe", "mc3", "ot"),
    (4, (11, 9, 9), "float", "Rusanov", "mc3", "blast"),
]


@pytest.mark.parametrize("cells,roots,bc,flux,limiter,state", CASES)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_units_match_oracle(cells, roots, bc, flux, limiter, state, precision):
    g, s, st, _ = configs.uniform_3d_case(roots, flux, limiter, 1.2 if limiter == "mc3" else 1.5, precision=precision,
                                          nCellBlock=(cells,) * 3, state=state, bc=bc)
    o = Oracle(g, s)
    o.set_state(st)
    o.exchange_messages()
    x = ExplicitSolver(g, s)
    x.set_state(st)
    x.advance(4)
    o.advance(4)
    a, b = x.get_state(), o.get_state()
    i = g.interior_slices()
    if precision == "fp64":
        assert rel_err(a[i], b[i]) < 4e-12
        assert abs(x.time()[0] - o.time()[0]) <= 1e-12 * o.time()[0]
    else:
        l1 = np.abs(a[i] - b[i]).sum() / np.abs(b[i]).sum()
        assert l1 < 1e-6
    # DtMax_B: the next step's time step is their minimum
    dt = x.block_dt()
    assert dt.shape == (g.nBlock,) and (dt > 0).all()
    assert x.set_global_timestep() == s.cfl * dt.min()
    x.close()
