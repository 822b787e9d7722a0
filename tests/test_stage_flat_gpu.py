"""The stage kernels of 1D blocks (one thread per face) and of 2D blocks (one
sweep per direction), which end the time step in the last stage, against the oracle: every block shape, one
block (its own periodic neighbour), odd counts, float sides, both orders, and
step counts that end a call right after one, two and several graph replays,
with a time limit in the last step.  A step's rounding is a few 1e-16; 1e-12
per step is the limit of the parity tests."""
import numpy as np
import pytest

from batsrus_b200 import initial
from batsrus_b200.explicit import ExplicitSolver
from batsrus_b200.grid import BlockGrid
from batsrus_b200.param import Scheme
from oracle import Oracle
from test_parity_gpu import rel_err

pytestmark = pytest.mark.gpu

CASES = [
    # block cells, root blocks, boundary, flux, limiter, order, stages
    ((64, 1, 1), (1, 1, 1), "periodic", "Linde", "mc3", 2, 2),
    ((64, 1, 1), (3, 1, 1), "float", "Rusanov", "minmod", 1, 1),
    ((8, 1, 1), (5, 1, 1), "float", "HLLD", "mc", 2, 2),
    ((8, 8, 1), (1, 1, 1), "periodic", "Rusanov", "minmod", 2, 2),
    ((8, 8, 1), (3, 5, 1), "float", "Linde", "mc3", 2, 2),
    ((8, 8, 1), (7, 2, 1), "periodic", "Roe", "mc", 2, 1),
]


@pytest.mark.parametrize("cells,roots,bc,flux,limiter,order,stages", CASES)
def test_flat_blocks_match_oracle(cells, roots, bc, flux, limiter, order, stages):
    dim = 1 if cells[1] == 1 else 2
    g = BlockGrid.uniform(dim, cells, roots, (0.0,) * 3, (1.0,) * 3, (bc,) * 6)
    s = Scheme(nOrder=order, nStage=stages, typeFlux=flux, typeLimiter=limiter,
               limiterBeta=1.2 if limiter == "mc3" else 1.5, cfl=0.4, gamma=5.0 / 3.0, useDivbSource=dim > 1,
               useHalfStep=True)
    st = initial.orszag_tang_3d(g)
    o, x = Oracle(g, s), ExplicitSolver(g, s)
    o.set_state(st)
    o.exchange_messages()
    x.set_state(st)
    i = g.interior_slices()
    n = 0
    for k in (1, 2, 3, 5):
        x.advance(k)
        o.advance(k)
        n += k
        assert x.time()[2] == n
        assert rel_err(x.get_state()[i], o.get_state()[i]) < 1e-12 * n
    t, dt, _ = x.time()
    limit = t + 1.5 * dt  # the second step is cut at the limit
    x.advance(2, limit)
    o.advance(2, limit)
    assert x.time()[0] == limit
    assert rel_err(x.get_state()[i], o.get_state()[i]) < 1e-12 * (n + 2)
    x.close()


@pytest.mark.parametrize("cells", [8, 64])
@pytest.mark.parametrize("flux,limiter,bc", [("Linde", "mc3", "periodic"), ("HLLD", "mc", "float"),
                                             ("Rusanov", "minmod", "float"), ("Roe", "mc", "periodic")])
def test_1d_powell_source_matches_oracle(cells, flux, limiter, bc):
    """1D blocks with the Powell source and a Bx that varies along x, so that
    div B and each of its parts (inner and at the two faces) are not zero"""
    g = BlockGrid.uniform(1, (cells, 1, 1), (5, 1, 1), (0.0,) * 3, (1.0,) * 3, (bc,) * 6)
    s = Scheme(nOrder=2, nStage=2, typeFlux=flux, typeLimiter=limiter, limiterBeta=1.2, cfl=0.4, gamma=5.0 / 3.0,
               useDivbSource=True, useHalfStep=True)
    st = initial.orszag_tang_3d(g)
    st[..., 4] = 0.5 + 0.3 * st[..., 5]
    assert np.ptp(st[..., 4]) > 0.1
    o, x = Oracle(g, s), ExplicitSolver(g, s)
    o.set_state(st)
    o.exchange_messages()
    x.set_state(st)
    x.advance(6)
    o.advance(6)
    i = g.interior_slices()
    a, b = x.get_state()[i], o.get_state()[i]
    assert rel_err(a, b) < 6e-12
    p = ExplicitSolver(g, Scheme(**{**s.__dict__, "useDivbSource": False}))
    p.set_state(st)
    p.advance(6)
    assert rel_err(p.get_state()[i], b) > 1e-6  # the source is what this test is about
    p.close()
