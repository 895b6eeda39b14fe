"""FP64 lattices whose bulk moves more than 200 MB a step, off the staged rows.

Their bulk kernels load a node's populations beside its type. The lattices lie
just above the line (0.66 million nodes): one with rows of odd length (whole
planes' rows as one range), one with rows longer than the staged kernel takes.
Twelve steps, among them a mass-correction step and the storing last step of
two calls, follow the oracle: both sides do the same FP64 operations but for
the order of the force sums (1e-16 each), so fields agree to 1e-11.
"""
import numpy as np
import pytest

from lbm_solver_3d_b200.params import Params

pytestmark = pytest.mark.gpu

DECK = dict(tau=0.9, squirmer=1, radius=5.2, b1=0.02, beta=2.0, traj_every=10)
CASES = {
    "odd rows": dict(DECK, nx=101, ny=85, nz=80, walls_y=1, fx=5e-7, planar=1, angle=20.0),
    "long rows": dict(DECK, nx=288, ny=49, nz=48, walls_y=0, planar=0, ex=0.5, ey=0.6, ez=0.62),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_dense_bulk_follows_the_oracle(case, oracle_mod):
    from lbm_solver_3d_b200.solver import Solver
    p = Params().update(**CASES[case])
    assert 2 * 19 * 8 * p.ncells > 200e6
    s, o = Solver(p), oracle_mod.PortSolver(p)
    s.run(5)
    s.run(7)
    o.run(12)
    flag, rho, u = s.fields()
    flo, ro, uo = o.fields()
    assert np.array_equal(flag, flo)
    fluid = flo == 0
    assert np.linalg.norm(u[fluid] - uo[fluid]) <= 1e-11 * np.linalg.norm(uo[fluid])
    assert np.linalg.norm(rho[fluid] - ro[fluid]) <= 1e-11 * np.linalg.norm(ro[fluid])
    s.close()
