"""Short lattices whose wall rows are launched in front of the bulk of their step.

Such a bulk starts beside the wall rows, before it has waited for the bulk of the
step before, and must all the same see everything that one wrote. A call of many
steps takes this way, in the flat kernel (rows of odd length) on all steps but
those with sums, in the staged rows on all. One step per call takes the storing
kernels, where the flat form does not start early. Both orders of the same steps
give the same populations and trajectories bit for bit. A lattice that continues
from a checkpoint taken on another step does too.
"""
import numpy as np
import pytest

from lbm_solver_3d_b200.params import Params

pytestmark = pytest.mark.gpu

DECK = dict(tau=0.9, squirmer=1, walls_y=1, radius=4.4, b1=0.02, beta=2.0, traj_every=5, fx=5e-7)
CASES = {
    "odd rows": dict(DECK, nx=41, ny=30, nz=26, angle=20.0),
    "odd rows, y and z walls": dict(DECK, nx=71, ny=38, nz=44, walls_z=1, angle=-15.0),
    "staged rows": dict(DECK, nx=96, ny=34, nz=30, angle=20.0),
}


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_early_start_bit_identical(case, precision):
    from lbm_solver_3d_b200.solver import Solver
    p = Params().update(precision=precision, **CASES[case])
    a, b, c = Solver(p), Solver(p), Solver(p)
    a.run(97)
    for _ in range(97):
        b.run(1)
    c.run(31)
    kept = c.checkpoint()
    c.run(6)                # the loaded steps have the parity and zone slots of these
    c.restore(kept)
    c.run(66)
    ref = b.get_f()
    for s in (a, c):
        assert np.array_equal(s.get_f().view(np.uint8), ref.view(np.uint8))
        for k in ("X", "e", "U", "W", "Fh", "Th"):
            assert np.array_equal(s.squirmer()[k], b.squirmer()[k]), k
    rows = b.traj_rows()
    assert np.array_equal(a.traj_rows(), rows)
    for s in (a, b, c):
        s.close()
