"""Spheres whose boundary links do not fit the remap's short way.

A list of more than 4096 links (R of about 15) walks the sphere's box on every
step. Node types equal the oracle's exactly and fields and rigid body follow to
1e-10 (the same FP64 operations but for the order of a few sums, over 40 steps),
with a sphere that covers and uncovers nodes on most steps, in a box and next to
a wall. Before and after a load the steps are the same bit for bit.
"""
import numpy as np
import pytest

from lbm_solver_3d_b200.params import Params

pytestmark = pytest.mark.gpu

FAST = dict(b1=0.07, tau=1.0, squirmer=1, traj_every=10)
CASES = {
    "box": dict(FAST, nx=52, ny=50, nz=51, walls_y=0, planar=0, radius=17.3, beta=1.0, ex=0.3, ey=0.5, ez=0.8),
    "wall": dict(FAST, nx=48, ny=50, nz=46, walls_y=1, planar=1, radius=16.1, beta=-2.0, y0=18.4, ex=0.8, ey=-0.6, ez=0.0),
}


def links(flag):
    """Fluid nodes with a particle node among the 18 neighbours."""
    solid = flag == 2
    near = np.zeros_like(solid)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if 0 < abs(dx) + abs(dy) + abs(dz) < 3:
                    near |= np.roll(solid, (dz, dy, dx), (0, 1, 2))
    return int((near & (flag == 0)).sum())


@pytest.mark.parametrize("case", sorted(CASES))
def test_large_sphere_follows_the_oracle(case, oracle_mod):
    from lbm_solver_3d_b200.solver import Solver
    p = Params().update(**CASES[case])
    s, o = Solver(p), oracle_mod.PortSolver(p)
    s.run(20)
    flag0, kept = s.fields()[0], s.checkpoint()
    assert links(flag0) > 4096
    s.run(20)
    o.run(40)
    flag, rho, u = s.fields()
    flo, ro, uo = o.fields()
    assert np.array_equal(flag, flo)
    assert (flag != flag0).sum() > 32
    fluid = flo == 0
    assert np.linalg.norm(u[fluid] - uo[fluid]) <= 1e-10 * np.linalg.norm(uo[fluid])
    assert np.linalg.norm(rho[fluid] - ro[fluid]) <= 1e-10 * np.linalg.norm(ro[fluid])
    a, b = s.squirmer(), o.squirmer()
    for k in ("X", "e", "U", "W"):
        assert np.abs(a[k] - b[k]).max() <= 1e-10, k
    s.restore(kept)
    s.run(20)
    for x, y in zip(s.fields(), (flag, rho, u)):
        assert np.array_equal(x, y)
    s.close()
