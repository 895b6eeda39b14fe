"""Small lattices without a squirmer, whose steps run many to a launch.

Lattices of at most 512 nodes per CTA of a 16-CTA cluster keep their populations
in the cluster's shared memory for all but the last step of a call. The results
must be those of the separate kernels (LBMGPU_BULK=node, read at creation) bit
for bit: runs that start on an even and on an odd step, walls on two, one and no
axes, one node per row, parts that end inside a plane, CTAs left without rows
(3x5x4), the largest size (512 nodes per CTA) and one row more than that (the
separate kernels again). One case is also compared with the oracle, to 1e-10
as everywhere in FP64.
"""
import os

import numpy as np
import pytest

from lbm_solver_3d_b200.params import Params

pytestmark = pytest.mark.gpu

SIZES = [(4, 34, 34, 1, 1), (1, 18, 20, 1, 1), (3, 5, 4, 1, 1), (2, 66, 7, 1, 0), (13, 12, 21, 0, 0), (8, 32, 32, 1, 1),
         (8, 27, 38, 1, 0)]


def make(size, precision, kind, fx=2e-6):
    from lbm_solver_3d_b200.solver import Solver
    nx, ny, nz, wy, wz = size
    old = os.environ.pop("LBMGPU_BULK", None)
    if kind:
        os.environ["LBMGPU_BULK"] = kind
    try:
        return Solver(Params().update(nx=nx, ny=ny, nz=nz, walls_y=wy, walls_z=wz, fx=fx, fy=0.0 if wy else 1e-7, tau=0.8,
                                      precision=precision))
    finally:
        os.environ.pop("LBMGPU_BULK", None)
        if old is not None:
            os.environ["LBMGPU_BULK"] = old


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("size", SIZES)
def test_cluster_steps_bit_identical(size, precision):
    a, b = make(size, precision, None), make(size, precision, "node")
    for n in (1, 6, 2, 35):   # later calls start on an odd step and on an even one
        a.run(n)
        b.run(n)
    assert np.array_equal(a.get_f().view(np.uint8), b.get_f().view(np.uint8))
    for x, y in zip(a.fields(), b.fields()):
        assert np.array_equal(x, y)
    assert np.array_equal(a.wall_force(), b.wall_force())
    a.close(), b.close()


def test_cluster_steps_follow_the_oracle(oracle_mod):
    a = make((4, 34, 34, 1, 1), "fp64", None)
    o = oracle_mod.PortSolver(a.params)
    a.run(300)
    o.run(300)
    flag, rho, u = a.fields()
    flo, ro, uo = o.fields()
    fluid = flo == 0
    assert np.array_equal(flag, flo)
    assert np.linalg.norm(u[fluid] - uo[fluid]) <= 1e-10 * np.linalg.norm(uo[fluid])
    assert np.linalg.norm(rho[fluid] - ro[fluid]) <= 1e-10 * np.linalg.norm(ro[fluid])
    a.close()
