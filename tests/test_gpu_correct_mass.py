"""The explicit mass correction in every storage form and parity.

lbmgpu_correct_mass sums the populations of the fluid nodes and adds w_i (1 -
mean) to each (lbm.cpp:324-339). The populations before and after are read back
in FP64 and compared with numpy: the sums agree to 1e-13 relative (1.3e6 terms,
added in another order), so the correction does to 1e-13 of the mean density of
1, and a stored population to that and one rounding of its form. On a lattice
larger than the L2 the call must not take more than five times a copy of the
bytes it moves (one read, one read and write of the populations) and 60 us:
measured 2 to 2.7 times; 7 to 9 times when it converted them on the way in.
"""
import time

import numpy as np
import pytest

from lbm_solver_3d_b200.params import Params

pytestmark = pytest.mark.gpu

W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
DECK = dict(squirmer=1, b1=0.02, beta=1.0, tau=0.9, mass_correction_every=0)
# one rounding: of the value (FP64), of its deviation from w_i (FP32: 2^-24, FP16: 2^-11, or the smallest step)
ROUND = {"fp64": (2.0 ** -52, 0.0), "fp32": (2.0 ** -23, 1e-30), "fp16": (2.0 ** -10, 2.0 ** -36)}


@pytest.mark.parametrize("steps", [8, 9])
@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp16"])
def test_correction(precision, steps):
    from lbm_solver_3d_b200.solver import Solver
    s = Solver(Params().update(nx=45, ny=40, nz=38, walls_y=1, radius=5.0, angle=20.0, precision=precision, **DECK))
    s.run(steps)
    f = s.get_f() * 1.002   # a mean density well away from 1
    s.set_f(f)
    f = s.get_f()           # as stored
    fluid = s.fields()[0] == 0
    s.correct_mass()
    g = s.get_f()
    w = W[:, None, None, None]
    d = 1.0 - f[:, fluid].sum() / fluid.sum()
    assert abs(d + 0.002) < 1e-3
    want = np.where(fluid[None], f + w * d, f)
    rel, least = ROUND[precision]
    scale = np.abs(want) if precision == "fp64" else np.abs(want - w)
    assert np.all(np.abs(g - want)[:, fluid] <= (2 * rel * scale + least + 1e-13)[:, fluid])
    assert np.array_equal(g[:, ~fluid], f[:, ~fluid])
    s.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp16"])
def test_correction_of_a_large_lattice_in_time(precision):
    import torch

    from lbm_solver_3d_b200.solver import Solver
    p = Params().update(nx=256, ny=128, nz=128, walls_y=0, planar=0, radius=8.0, precision=precision, **DECK)
    s = Solver(p)
    nbytes = 19 * p.ncells * {"fp64": 8, "fp32": 4, "fp16": 2}[precision]
    a = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    b = torch.empty_like(a)
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    copies = []
    for _ in range(8):
        e[0].record()
        b.copy_(a)
        e[1].record()
        torch.cuda.synchronize()
        copies.append(e[0].elapsed_time(e[1]) * 1e-3)
    copy = 1.5 * np.median(copies)   # read + read + write against a copy's read + write
    for steps in (4, 1):             # even and odd parity
        s.run(steps)
        times = []
        for _ in range(12):
            t = time.perf_counter()
            s.correct_mass()
            times.append(time.perf_counter() - t)
        assert np.median(times[2:]) <= 5.0 * copy + 60e-6
    s.close()
