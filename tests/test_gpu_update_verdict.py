"""A call of advance_squirmer that finds the body invalid reports it, whole.

The update's warps decide by the status word whether to go on, and two of them
may set it in the same call. All must take one verdict: the error is returned
every time, and the state that was stored is the body's after this step in all
its words (each thread stores one).
"""
import numpy as np
import pytest

from lbm_solver_3d_b200.params import Params

pytestmark = pytest.mark.gpu


def test_invalid_advance_is_reported_and_stored_whole():
    from lbm_solver_3d_b200._lib import LBMGPU_ERR_DEVICE, LbmgpuError
    from lbm_solver_3d_b200.solver import Solver
    s = Solver(Params().update(nx=26, ny=22, nz=20, tau=1.0, walls_y=1, squirmer=1, radius=4.3, b1=0.02, beta=-2.0, angle=25.0))
    s.run(7)
    s.step()
    q = s.squirmer()
    U = np.array([1.25, 0.0, 0.0])
    s.set_squirmer(q["X"], q["e"], U, q["W"])
    before, kept = s.squirmer(), s.checkpoint()
    for _ in range(40):
        s.restore(kept)
        with pytest.raises(LbmgpuError, match="one lattice cell") as ei:
            s.advance_squirmer()
        assert ei.value.code == LBMGPU_ERR_DEVICE
        after = s.squirmer()
        # Squirmer::integrate in the reference's order
        want = before["U"] + (before["Fh"] + before["Fc"] + after["Fw"]) / before["M"]
        want[2] = 0.0
        assert np.array_equal(after["U"], want)
        assert np.array_equal(after["X"], before["X"] + want)
        W = before["W"] + (before["Th"] + before["Tc"]) / before["I"]
        W[:2] = 0.0
        assert np.array_equal(after["W"], W)
        assert not after["Fc"].any() and not after["Tc"].any()
        assert np.array_equal(after["Fh"], before["Fh"])
    s.close()
