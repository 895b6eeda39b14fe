"""Two lattices stepped at the same time from two threads.

Their kernels share the chip, so a persistent staged-row bulk finds only part of
it free. Results must not depend on it, and the two together should take about
twice as long as one alone: the bulk leaves some SMs to its second stream, and
the CTAs that leave them must not take the rest of the grid along. Measured: 1.9
times; 4 to 19 times when they did. Three times, in the median of five calls, is
taken as the line.
"""
import threading
import time

import numpy as np
import pytest

from lbm_solver_3d_b200.params import Params

pytestmark = pytest.mark.gpu

CASES = {
    "fp32 slit": dict(nx=192, ny=96, nz=96, walls_y=1, planar=1, precision="fp32"),
    "fp16 box": dict(nx=256, ny=128, nz=128, walls_y=0, planar=0, precision="fp16"),
}
DECK = dict(squirmer=1, radius=8.0, b1=1.5e-3, beta=1.0, tau=0.9, traj_every=50)


@pytest.mark.parametrize("case", sorted(CASES))
def test_two_at_once(case):
    from lbm_solver_3d_b200.solver import Solver
    p = Params().update(**DECK, **CASES[case])
    calls, steps = 6, 300
    alone, pair = Solver(p), [Solver(p), Solver(p)]
    one = []
    for _ in range(calls):
        t = time.perf_counter()
        alone.run(steps)
        one.append(time.perf_counter() - t)
    two = [[], []]
    start = threading.Barrier(2)

    def go(i):
        for _ in range(calls):
            start.wait()
            t = time.perf_counter()
            pair[i].run(steps)
            two[i].append(time.perf_counter() - t)

    threads = [threading.Thread(target=go, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    ref, rows = alone.fields(), alone.traj_rows()
    for s in pair:
        for x, y in zip(s.fields(), ref):
            assert np.array_equal(x, y)
        assert np.array_equal(s.traj_rows(), rows)
    assert np.median([max(a, b) for a, b in zip(*(t[1:] for t in two))]) <= 3.0 * np.median(one[1:])
    for s in (alone, *pair):
        s.close()
