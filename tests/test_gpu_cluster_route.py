"""Which lattices take the cluster's many steps per launch, and long calls.

The kernel launches of a call tell the two ways apart: one for all but the last
step and up to four for that step, or at least one per step. A call of more
steps than one launch takes (131,072) is several launches; the second starts
where the first ended, on an odd step too, and gives the separate kernels'
populations bit for bit.
"""
import numpy as np
import pytest

from test_gpu_cluster import SIZES, make

pytestmark = pytest.mark.gpu

REFUSED = [(8, 27, 38, 1, 0), (16, 32, 32, 1, 1)]   # more than 512 nodes per CTA


def launches(s, steps):
    before = s.launch_count()
    s.run(steps)
    return s.launch_count() - before


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("size", SIZES + REFUSED[1:])
def test_route_by_launches(size, precision):
    s, plain = make(size, precision, None), make(size, precision, "node")
    if size in REFUSED:
        assert launches(s, 35) >= 35
    else:
        assert launches(s, 35) <= 5
        assert launches(s, 2) >= 2   # too short a call for it
    assert launches(plain, 35) >= 35
    s.close(), plain.close()


@pytest.mark.parametrize("first", [0, 1])
def test_call_of_several_launches(first):
    size, steps = (3, 5, 4, 1, 1), (1 << 17) + 38
    a, b = make(size, "fp64", None), make(size, "fp64", "node")
    if first:
        a.run(first)
        b.run(first)
    assert launches(a, steps) <= 6
    b.run(steps)
    assert np.array_equal(a.get_f(), b.get_f())
    for x, y in zip(a.fields(), b.fields()):
        assert np.array_equal(x, y)
    a.close(), b.close()
