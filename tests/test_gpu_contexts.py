"""Two contexts of different grids alive in one process: what the smaller one's
set-up sets for the whole process (the kernels' limits of dynamic shared memory)
must not refuse the larger one's launches.  The larger context is set up first,
the smaller second, and the larger one then gives what it gives alone, to the
last bit.  Every larger grid here needs more than the 48 KB a launch may take
without a raised limit."""
import numpy as np
import pytest

from simson_b200.fields import channel_field

pytestmark = pytest.mark.gpu

SMALL = (16, 17, 16)


def channel(grid, precision, les):
    from simson_b200.bla import FP64, MIXED, Channel
    nx, ny, nz = grid
    xl, zl = 4 * np.pi, 2 * np.pi
    u, v, w = channel_field(nx, ny, nz, xl, zl, 0.05, 5)
    ch = Channel(nx, ny, nz, 4200.0, xl, zl, 0.002, precision=FP64 if precision == "fp64" else MIXED)
    if les:
        ch.set_les(**les)
    ch.set_velocity(u, v, w)
    return ch


def run(ch, what):
    ch.start()
    if what == "xys":
        ch.xys_sample()
        return [ch.xys()[0]]
    if what == "box":
        return list(ch.box_filter_sample(2))
    ch.step(1)
    return list(ch.state(7))


@pytest.mark.parametrize("grid,precision,what,les", [
    ((16, 161, 16), "fp64", "step", dict(iles=1)),        # wall-normal filter product
    ((16, 161, 16), "mixed", "step", dict(iles=1)),
    ((16, 193, 16), "mixed", "step", None),               # the mixed start's Chebyshev transform
    ((16, 271, 16), "fp64", "step", None),                # a Chebyshev length without a two-pass kernel
    ((144, 17, 16), "fp64", "step", dict(iles=2)),        # stress transforms of the general lengths, x
    ((16, 17, 400), "mixed", "step", dict(iles=2)),       # and z
    ((200, 17, 50), "fp64", "xys", None),                 # statistics of the general lengths
    ((200, 17, 16), "mixed", "box", None),                # filtered samples
])
def test_smaller_context_leaves_the_larger_one(grid, precision, what, les):
    ch = channel(grid, precision, les)
    try:
        alone = run(ch, what)
    finally:
        ch.close()
    ch = channel(grid, precision, les)
    try:
        other = channel(SMALL, precision, les)
        try:
            run(other, what)
            got = run(ch, what)
        finally:
            other.close()
    finally:
        ch.close()
    for a, b in zip(alone, got):
        np.testing.assert_array_equal(a, b)
