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


def test_contexts_in_several_threads():
    """Contexts made, stepped (with captured steps), sampled and closed by
    several host threads at once give what they give one after another."""
    import threading
    from simson_b200.bla import FP64, MIXED, Channel
    runs = [((16, 161, 16), FP64, dict(iles=1)), ((16, 33, 16), FP64, dict(iles=1)), ((16, 193, 16), MIXED, None),
            ((144, 17, 16), FP64, dict(iles=2)), ((200, 17, 50), MIXED, None), ((48, 65, 48), FP64, None)]
    xl, zl = 4 * np.pi, 2 * np.pi
    fields = [channel_field(*grid, xl, zl, 0.05, 5) for grid, _, _ in runs]

    def work(i, out):
        grid, precision, les = runs[i]
        for _ in range(3):
            ch = Channel(*grid, 4200.0, xl, zl, 0.002, precision=precision)
            try:
                if les:
                    ch.set_les(**les)
                ch.set_velocity(*fields[i])
                ch.start()
                ch.step(3)
                ch.xys_sample()
                out[i].append(ch.state(7) + [ch.xys()[0], ch.pressure()])
            finally:
                ch.close()

    alone = [[] for _ in runs]
    for i in range(len(runs)):
        work(i, alone)
    at_once = [[] for _ in runs]
    threads = [threading.Thread(target=work, args=(i, at_once)) for i in range(len(runs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, at_once):
        assert len(b) == 3
        for r in b:
            for p, q in zip(a[0], r):
                np.testing.assert_array_equal(p, q)
