"""Calls that make device buffers of their own, on a GPU without room for them:
the call reports it or does without, and the context works on as it was."""
import ctypes

import numpy as np
import pytest

from simson_b200.fields import channel_field

pytestmark = pytest.mark.gpu


class Full:
    """Every free byte of the device but (about) leave, down to pieces of 1 kB."""

    def __init__(self, leave=0):
        import torch
        self.rt = ctypes.CDLL("libcudart.so.%s" % torch.version.cuda.split(".")[0])
        self.held = []
        size = torch.cuda.mem_get_info()[0] - leave
        while size >= 1024:
            p = ctypes.c_void_p()
            if self.rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
                self.held.append(p)
                if leave:
                    break
            else:
                self.rt.cudaGetLastError()
                size //= 2

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        for p in self.held:
            self.rt.cudaFree(p)


def channel(grid, precision="fp64"):
    from simson_b200.bla import FP64, MIXED, Channel
    nx, ny, nz = grid
    xl, zl = 4 * np.pi, 2 * np.pi
    ch = Channel(nx, ny, nz, 4200.0, xl, zl, 0.002, precision=FP64 if precision == "fp64" else MIXED)
    ch.set_velocity(*channel_field(nx, ny, nz, xl, zl, 0.05, 5))
    return ch


@pytest.mark.parametrize("leave", [0, 100 << 20])
def test_pencil_kernel_without_room_stays(leave):
    """The thread kernel's 15 columns (238 MB on this grid) do not fit: with 0
    bytes left none of them, with 100 MB the first and not the last."""
    from simson_b200.bla import SimsonError
    grid = (192, 129, 160)
    ch = channel(grid)
    try:
        ch.start()
        ch.step(1)
        ch.step(2)
        want = ch.state(7)
    finally:
        ch.close()
    ch = channel(grid)
    try:
        ch.start()
        ch.step(1)
        with Full(leave):
            with pytest.raises(SimsonError):
                ch.set_pencil_kernel(False)
        ch.step(2)
        for a, b in zip(want, ch.state(7)):
            np.testing.assert_array_equal(a, b)
        ch.set_pencil_kernel(False)  # there is room again
        ch.step(1)
        assert np.isfinite(ch.scalars()["px"])
    finally:
        ch.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_filter_without_room_for_its_matrix(precision):
    """The tensorial filter without room for its matrix (685 kB here) solves
    column by column; the two agree to the round-off of n = 289 rows."""
    grid = (16, 289, 16)
    gu = []
    for full in (False, True):
        ch = channel(grid, precision)
        try:
            ch.set_les(iles=1, ihighorder=1)  # makes the model's other buffers
            if full:
                with Full():
                    ch.set_les(iles=1, ihighorder=2)
            else:
                ch.set_les(iles=1, ihighorder=2)
            ch.start()
            ch.step(1)
            gu.append(np.stack(ch.les_gu()))
        finally:
            ch.close()
    err = np.linalg.norm(gu[1] - gu[0]) / np.linalg.norm(gu[0])
    print(precision, "%.1e" % err)
    # six solves of diagonally dominant rows: some tens of eps, under FP32
    # storage the same of the state both filter
    assert err <= (1e-12 if precision == "fp64" else 1e-6)
    assert err > 0.0  # the column solves ran
