"""The chunked pencil kernel (pencil_chunk.cuh) against the thread-per-pencil
kernel at the sizes where it can go wrong: the first and last ny of each
number of rows per chunk (4 up to ny = 112, 6 up to 168, 8 up to 224, 10
beyond), a last chunk of one row, empty chunks behind it, pencil tiles that
straddle kz planes and end beyond the last pencil, and the kx = kz = 0 pencil
with and without the constant flux.

Both solve the same tau systems in another order of summation; the
stiff solves amplify round-off (eps) by the condition of the tau rows, seen as
1e-12 to 1e-11 between the reference's own builds with and without fused
multiply-adds; 5e-11 per slot, as the other comparison of the two kernels."""
import numpy as np
import pytest

from simson_b200.fields import channel_field

pytestmark = pytest.mark.gpu


def rel(a, b):
    keep = np.ones(a.shape[0], bool)
    keep[a.shape[0] // 2] = False
    return float(np.linalg.norm(a[keep] - b[keep]) / max(np.linalg.norm(b[keep]), 1e-300))


@pytest.mark.parametrize("grid", [(4, 9, 4), (12, 17, 6), (20, 33, 10), (20, 109, 10), (12, 121, 18), (12, 161, 6),
                                  (20, 181, 10), (12, 217, 6), (12, 241, 10), (8, 257, 8), (20, 97, 12)])
@pytest.mark.parametrize("cflux", [True, False])
def test_chunk_kernel_matches_thread_kernel(grid, cflux):
    from simson_b200.bla import FP64, Channel
    nx, ny, nz = grid
    xl, zl = 4 * np.pi, 2 * np.pi
    u, v, w = channel_field(nx, ny, nz, xl, zl, 0.05, 3)
    out = []
    for kernel in (False, "auto"):
        ch = Channel(nx, ny, nz, 2000.0, xl, zl, 0.01, cflux=cflux, px=None if cflux else -1e-3,
                     precision=FP64)
        try:
            ch.set_pencil_kernel(kernel)
            ch.set_velocity(u, v, w)
            ch.start()
            ch.step(1)
            ch.set_dt(0.008)  # another dt: new tau coefficients in two stages
            ch.step(2)
            out.append((ch.state(7), ch.puw(), ch.scalars()))
        finally:
            ch.close()
    (s0, p0, c0), (s1, p1, c1) = out
    errs = [rel(s1[k], s0[k]) for k in range(7)]
    print(grid, ["%.1e" % e for e in errs])
    tol = 5e-11
    assert max(errs) <= tol, errs
    assert np.linalg.norm(p1 - p0) <= tol * np.linalg.norm(p0)
    # px moves by ~1e-9 for a 1e-14 change of the flux (the parity tests' 1e-7)
    assert abs(c1["px"] - c0["px"]) <= 1e-7 * abs(c0["px"])
