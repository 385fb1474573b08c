"""The two-pass FP64 transforms (fft2.cuh) against numpy: step 2 (H after
sgpu_nonlin) and the Chebyshev transform (H after the forward, omega after the
inverse one in prhs) at lengths of every kind of split -- equal and unequal
factors either way, odd lengths, a single butterfly, the smallest and largest
-- with kx columns that do not fill the last tile, an odd number of z rows, and
at lengths without a two-pass kernel (the runtime plan).

Tolerance: a length-N transform in FP64 has a relative error of a few eps
log2(N) (eps = 1.1e-16); H takes three transforms and a product of two:
4 log2(N) sqrt(3) eps < 1e-14 of the norm, 1e-13 stated (as the step-2 gate)."""
import numpy as np
import pytest

from simson_b200.fields import wavenumbers

pytestmark = pytest.mark.gpu


def field(nx, ny, nz, seed):
    """Seeded coefficients on every stored mode, real in physical space, no
    oddball mode; slots u, v, w, omega_x, omega_z (not related by the curl:
    step 2 does not need that)."""
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((5, nz, ny, nx // 2)) + 1j * rng.standard_normal((5, nz, ny, nx // 2))
    back = (-np.arange(nz)) % nz
    a[..., 0] = 0.5 * (a[..., 0] + a[:, back][..., 0].conj())
    a[:, nz // 2] = 0
    return a


def step2(a, nx, nz, xl, zl):
    al, be = wavenumbers(nx, nz, xl, zl)
    u, v, w, ox, oz = a
    oy = 1j * be[:, None, None] * u - 1j * al * w
    nxp, nzp, h = 3 * nx // 2, 3 * nz // 2, nz // 2

    def phys(f):
        g = np.zeros((nzp, f.shape[1], nxp // 2 + 1), complex)
        g[:h, :, :nx // 2] = f[:h]
        g[nzp - h + 1:, :, :nx // 2] = f[h + 1:]
        return np.fft.irfft(np.fft.ifft(g, axis=0), n=nxp, axis=2) * nxp * nzp

    def spec(p):
        g = np.fft.fft(np.fft.rfft(p, axis=2)[:, :, :nx // 2], axis=0)
        return np.concatenate([g[:h], g[nzp - h:]])

    u, v, w, ox, oy, oz = (phys(q) for q in (u, v, w, ox, oy, oz))
    return [spec(v * oz - w * oy), spec(w * ox - u * oz), spec(u * oy - v * ox)]


@pytest.mark.parametrize("nx,nz", [(16, 16), (24, 18), (32, 24), (40, 30), (48, 36), (60, 54), (64, 72), (80, 90),
                                   (96, 100), (100, 128), (120, 150), (128, 162), (144, 160), (160, 192), (180, 200),
                                   (192, 216), (200, 240), (216, 256), (240, 270), (256, 288), (288, 300), (300, 320),
                                   (320, 384), (384, 20)])
def test_step2(nx, nz):
    from simson_b200.bla import Channel
    ny, xl, zl = 9, 4 * np.pi, 2 * np.pi
    a = field(nx, ny, nz, nx + nz)
    ref = step2(a, nx, nz, xl, zl)
    ch = Channel(nx, ny, nz, 1000.0, xl, zl, 1e-9)
    try:
        ch.set_state(list(a) + [np.zeros_like(a[0])] * 2)
        ch.nonlinbl()
        got = ch.state(3)
    finally:
        ch.close()
    for g, r in zip(got, ref):
        assert np.linalg.norm(g - r) <= 1e-13 * np.linalg.norm(r)


@pytest.mark.parametrize("ny", [9, 17, 19, 25, 33, 41, 49, 51, 55, 61, 65, 73, 81, 91, 97, 101, 109, 121, 129, 145, 151,
                                161, 163, 181, 193, 201, 217, 241, 251, 257])
def test_chebyshev(ny):
    """omega_x = D w - i beta v and omega_z = i alpha v - D u of prhs: a forward
    and an inverse transform around a derivative.  u, v, w are polynomials of
    degree 8, known from nine points, so the reference is exact to a few eps.
    Each coefficient of the forward transform is off by up to eps log2(2 ny)
    of the field, and a derivative coefficient sums up to ny / 2 of them times
    2 k: eps log2(2 ny) ny^2 / 2 of the field's norm, times two for the sum of
    real and imaginary parts' worst cases."""
    from simson_b200.bla import Channel
    from simson_b200.fields import channel_field
    nx, nz, xl, zl = 20, 10, 4 * np.pi, 2 * np.pi
    u, v, w = channel_field(nx, ny, nz, xl, zl, 0.1, 4)
    al, be = wavenumbers(nx, nz, xl, zl)

    def derivative(f9):
        n, k = 8, np.arange(9)
        cb = np.where((k == 0) | (k == n), 2.0, 1.0)
        c = np.einsum("jk,zkx->jzx", 2 / n * np.cos(np.pi * np.outer(k, k) / n) / np.outer(cb, cb), f9)
        c = np.polynomial.chebyshev.chebder(c, axis=0)
        t = np.cos(np.pi * np.outer(np.arange(ny), np.arange(8)) / (ny - 1))
        return np.einsum("jk,kzx->zjx", t, c)

    u9, _, w9 = channel_field(nx, 9, nz, xl, zl, 0.1, 4)
    ox = derivative(w9) - 1j * be[:, None, None] * v
    oz = 1j * al * v - derivative(u9)
    ch = Channel(nx, ny, nz, 1000.0, xl, zl, 0.01)
    try:
        ch.set_velocity(u, v, w)
        ch.start()
        s = ch.state(5)
    finally:
        ch.close()
    bound = 1.1e-16 * np.log2(2 * ny) * ny * ny
    for g, r, f in ((s[3], ox, w), (s[4], oz, u)):
        err = np.linalg.norm(g - r)
        print(ny, "%.1e of the field, bound %.1e" % (err / np.linalg.norm(f), bound))
        assert err <= bound * np.linalg.norm(f) + 1e-14 * np.linalg.norm(r)
