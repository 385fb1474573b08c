"""The LES stress and filter and the xy statistics at the edges of their
kernels' ranges, against the plain 64-bit torch reference of perf/cases.py with
that file's tolerances (four times the distance seen, per kind and precision):

* statistics: the smallest and largest transform lengths of the two-pass
  kernels, ny below the moments' groups, and lengths that only the general
  transforms take, in x, in z and in both;
* Smagorinsky stress: the shortest two-pass lengths, and lengths of the
  general transforms beside two-pass ones;
* ADM-RT: ny at the ends of the filter product's row tiles, the last ny whose
  product fits a CTA's shared memory and the next one, which the column solves
  filter."""
import importlib.util
import math
import os

import pytest

pytestmark = pytest.mark.gpu

CASES = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "perf", "cases.py")


@pytest.fixture(scope="module")
def cases():
    spec = importlib.util.spec_from_file_location("perf_cases", CASES)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def check(cases, kind, model, grid, precision, steps):
    import torch
    nx, ny, nz = grid
    case = dict(kind=kind, model=model, nx=nx, ny=ny, nz=nz, precision=precision, steps=steps, re=4200.0,
                xl=4 * math.pi, zl=2 * math.pi, dt=0.004, rms=0.05)
    s = cases.prepare(case, 3)
    try:
        got = cases.run(s)
        s.ch.sync()
        got = [torch.as_tensor(g).double().cpu() for g in got]
    finally:
        s.ch.close()
    want = [torch.as_tensor(w).double().cpu() for w in cases.exact(case, 3)]
    tol = cases.tolerance(case)["rel"]
    errs = []
    for g, w in zip(got, want):
        scale = float(w.norm())
        errs.append(float((g - w).norm()) / scale if scale else float(g.abs().max()))
    print(kind, model, grid, precision, "%.1e of %.1e" % (max(errs), tol))
    assert max(errs) <= tol, errs


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grid", [(32, 9, 32), (36, 17, 40), (384, 9, 32), (32, 9, 384), (32, 17, 50), (20, 17, 36),
                                  (20, 9, 18), (100, 33, 108)])
def test_statistics(cases, grid, precision):
    check(cases, "xys", "none", grid, precision, 2)


@pytest.mark.parametrize("grid", [(32, 17, 32), (36, 33, 40), (40, 17, 100), (16, 17, 48), (48, 17, 20), (20, 17, 20)])
def test_smagorinsky(cases, grid):
    check(cases, "les", "smagorinsky", grid, "fp64", 2)


@pytest.mark.parametrize("grid", [(20, 17, 12), (16, 33, 16), (16, 65, 16), (32, 81, 16), (16, 97, 20), (16, 129, 16),
                                  (16, 161, 16)])
def test_filter(cases, grid):
    check(cases, "les", "admrt", grid, "fp64", 2)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ny", [161, 451, 481])
def test_filtered_velocity(cases, ny, precision):
    """The filtered velocities themselves, of columns rough enough that the high
    pass keeps them: 1e-12, the gate of the model's other tests, of six solves
    of diagonally dominant rows and a sum of ny products."""
    import numpy as np
    import torch
    from simson_b200.bla import Channel
    nx, nz = 16, 16
    rng = np.random.default_rng(7)
    vel = rng.standard_normal((3, nz, ny, nx // 2)) + 1j * rng.standard_normal((3, nz, ny, nx // 2))
    vel[:, nz // 2] = 0.0
    vel[:, 0, :, 0] = vel[:, 0, :, 0].real
    ch = Channel(nx, ny, nz, 4200.0, 4 * math.pi, 2 * math.pi, 0.004, precision=precision)
    try:
        ch.set_les(iles=1)
        ch.set_velocity(*vel)
        ch.start()
        got = ch.les_gu()
    finally:
        ch.close()
    if precision == "mixed":  # the stored state is what is filtered
        vel = vel.real.astype(np.float32).astype(np.float64) + 1j * vel.imag.astype(np.float32).astype(np.float64)
    filt = cases._Exact(dict(nx=nx, ny=ny, nz=nz, xl=4 * math.pi, zl=2 * math.pi)).high_pass()
    keep = np.arange(nz) != nz // 2
    for g, v in zip(got, vel):
        want = filt(torch.tensor(v.transpose(1, 0, 2)).to(cases._device())).cpu().numpy().transpose(1, 0, 2)
        err = np.linalg.norm(g[keep] - want[keep]) / np.linalg.norm(want[keep])
        print(ny, precision, "%.1e" % err)
        assert err <= 1e-12
