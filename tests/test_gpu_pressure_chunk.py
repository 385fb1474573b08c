"""The pressure at the first and last ny of each number of rows per chunk of
its pencil kernel (4 up to 112, 6 up to 168, 8 up to 224, 10 up to 280) and
beyond all of them, against the plain 64-bit torch reference of perf/cases.py
with that file's tolerances.  Under FP32 storage the rounding of v enters
through D^2 v at the walls, whose rows grow as ((ny - 1)^4 - 1) / 15: beyond
the file's largest ny the tolerance grows as that.

The statistics' pressure entries have no such reference: there the two-pass
kernels are compared with the general ones on one field, zero-padded in kz to
a length of each.  Its |kz| <= 3, so the pressure's is at most 6 and every
z mean (fourth moments: 24 < nz) is exact on both; only roundoff differs,
amplified 1e3 by the pressure solve's differences: 1e-10 of an entry group's
largest value in FP64, 1e-5 with FP32 storage as for the other entries."""
import importlib.util
import math
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "perf", "cases.py")


@pytest.fixture(scope="module")
def cases():
    spec = importlib.util.spec_from_file_location("perf_cases", CASES)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def check(cases, grid, precision):
    import torch
    nx, ny, nz = grid
    case = dict(kind="pressure", model="none", nx=nx, ny=ny, nz=nz, precision=precision, steps=1, re=4200.0,
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
    if precision == "mixed":  # that tolerance is for ny up to 193
        tol *= max(1.0, ((ny - 1) / 192) ** 4)
    errs = []
    for g, w in zip(got, want):
        scale = float(w.norm())
        errs.append(float((g - w).norm()) / scale if scale else float(g.abs().max()))
    print(grid, precision, "%.1e of %.1e" % (max(errs), tol))
    assert max(errs) <= tol, errs


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grid", [(20, 17, 10), (16, 109, 12), (12, 121, 18), (16, 161, 16), (20, 181, 10),
                                  (16, 217, 16), (12, 241, 10), (16, 271, 16), (16, 289, 16)])
def test_pressure(cases, grid, precision):
    check(cases, grid, precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pressure_statistics_two_pass_against_general(precision):
    from simson_b200.bla import Channel
    from simson_b200.fields import channel_field
    nx, ny, xl, zl = 32, 33, 4 * np.pi, 2 * np.pi
    vel = channel_field(nx, ny, 8, xl, zl, 0.05, 5)
    out = []
    for nz in (48, 50):
        wide = []
        for f in vel:
            q = np.zeros((nz,) + f.shape[1:], f.dtype)
            q[:4], q[-3:] = f[:4], f[-3:]
            wide.append(q)
        ch = Channel(nx, ny, nz, 4200.0, xl, zl, 0.01, precision=precision)
        try:
            ch.set_velocity(*wide)
            ch.prhs()
            for dtn in (0.01, 0.007):
                ch.pressure()
                ch.xys_sample(dtn)
            out.append(ch.xys())
        finally:
            ch.close()
    (a, wa), (b, wb) = out
    assert wa == wb
    cuts = (0, 3, 6, 9, 12, 15, 24, 27, 30, 33, 36, 42, 44, 45, 51, 62, 72, 73, 74, 77, 78, 79, 96)
    worst = 0.0
    for lo, hi in zip(cuts, cuts[1:]):
        if lo == 42:  # extremes over z: other sample points
            continue
        scale = np.abs(b[lo:hi]).max()
        if lo in (30, 72, 73, 77, 78):
            assert scale > 0.0, lo
        err = np.abs(a[lo:hi] - b[lo:hi]).max()
        worst = max(worst, err / scale if scale else err)
    print("worst entry group %.1e" % worst)
    assert worst <= (1e-10 if precision == "fp64" else 1e-5)
