"""Rotation and the fringe force in the x passes of step 2 and of the pressure,
on the two-pass transforms and on the general ones, against plain torch at 64
bits: H1 = v (omega_z + 2 rot) - w omega_y - lambda (u - U_b) and its like.

Tolerances: H 1e-13 as without forcing (test_gpu_f64_transforms.py; 1e-5 with
FP32 storage, the mixed path's gate), the pressure that of perf/cases.py."""
import importlib.util
import math
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "perf", "cases.py")
ROT = 0.3
FRINGE = dict(fstart=-3.0, fend=0.0, frise=1.5, ffall=0.8, fmax=1.0)


@pytest.fixture(scope="module")
def cases():
    spec = importlib.util.spec_from_file_location("perf_cases", CASES)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def make(cases, grid, precision, rot, fringe):
    """A context and the 64-bit restatement of the same run."""
    import torch
    from simson_b200.bla import Channel, fringe_function
    nx, ny, nz = grid
    xl, zl = 4 * math.pi, 2 * math.pi
    case = dict(kind="pressure", model="none", nx=nx, ny=ny, nz=nz, precision=precision, steps=1, re=4200.0, xl=xl,
                zl=zl, dt=0.004, rms=0.05)
    nxp = 3 * nx // 2
    ch = Channel(nx, ny, nz, 4200.0, xl, zl, 0.004, rot=rot, precision=precision)
    rng = np.random.default_rng(5)
    lam, base = np.zeros(nxp), np.zeros((3, ny, nxp))
    if fringe:
        bu = rng.standard_normal((2, 3, ny, nxp // 2 + 1))
        ch.set_base_flow(bu[0], bu[1])
        ch.set_fringe(**FRINGE)
        lam = fringe_function(nxp, xl, **FRINGE)
        base[..., 0::2], base[..., 1::2] = bu[0, ..., :-1], bu[1, ..., :-1]

    class Forced(cases._Exact):
        def products(self, st):
            u, v, w, ox, oz = st
            oy = 1j * self.be[:, None] * u - 1j * self.al * w
            n = 3 * nx // 2, 3 * nz // 2
            u, v, w, ox, oy, oz = (self.phys(q, *n) for q in (u, v, w, ox, oy, oz))
            oz = oz + 2 * rot
            la = self._mat(lam)
            f = [la * (q - self._mat(b)[:, None, :]) for q, b in zip((u, v, w), base)]
            return (self.spec(v * oz - w * oy - f[0]), self.spec(w * ox - u * oz - f[1]),
                    self.spec(u * oy - v * ox - f[2]), self.spec((u * u + v * v + w * w) / 2))

    vel = cases._velocity(case, 3)
    ch.set_velocity(*(q.permute(1, 0, 2).cpu().numpy() for q in vel))
    ch.start()
    return ch, Forced(case), torch


GRIDS = [(16, 17, 16), (48, 17, 30), (60, 33, 20), (20, 17, 24), (40, 9, 18), (36, 17, 20)]
FORCING = [(ROT, False), (0.0, True), (ROT, True)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("rot,fringe", FORCING)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_step2(cases, grid, rot, fringe, precision):
    ch, x, torch = make(cases, grid, precision, rot, fringe)
    try:
        st = [torch.tensor(f.transpose(1, 0, 2)).to(x.dev) for f in ch.state(5)]
        ch.nonlinbl()
        got = ch.state(3)
    finally:
        ch.close()
    nx, ny, nz = grid
    scale = 1.5 * nx * 1.5 * nz
    keep = np.arange(nz) != nz // 2
    for g, w in zip(got, x.products(st)):
        w = w.cpu().numpy().transpose(1, 0, 2) * scale
        err = np.linalg.norm(g[keep] - w[keep]) / np.linalg.norm(w[keep])
        assert err <= (1e-13 if precision == "fp64" else 1e-5), err


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("rot,fringe", FORCING)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pressure(cases, grid, rot, fringe, precision):
    ch, x, torch = make(cases, grid, precision, rot, fringe)
    try:
        p = ch.pressure()
    finally:
        ch.close()
    re, im = (q.cpu().numpy() for q in x.pressure(3))
    keep = np.arange(grid[2]) != grid[2] // 2
    want = (re + 1j * im)[keep]
    err = np.linalg.norm(p[keep] - want) / np.linalg.norm(want)
    print(grid, rot, fringe, precision, "%.1e" % err)
    assert err <= cases.tolerance(x.case)["rel"], err
