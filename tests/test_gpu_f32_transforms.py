"""One mixed-precision step with every FP32 transform length that has a
compile-time plan (SB_FIXED_LENGTHS, step2_launch.cuh), in z and, where nx
allows it, in x, beside lengths of the runtime plan, against the plain 64-bit
torch reference of perf/cases.py with that file's tolerance (four times the
distance seen, that of FP32 storage under the wall-normal derivatives)."""
import importlib.util
import math
import os

import pytest

pytestmark = pytest.mark.gpu

CASES = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "perf", "cases.py")
LENGTHS = (24, 36, 48, 54, 60, 72, 75, 81, 90, 96, 108, 120, 135, 144, 150, 162, 180, 192, 216, 225, 240, 270, 288, 300,
           324, 360, 375, 384, 405, 432, 450, 480, 486, 540, 576)
GRIDS = ([(16, 17, 2 * n // 3) for n in LENGTHS] + [(2 * n // 3, 17, 16) for n in LENGTHS if 2 * n // 3 % 4 == 0]
         + [(12, 17, 20), (20, 17, 400), (400, 17, 12)])


@pytest.fixture(scope="module")
def cases():
    spec = importlib.util.spec_from_file_location("perf_cases", CASES)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("grid", GRIDS)
def test_mixed_step(cases, grid):
    import torch
    nx, ny, nz = grid
    case = dict(kind="dns", model="none", nx=nx, ny=ny, nz=nz, precision="mixed", steps=1, re=4200.0,
                xl=4 * math.pi, zl=2 * math.pi, dt=0.002, rms=0.05)
    s = cases.prepare(case, 3)
    try:
        got = cases.run(s)
        s.ch.sync()
        got = [torch.as_tensor(g).double().cpu() for g in got]
    finally:
        s.ch.close()
    want = [torch.as_tensor(w).double().cpu() for w in cases.exact(case, 3)]
    errs = [float((g - w).norm() / w.norm()) for g, w in zip(got, want)]
    print(grid, "%.1e" % max(errs))
    assert max(errs) <= cases.tolerance(case)["rel"], errs
