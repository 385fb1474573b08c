"""The xy statistics of a field with a non-finite coefficient in one component:
it reaches the entries formed from that component and those that share an x
transform with them (fields go in pairs), in its own xz-plane, and no others.
With u spoilt at one mode, w, w^2, omega_x and omega_x^2 are those of the field
without it, on the two-pass transforms as on the general ones."""
import numpy as np
import pytest

from simson_b200.fields import channel_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("grid", [(32, 17, 32), (20, 17, 18)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_non_finite_component_stays_in_its_entries(grid, precision, bad):
    from simson_b200.bla import FP64, MIXED, Channel
    nx, ny, nz = grid
    xl, zl = 4 * np.pi, 2 * np.pi
    ch = Channel(nx, ny, nz, 4200.0, xl, zl, 0.01, precision=FP64 if precision == "fp64" else MIXED)
    try:
        ch.set_velocity(*channel_field(nx, ny, nz, xl, zl, 0.05, 5))
        ch.start()
        ch.xys_sample()
        want = ch.xys()[0]
        slots = ch.state(5)
        slots[0] = np.array(slots[0])
        slots[0][3, 7, 2] = bad
        ch.set_state(slots)
        ch.xys_reset()
        ch.xys_sample()
        got = ch.xys()[0]
    finally:
        ch.close()
    for entry in (2, 5, 6, 9):  # w, w^2, omega_x, omega_x^2
        np.testing.assert_array_equal(got[entry], want[entry])
    assert not np.isfinite(got[0]).all()  # u itself
