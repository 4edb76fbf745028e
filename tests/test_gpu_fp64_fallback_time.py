"""FP64 lane: tiles outside the integer arithmetic's window cost what their FP64
instructions cost, once."""
import pytest

from conformal_cubed_sphere_gb300 import model as M
from tests.helpers import seeded_case

pytestmark = pytest.mark.gpu


def _stage_ms(mesh, s, dt):
    g = M.Stepper(mesh, dt, precision="fp64")
    g.set_variant(1)
    g.set_state(s)
    best = float("inf")
    for _ in range(5):
        g.timing(1, 1)
        g.step(1)
        ms, n = g.timing(0, 0)
        best = min(best, ms / n)
    assert g.check_state() == 0
    return best


def test_time_of_tiles_outside_the_window():
    """An out-of-window stage issues about 1 880 FP64 instructions a cell against 510 of an
    ordinary one on the pipe both are bound by: 3.7 times as long.  With the two sides of a
    face in separate passes of a warp it would be 7; the limit lies half-way."""
    mesh, s, dt = seeded_case(192, 3, seed=2)
    ordinary = _stage_ms(mesh, s, dt)
    big = s.copy()  # the same flow in units in which the depth is 2^216, in every stage
    for k in ("phi", "phiG"):
        big[k] *= 2.0 ** 200
    for k in ("u", "v", "uC", "vC", "zonal_wind", "meridional_wind"):
        big[k] *= 2.0 ** 100
    outside = _stage_ms(mesh, big, M.cfl_dt(mesh, big, 0.5))
    print(f"stage {ordinary:.4f} ms, outside the window {outside:.4f} ms")
    assert outside < 5.3 * ordinary, (outside, ordinary)
