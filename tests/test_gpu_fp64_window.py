"""FP64 lane: tiles whose field values leave the exponent window of the integer
arithmetic take the FP64 instructions, the others the integer ones; both, and the
mixture, give the oracle's bits."""
import copy

import numpy as np
import pytest

from conformal_cubed_sphere_gb300 import _lib as L
from conformal_cubed_sphere_gb300 import model as M
from oracle import oracle as O
from tests.helpers import CHECK_FIELDS, bitwise_equal, max_rel, seeded_case, valid_mask

pytestmark = pytest.mark.gpu


def _check(mesh, s, dt, ediss, steps):
    g = M.Stepper(mesh, dt, precision="fp64", e_dissipation=ediss)
    g.set_state(s)
    o = O.Oracle.from_mesh(mesh, e_dissipation=ediss)
    o.set_state(s.arrays)
    im, m = mesh.interior_mask(), valid_mask(mesh)
    for a, b in zip(g.spatial_operator(), o.spatial_operator()):
        assert bitwise_equal(a, b, im), max_rel(a, b, im)
    g.step(steps)
    o.run(dt, steps)
    a, b = g.get_state(), o.get_state()
    for k in CHECK_FIELDS:
        assert bitwise_equal(a[k], b[k], m), (k, max_rel(a[k], b[k], m))


# winds scaled by 2^k on half of the sphere: inside the window (fluxes of 2^-60), below it
# (2^-210), far below it, and a flow at rest (fluxes, differences and indicators zero)
@pytest.mark.parametrize("k", [-100, -250, -600, None])
@pytest.mark.parametrize("ediss", [0, 1])
def test_values_in_and_out_of_the_window(k, ediss):
    mesh, s, dt = seeded_case(40, 3, seed=31, oro=True)
    half = np.where(np.abs(mesh.lon) < 10.0, mesh.lon, 0.0) > np.pi
    for f in ("u", "v", "uC", "vC", "zonal_wind", "meridional_wind"):
        s[f][half] *= 0.0 if k is None else 2.0 ** k
    _check(mesh, s, dt, ediss, 2)


def test_constant_state():
    """No wind and a constant depth: every difference is zero."""
    mesh, s, dt = seeded_case(24, 3, seed=3, oro=False)
    for f in ("u", "v", "uC", "vC", "zonal_wind", "meridional_wind"):
        s[f][:] = 0.0
    s["phi"][:] = 8.0e4
    s["phiG"] = s["phi"] * mesh.sqrtG
    _check(mesh, s, dt, L.CCS_EDISS_ZERO, 3)


@pytest.mark.parametrize("k", [-500, -405, -390, 280, 310, 480])
def test_grid_spacings_beyond_the_quotients_range(k):
    """dx and dy scaled by 2^k, dt with small ones: the integer quotients by dx, dy, 60 dx and
    60 dy end at 2^-400 and 2^300."""
    mesh, s, dt = seeded_case(16, 3, seed=7, oro=True)
    mesh = copy.copy(mesh)
    mesh.dx, mesh.dy = mesh.dx * 2.0 ** k, mesh.dy * 2.0 ** k
    _check(mesh, s, dt * 2.0 ** min(k, 0), L.CCS_EDISS_RECONSTRUCT, 1)
