"""FP64 lane: what is not finite comes out where the oracle has it, and every other cell
with the oracle's bits."""
import copy

import numpy as np
import pytest

from conformal_cubed_sphere_gb300 import _lib as L
from conformal_cubed_sphere_gb300 import model as M
from oracle import oracle as O
from tests.helpers import CHECK_FIELDS, seeded_case

pytestmark = pytest.mark.gpu


def _same(a, b, m, what):
    a, b = a[m], b[m]
    nan = np.isnan(b)
    assert np.array_equal(np.isnan(a), nan), (what, int(np.isnan(a).sum()), int(nan.sum()))
    assert np.array_equal(a[~nan].view(np.int64), b[~nan].view(np.int64)), what
    return int((~np.isfinite(b)).sum())


# one cell's wave-speed metric negative (its square root is NaN), NaN, infinite, and so
# large that its product with the depth overflows: the reference's never-written E slots
# (CCS_EDISS_ZERO) then contribute inf * 0
@pytest.mark.parametrize("value", [-1.0, np.nan, np.inf, 1.0e306])
@pytest.mark.parametrize("ediss", [L.CCS_EDISS_ZERO, L.CCS_EDISS_RECONSTRUCT])
@pytest.mark.parametrize("entry", [0, 3])
def test_wave_speed_that_is_not_finite(value, ediss, entry):
    mesh, s, dt = seeded_case(20, 3, seed=6, oro=True)
    mesh = copy.copy(mesh)
    mesh.matrixIG = mesh.matrixIG.copy()
    nh = 26
    c = (2 * nh + 12) * nh + 9  # panel 3, an interior cell
    mesh.matrixIG.reshape(-1, 4)[c, entry] = value
    g = M.Stepper(mesh, dt, precision="fp64", e_dissipation=ediss)
    g.set_state(s)
    o = O.Oracle.from_mesh(mesh, e_dissipation=ediss)
    o.set_state(s.arrays)
    im = mesh.interior_mask()
    bad = [_same(a, b, im, q) for q, (a, b) in enumerate(zip(g.spatial_operator(), o.spatial_operator()))]
    assert bad[0] > 0 and max(bad[1:]) > 0  # (phiG, and the wind across the face)


@pytest.mark.parametrize("seed", range(4))
def test_doubled_tendencies_that_overflow(seed):
    """RK4 adds 2 k2 to k1: where k2 is beyond 2^1023 the reference's product is infinite,
    whatever k1 is.  A state of huge phiG over a huge sqrtG (so that the depth stays small
    and the wind moderate) has such cells with k1 of the other sign."""
    mesh, s, dt = seeded_case(16, 3, seed=3 + seed, oro=False)
    mesh = copy.copy(mesh)
    mesh.sqrtG, mesh.f, dt = mesh.sqrtG * 2.0 ** 975, mesh.f * 0, 1.0
    for k in ("u", "v", "uC", "vC"):
        s[k] *= 1e5
    rng = np.random.default_rng(seed)
    s["phi"][:] = 1.0
    s["phiG"][:] = 2.0 ** 1021 * rng.uniform(-1, 1, size=mesh.ncell)
    o = O.Oracle.from_mesh(mesh, operator=L.CCS_OP_CENTRAL2)
    o.set_state(s.arrays)
    o.rk4_once(dt)
    im, m = mesh.interior_mask(), ~mesh.corner_mask()
    k1, k2 = (o.get_tend(q)[0][im] for q in (-1, -2))
    with np.errstate(all="ignore"):
        cells = np.isinf(k1 + 2 * k2) & (np.abs(k1 / 4 + k2 / 2) < 2.0 ** 1021.9)
    assert cells.sum() > 0
    g = M.Stepper(mesh, dt, precision="fp64", operator=L.CCS_OP_CENTRAL2)
    g.set_state(s)
    g.step(1)
    a, b = g.get_state(), o.get_state(1)
    for k in ("phiG", "u", "v"):
        _same(a[k], b[k], m, k)


@pytest.mark.parametrize("seed", range(24))
def test_damaged_states(seed):
    """Cells set to zeros, infinities, NaNs, subnormals and magnitudes whose smoothness
    indicators or products overflow: NaNs and infinities come out where the oracle has them
    (a comparison of the WENO switches with a NaN is false)."""
    rng = np.random.default_rng(seed)
    N, halo = int(rng.choice([8, 20, 33])), int(rng.choice([3, 4]))
    mesh = M.Mesh(N, halo, pole_inverse=N % 2 == 1)
    s = M.initial_state(mesh, kind=L.CCS_IC_SEEDED, seed=seed, lmax_oro=8)
    dt = M.cfl_dt(mesh, s, 0.4)
    values = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -1e-310, 1e60, -1e100, 1e154, -1e157, 1e200, 1e300]
    for k in rng.choice(["phiG", "u", "v", "phi", "uC", "vC"], 1 + seed % 3, replace=False):
        cells = np.flatnonzero(rng.random(mesh.ncell) < rng.choice([0.003, 0.1]))
        s[k][cells] = rng.choice(values, size=cells.size) if seed % 2 else rng.choice(values)
    ediss, scheme = int(rng.integers(0, 2)), str(rng.choice(["RK4", "RK3_TVD"]))
    g = M.Stepper(mesh, dt, precision="fp64", scheme=scheme, e_dissipation=ediss)
    g.set_variant(seed % 3)
    g.set_state(s)
    o = O.Oracle.from_mesh(mesh, e_dissipation=ediss)
    o.set_state(s.arrays)
    im, m = mesh.interior_mask(), ~mesh.corner_mask()
    for q, (a, b) in enumerate(zip(g.spatial_operator(), o.spatial_operator())):
        _same(a, b, im, q)
    g.step(1)
    o.run(dt, 1, scheme)
    a, b = g.get_state(), o.get_state()
    for k in CHECK_FIELDS:
        _same(a[k], b[k], m, k)
