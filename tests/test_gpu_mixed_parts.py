"""Mixed lane: small launches run their work items in smaller tiles (two sizes), larger
ones whole.  All give the same bits: a grid alone runs in parts, the same grid as member
of a batch with many items whole, with every tile variant."""
import numpy as np
import pytest

from conformal_cubed_sphere_gb300 import _lib as L
from conformal_cubed_sphere_gb300 import model as M
from tests.helpers import CHECK_FIELDS, bitwise_equal, seeded_case, valid_mask

pytestmark = pytest.mark.gpu

OPTIONS = [("RK4", L.CCS_EDISS_ZERO, L.CCS_OP_WENO), ("RK3_TVD", L.CCS_EDISS_RECONSTRUCT, L.CCS_OP_WENO),
           ("RK4", L.CCS_EDISS_ZERO, L.CCS_OP_CENTRAL4)]


def _member(mesh, s, dt, opt, var):
    g = M.Stepper(mesh, dt, precision="mixed", scheme=opt[0], e_dissipation=opt[1], operator=opt[2],
                  phi_mean=8000.0 * mesh.gravity)
    g.set_variant(var)
    g.set_state(s)
    return g


def _same(a, b, mesh, what):
    m = valid_mask(mesh)
    for k in CHECK_FIELDS:
        assert bitwise_equal(a[k], b[k], m), (what, k)


# alone: 16 x 8 tiles; two members of N = 100: 16 x 16 tiles; 40 members: whole items
@pytest.mark.parametrize("var", [0, 1, 2, 3])
@pytest.mark.parametrize("opt", OPTIONS, ids=["rk4", "rk3_ediss", "central"])
def test_parts_and_whole_items_agree_bitwise(var, opt):
    for N, halo, n in ((100, 3, 2), (40, 5, 40), (4, 3, 600)):
        mesh, s, dt = seeded_case(N, halo, seed=N)
        alone = _member(mesh, s, dt, opt, 0)
        alone.step(2)
        ref = alone.get_state()
        owner = _member(mesh, s, dt, opt, var)
        members = [owner]
        for _ in range(n - 1):
            g = M.Stepper(mesh, dt, precision="mixed", scheme=opt[0], e_dissipation=opt[1], operator=opt[2],
                          phi_mean=8000.0 * mesh.gravity, share_with=owner)
            members.append(g)
        members[-1].set_variant(var)
        for g in members[1:]:
            g.set_state(s)
        b = M.Batch(members)
        b.step(2)
        for k in sorted({0, n // 2, n - 1}):
            _same(members[k].get_state(), ref, mesh, (N, n, k))


# both sides of the two lines for a grid alone (C99 / C113 and C176 / C200, odd sizes
# with partial tiles), against the same grid twice in a batch
@pytest.mark.parametrize("N", [12, 99, 113, 176, 200])
def test_grid_sizes_around_the_lines(N):
    mesh = M.Mesh(N, 3, pole_inverse=N % 2 == 1)
    s = M.initial_state(mesh, kind=L.CCS_IC_SEEDED, seed=N, lmax_oro=8)
    dt = M.cfl_dt(mesh, s, 0.5)
    alone = _member(mesh, s, dt, OPTIONS[0], 0)
    tend = alone.spatial_operator()
    alone.step(2)
    n = 5  # (five members: whole items from N = 99 on)
    members = [_member(mesh, s, dt, OPTIONS[0], 1) for _ in range(n)]
    M.Batch(members).step(2)
    _same(members[n - 1].get_state(), alone.get_state(), mesh, N)
    fp = M.Stepper(mesh, dt, precision="fp64")
    fp.set_state(s)
    im = mesh.interior_mask()
    for a, b in zip(tend, fp.spatial_operator()):  # FP32 stencils against FP64
        assert np.linalg.norm(a[im] - b[im]) < 2e-4 * np.linalg.norm(b[im])
