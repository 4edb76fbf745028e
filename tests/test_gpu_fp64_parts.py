"""FP64 lane: small launches run their work items in parts of 8 x 8 or 16 x 8 cells, larger
ones whole; both sides of the lines, with partial tiles and parts beyond the panel's edge,
give the oracle's bits."""
import pytest

from conformal_cubed_sphere_gb300 import _lib as L
from conformal_cubed_sphere_gb300 import model as M
from oracle import oracle as O
from tests.helpers import CHECK_FIELDS, bitwise_equal, max_rel, seeded_case, valid_mask

pytestmark = pytest.mark.gpu


# N = 4: one part of an item holds all cells; 12 and 41: parts beyond the edge; 48: the
# largest grid in quarters; 52 and 95: halves, the last ones partial or beyond the edge;
# 100: whole items, the last ones partial
@pytest.mark.parametrize("N", [4, 12, 41, 48, 52, 95, 100])
@pytest.mark.parametrize("var", [0, 1])
def test_parts_and_whole_items_bitwise(N, var):
    ediss = L.CCS_EDISS_RECONSTRUCT if var else L.CCS_EDISS_ZERO
    scheme = "RK3_TVD" if N in (12, 52) else "RK4"
    if N % 2:  # (a cell on each pole)
        mesh = M.Mesh(N, 3, pole_inverse=True)
        s = M.initial_state(mesh, kind=L.CCS_IC_SEEDED, seed=N, lmax_oro=8)
        dt = M.cfl_dt(mesh, s, 0.5)
    else:
        mesh, s, dt = seeded_case(N, 3, seed=N)
    g = M.Stepper(mesh, dt, precision="fp64", scheme=scheme, e_dissipation=ediss)
    g.set_variant(var)
    g.set_state(s)
    g.step(2)
    o = O.Oracle.from_mesh(mesh, e_dissipation=ediss)
    o.set_state(s.arrays)
    o.run(dt, 2, scheme)
    a, b = g.get_state(), o.get_state()
    m = valid_mask(mesh)
    for k in CHECK_FIELDS:
        assert bitwise_equal(a[k], b[k], m), (k, max_rel(a[k], b[k], m))


def test_whole_items_of_a_batch_of_small_grids():
    """A batch with enough items runs them whole, each member's bits as alone in parts."""
    mesh, s, dt = seeded_case(20, 4, seed=5)
    members = []
    for k in range(14):  # 14 x 24 items of 16 x 16 cells
        x = M.Stepper(mesh, dt * (1 - 0.01 * k), precision="fp64")
        x.set_variant(1)
        x.set_state(s)
        members.append(x)
    M.Batch(members).step(2)
    m = valid_mask(mesh)
    for k in (0, 6, 13):
        r = M.Stepper(mesh, dt * (1 - 0.01 * k), precision="fp64")
        r.set_state(s)
        r.step(2)
        a, b = members[k].get_state(), r.get_state()
        for q in CHECK_FIELDS:
            assert bitwise_equal(a[q], b[q], m), (k, q)
