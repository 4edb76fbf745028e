"""FP64 lane, central operators: every tile holds at least two CTAs an SM (the 64 x 4 tile
runs them in a kernel without the face phases' shared memory), and a handle that changes
its operator family between steps gives the oracle's bits."""
import pytest

from conformal_cubed_sphere_gb300 import _lib as L
from conformal_cubed_sphere_gb300 import model as M
from oracle import oracle as O
from tests.helpers import CHECK_FIELDS, bitwise_equal, max_rel, seeded_case, valid_mask

pytestmark = pytest.mark.gpu


def _oracle_step(mesh, arrays, dt, op, n):
    o = O.Oracle.from_mesh(mesh, operator=op)
    o.set_state(arrays)
    o.run(dt, n)
    return o.get_state()


@pytest.mark.parametrize("var", [0, 1, 2])
def test_two_ctas_an_sm(var):
    mesh, s, dt = seeded_case(112, 3, seed=1)  # (whole items in every variant)
    g = M.Stepper(mesh, dt, precision="fp64", operator=L.CCS_OP_CENTRAL4)
    g.set_variant(var)
    assert g.stage_tile[:2] == g.variant[1:]
    assert g.stage_tile[2] >= 2
    g.set_operator(L.CCS_OP_WENO)
    g.set_operator(L.CCS_OP_CENTRAL6)
    assert g.stage_tile[2] >= 2


# partial tiles of both extents; 17 steps replay the graph of several steps
@pytest.mark.parametrize("N,halo", [(6, 6), (34, 3), (70, 4)])
def test_operator_changes_between_steps(N, halo):
    mesh, s, dt = seeded_case(N, halo, seed=N)
    dt *= 0.2
    g = M.Stepper(mesh, dt, precision="fp64")
    g.set_variant(2)
    g.set_state(s)
    ref = s.arrays
    m = valid_mask(mesh)
    for op, n in ((L.CCS_OP_CENTRAL2, 2), (L.CCS_OP_WENO, 1), (L.CCS_OP_CENTRAL6, 17), (L.CCS_OP_CENTRAL4, 1),
                  (L.CCS_OP_WENO, 17), (L.CCS_OP_CENTRAL4, 2)):
        g.set_operator(op)
        g.step(n)
        ref = _oracle_step(mesh, ref, dt, op, n)
        a = g.get_state()
        for k in CHECK_FIELDS:
            assert bitwise_equal(a[k], ref[k], m), (op, n, k, max_rel(a[k], ref[k], m))


def test_batch_of_central_members():
    mesh, s, dt = seeded_case(70, 3, seed=9)
    members = []
    for k in range(9):  # (9 x 216 items: several a CTA)
        x = M.Stepper(mesh, dt * (0.5 - 0.01 * k), precision="fp64", operator=L.CCS_OP_CENTRAL4)
        x.set_variant(2)
        x.set_state(s)
        members.append(x)
    b = M.Batch(members)
    assert b.stage_tile(0)[:2] == (64, 4) and b.stage_tile(0)[2] >= 2
    b.step(2)
    m = valid_mask(mesh)
    for k in (0, 8):
        ref = _oracle_step(mesh, s.arrays, dt * (0.5 - 0.01 * k), L.CCS_OP_CENTRAL4, 2)
        a = members[k].get_state()
        for q in CHECK_FIELDS:
            assert bitwise_equal(a[q], ref[q], m), (k, q)
