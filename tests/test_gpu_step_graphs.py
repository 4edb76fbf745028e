"""Many steps in one call replay a graph of several steps; the bits are those of single
steps, for a handle and for a batch, also after the tile variant changed."""
import pytest

from conformal_cubed_sphere_gb300 import model as M
from tests.helpers import CHECK_FIELDS, bitwise_equal, seeded_case, valid_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("scheme", ["RK4", "RK3_TVD"])
def test_many_steps_equal_single_steps(precision, scheme):
    mesh, s, dt = seeded_case(20, 3, seed=9)
    kw = dict(precision=precision, scheme=scheme, phi_mean=8000.0 * mesh.gravity)
    one, many, member = (M.Stepper(mesh, dt, **kw) for _ in range(3))
    other = M.Stepper(mesh, dt, precision="mixed" if precision == "fp64" else "fp64", phi_mean=8000.0 * mesh.gravity)
    for g in (one, many, member, other):
        g.set_state(s)
    batch = M.Batch([member, other])
    m = valid_mask(mesh)
    for n, var in ((37, 1), (16, 0), (17, 2)):  # 8 steps a graph from 16 or 17 steps on
        many.set_variant(var)
        many.step(n)
        batch.step(n)
        for _ in range(n):
            one.step(1)
        a = one.get_state()
        for g in (many, member):
            b = g.get_state()
            for k in CHECK_FIELDS:
                assert bitwise_equal(a[k], b[k], m), (n, k)
