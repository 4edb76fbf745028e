"""The autotuner on grids that run in parts, alike in every variant: its choice does not
hang on timing noise, so a batch of such grids, which may run whole items, inherits the
variant that is fastest there."""
import pytest

from conformal_cubed_sphere_gb300 import _lib as L
from conformal_cubed_sphere_gb300 import model as M
from tests.helpers import seeded_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,N,alike", [("mixed", 24, [0, 1, 2, 3]), ("mixed", 96, [0, 1, 2, 3]),
                                               ("mixed", 150, [0, 1, 2, 3]), ("fp64", 24, [0, 1]),
                                               ("fp64", 64, [0, 1])])
def test_variants_that_run_alike_time_alike(precision, N, alike):
    mesh, s, dt = seeded_case(N, 3, seed=1)
    g = M.Stepper(mesh, dt, precision=precision, phi_mean=8000.0 * mesh.gravity)
    g.set_state(s)
    shapes = set()
    for v in alike:
        g.set_variant(v)
        shapes.add(g.stage_tile)
    assert len(shapes) == 1
    for _ in range(6):
        var, times = g.autotune(reps=2, force=True)
        assert var == 1 and g.variant[0] == 1
        assert len({times[v] for v in alike}) == 1 and times[1] > 0


def test_batch_of_autotuned_members_takes_the_variant_for_whole_items():
    mesh, s, dt = seeded_case(40, 3, seed=2)
    kw = dict(precision="mixed", phi_mean=8000.0 * mesh.gravity)
    owner = M.Stepper(mesh, dt, **kw)
    members = [owner] + [M.Stepper(mesh, dt, share_with=owner, **kw) for _ in range(39)]
    for x in members:
        x.set_state(s)
        x.autotune(reps=2, force=x is owner)
    b = M.Batch(members)
    assert [v for _, v, _ in b.info()[1]] == [1]
    assert b.stage_tile(0)[:2] == (32, 16)
    assert L.MIXED_VARIANTS[1][:2] == (32, 16)
