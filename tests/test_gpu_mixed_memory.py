"""Device memory of a mixed-lane mesh: what the lane's kernels read, and no more."""
import pytest

from conformal_cubed_sphere_gb300 import model as M
from tests.helpers import seeded_case

pytestmark = pytest.mark.gpu


def test_mesh_of_a_mixed_handle_holds_no_array_of_the_fp64_stage_kernel():
    """Per cell of the padded field the mesh is 15 FP64 arrays (120 bytes), two FP32 fields
    (8) and eight panel-sized FP32 entries (32 / 6): 133 bytes; the FP64 stage kernel's four
    products would add 32.  The limit lies half-way."""
    torch = pytest.importorskip("torch")
    N = 384
    mesh, s, dt = seeded_case(N, 3, seed=1)
    kw = dict(precision="mixed", phi_mean=8000.0 * mesh.gravity)

    def taken(**share):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        g = M.Stepper(mesh, dt, **kw, **share)
        return g, before - torch.cuda.mem_get_info()[0]

    warm, _ = taken()  # (kernels and pools of the first use)
    warm.close()
    owner, whole = taken()
    member, without_mesh = taken(share_with=owner)
    field = 6 * (N + 6) * (N + 8)  # rows padded to a multiple of four
    per_cell = (whole - without_mesh) / field
    print(f"{per_cell:.1f} bytes a cell")
    assert per_cell < 149, per_cell
    member.close()
    owner.close()
