"""The bounds-checked build runs every tile and part shape of the stage kernels, with every
operator, E-flux option and RK scheme, and records no out-of-range index."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

from tests.bounds_parts_cases import OPTIONS

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
SHAPES = {"fp64": [(8, 8), (16, 8), (16, 16), (32, 8), (64, 4)], "mixed": [(16, 8), (16, 16), (32, 16), (32, 32)]}


def checked_env():
    from conformal_cubed_sphere_gb300 import build as B
    return dict(os.environ, CCS_GPU_LIB=str(B.build_bounds()))


def test_checked_build_reaches_every_shape_and_records_nothing():
    r = subprocess.run([sys.executable, str(ROOT / "tests" / "bounds_parts_cases.py")], env=checked_env(),
                       capture_output=True, text=True, timeout=1200, cwd=ROOT)
    assert r.returncode == 0, (r.stdout + r.stderr)[-4000:]
    seen = {tuple(line.split()[1:]) for line in r.stdout.splitlines() if line.startswith("shape ")}
    want = {(lane, str(x), str(y), str(opt)) for lane, xy in SHAPES.items() for x, y in xy
            for opt in range(len(OPTIONS))}
    assert want <= seen, sorted(want - seen)


CHILD = """
import sys
import numpy as np
sys.path.insert(0, %r)
from tests import bounds_parts_cases as B
out = {}
for key, tile, tend, state in B.runs(%r):
    name = "_".join(map(str, key))
    out[name + ".tile"] = np.array(tile)
    for q, a in enumerate(tend):
        out[name + ".t%%d" %% q] = a
    for k in B.L.STATE_FIELDS[:8]:
        out[name + "." + k] = state[k]
np.savez(sys.argv[1], **out)
"""


def test_every_shape_computes_the_same_bits(tmp_path):
    """The normal build runs these grids in 16 x 8 (mixed) and 8 x 8 or 16 x 8 parts (FP64)
    whatever the variant; the checked build runs the same grids in larger tiles, with every
    variant and option.  Tendencies and states are the same, bit for bit."""
    import numpy as np

    from conformal_cubed_sphere_gb300 import model as M
    from tests import bounds_parts_cases as B
    from tests.helpers import bitwise_equal
    grids = [(33, 3), (40, 5), (66, 4)]
    out = tmp_path / "checked.npz"
    r = subprocess.run([sys.executable, "-c", CHILD % (str(ROOT), grids), str(out)], env=checked_env(),
                       capture_output=True, text=True, timeout=1200, cwd=ROOT)
    assert r.returncode == 0, (r.stdout + r.stderr)[-4000:]
    checked = np.load(out)
    other = {"fp64": set(), "mixed": set()}
    for key, tile, tend, state in B.runs(grids):
        name = "_".join(map(str, key))
        mesh = M.Mesh(key[0], key[1], pole_inverse=key[0] % 2 == 1)
        im, m = mesh.interior_mask(), ~mesh.corner_mask()
        there = tuple(int(x) for x in checked[name + ".tile"])
        if there != tile:
            other[key[2]].add((there, tile, key[4]))
        for q, a in enumerate(tend):
            assert bitwise_equal(a, checked[name + ".t%d" % q], im), (key, tile, there, q)
        for k in B.L.STATE_FIELDS[:8]:
            assert bitwise_equal(state[k], checked[name + "." + k], m), (key, tile, there, k)
    for opt in range(len(OPTIONS)):  # every larger tile has been compared with the small parts
        for shape in ((16, 16), (32, 16), (32, 32)):
            assert (shape, (16, 8), opt) in other["mixed"], (shape, opt)
        for shape in ((16, 16), (32, 8)):
            assert any(x[0] == shape and x[2] == opt for x in other["fp64"]), (shape, opt)


@pytest.mark.parametrize("N,pairs", [(96, {(16, 8)}), (97, {(16, 16)}), (192, {(16, 16)}), (193, {(32, 16), (32, 32)})])
def test_part_rules_of_the_mixed_lane(N, pairs):
    """Where a grid alone leaves the 16 x 8 and the 16 x 16 parts."""
    from conformal_cubed_sphere_gb300 import _lib as L
    from conformal_cubed_sphere_gb300 import model as M
    from tests.bounds_parts_cases import grid_state
    mesh, s, dt = grid_state(N, 3)
    g = M.Stepper(mesh, dt, precision="mixed", phi_mean=8000.0 * mesh.gravity)
    g.set_state(s)
    seen = set()
    for var in range(len(L.MIXED_VARIANTS)):
        g.set_variant(var)
        seen.add(g.stage_tile[:2])
    assert seen == pairs, seen
