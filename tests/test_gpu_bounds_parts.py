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
