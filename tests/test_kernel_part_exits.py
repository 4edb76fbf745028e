"""The stage kernels keep the descriptor of a CTA's work item in shared memory and write the
next item's over it.  A part beyond the panel's edge leaves its iteration early: past a
barrier, so that no thread still reads the descriptor, or out of the kernel."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "conformal_cubed_sphere_gb300" / "csrc"


@pytest.mark.parametrize("src", ["ccs_fp64.cu", "ccs_mixed.cu"])
def test_parts_beyond_the_edge_leave_past_a_barrier(src):
    code = "\n".join(line.split("//", 1)[0] for line in (CSRC / src).read_text().splitlines())
    exits = re.findall(r"if \((?:T::PART && \()?i0 > N \|\| j0 > N\)+\s*(\{[^}]*\}|[^;{]*;)", code)
    assert exits, "no early exit found"
    for body in exits:
        assert re.fullmatch(r"\s*return;\s*|\{\s*__syncthreads\(\);\s*continue;\s*\}", body), body
