"""Warp votes in the kernels name the lanes that take part by a mask that a vote of the
whole group has made.  __activemask() names whichever lanes happen to run together at that
moment: the lanes of one branch may pass it in several groups, and a vote over a mask that
another group's lanes are missing from waits for them."""
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "conformal_cubed_sphere_gb300" / "csrc"


def test_no_vote_over_the_active_mask():
    for src in sorted(CSRC.glob("*.cu*")):
        code = "\n".join(line.split("//", 1)[0] for line in src.read_text().splitlines())
        assert "activemask" not in code, src.name
