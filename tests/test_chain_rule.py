"""Which launches of whole mixed tiles are chained (csrc/ccs_kernels.h), compiled for the
host: not those with at most two 32 x 32 tiles an SM, where early CTAs would crowd."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "conformal_cubed_sphere_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "ccs_kernels.h"
using namespace ccs;
int main() {
  const int counts[] = {294, 304, 305, 384, 600, 864};  // C193 - C224, the line, C225 - C256, C320, C384
  for (int v = 0; v < MX_NVAR; v++)
    for (int n : counts) std::printf("%d", (int)mixed_chains(kMxTiles[v], n, 152));
  std::puts("");
}
"""


def test_chain_rule(tmp_path):
    from conformal_cubed_sphere_gb300 import build as B
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    cuda = Path(B._nvcc()).resolve().parents[1]
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", f"-I{cuda}/include", f"-I{cuda}/targets/sbsa-linux/include",
                    f"-I{cuda}/targets/x86_64-linux/include", str(src), "-o", str(tmp_path / "t"), f"-L{cuda}/lib64",
                    "-lcudart_static", "-ldl", "-lpthread", "-lrt"], check=True)
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout.strip()
    assert out == "001111" + "111111" + "001111" + "111111", out
