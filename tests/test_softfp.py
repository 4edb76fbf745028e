"""The integer arithmetic of the FP64 lane (csrc/ccs_softfp.cuh), built for the host:
every routine must give the bits of the IEEE double operation it stands for, whatever
approximate reciprocal the device returns within its documented error."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "conformal_cubed_sphere_gb300" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "ccs_softfp.cuh"
using namespace ccs::softfp;
static std::mt19937_64 R(20);
// significands: random, few leading bits, long runs of ones, powers of two and their neighbours
static double rnd(int lo, int hi) {
  uint64_t m = R() & 0xfffffffffffffull;
  switch (R() % 6) {
    case 1: m &= ~0ull << (R() % 52); break;
    case 2: m |= (1ull << (R() % 53)) - 1; break;
    case 3: m = R() % 3 ? 0 : 0xfffffffffffffull; break;
    case 4: m = R() % 16; break;
    case 5: m = 0xfffffffffffffull - R() % 16; break;
  }
  return from_bits((uint64_t)(1023 + lo + (int)(R() % (hi - lo + 1))) << 52 | m);
}
int main() {
  long bad[9] = {0};
  for (long i = 0; i < 1500000; i++) {
    const double a = rnd(-200, 200), b = rnd(-200, 200), c = rnd(-70, 70), d = rnd(-3, 3);
    const Unp A = unpack(a), B = unpack(b);
    const Divisor D = divisor(B);
    bad[0] += pack(A) != a || pack(unpack(-a)) != a;
    bad[1] += round_double(mul(A, B)) != a * b || pack(round_unp(mul(A, B))) != a * b;
    bad[2] += round_double(div(A, D)) != a / b || pack(round_unp(div(A, D))) != a / b;
    bad[3] += round_double(one_plus(unpack(c))) != 1. + c || round_double(one_plus(unpack(0.))) != 1. ||
              pack(round_unp(add(unpack(c), unpack(d)))) != c + d || round_double(add(unpack(d), unpack(c))) != c + d;
    bad[4] += round_double(div3(A)) != a / 3. || pack(round_unp(div3(A))) != a / 3.;
    bad[5] += pack(round_unp(mul13(A))) != 13. * a;
    // square roots, also of numbers next to squares
    const double z = from_bits(bits_of(d * d) + (R() % 5) - 2);
    bad[8] += square_root(A) != std::sqrt(a) || square_root(unpack(z)) != std::sqrt(z);
    const double one = 1. + (double)(R() % (1ull << 33)) * 0x1p-52, four = 4. - (double)(R() % (1ull << 33)) * 0x1p-51;
    bad[8] += square_root(unpack(one)) != std::sqrt(one) || square_root(unpack(four)) != std::sqrt(four);
    bad[2] += round_double(div(A, divisor(unpack(one)))) != a / one || round_double(div(A, divisor(unpack(four)))) != a / four;
    // quotients next to representable and half-way values
    const double q = from_bits(bits_of(d * b) + (R() % 5) - 2);
    bad[6] += round_double(div(unpack(q), D)) != q / b ||
              round_double(one_plus(div(unpack(q), D))) != 1. + q / b;
    bad[7] += round_double(one_plus(div(A, D))) != 1. + a / b;
  }
  for (int k = 0; k < 9; k++) std::printf("%ld ", bad[k]);
  std::puts("");
}
"""

@pytest.mark.parametrize("units", [-3, -1, 0, 2])
def test_integer_operations_round_like_ieee(tmp_path, units):
    """units: how far, in units in the last place, the approximate reciprocal is off."""
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-DSF_RCP_PERTURB={units}", f"-I{CSRC}",
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    assert out.split() == ["0"] * 9, out
