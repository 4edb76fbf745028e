// ccs_fp64.cu -- FP64 parity lane: one fused launch per RK stage.
//
// Built with -fmad=false: every operation below is a separately rounded IEEE
// double operation in the order of the Fortran source (left to right), so the
// result is bitwise the reference arithmetic (gfortran -fdefault-real-8 on x86-64
// emits no FMA).
//
// Bound: the FP64 pipe, two lanes per SM and cycle (about 80 % busy at C384).  So the
// reconstructions take what depends on one cell or one second difference from shared
// memory, where each is formed once; quotients, square roots, the alphas of the WENO-Z
// weights and the constant multiples of cell values run on the integer pipes
// (ccs_softfp.cuh), which also round like IEEE; what stays is written as FMAs (F64Ops).
// C384 stage with 16 x 16 tiles: 3160 us with every operation on the FP64 pipe, 1219 with
// shared products and integer quotients, 921 now; FP64 thread instructions per cell and
// stage 1780 -> 485.  Products of two variables (squares, weight times stencil) are no
// faster in integers (+2 %) and stay.
//
// A CTA owns a tile of F64_TX x F64_TY interior cells of one panel.  It stages the
// halo'd tile (3 cells each side) of the cell quantities of the spatial operator
// in shared memory, reconstructs every face value it needs (12 live WENO-Z calls
// per cell, spatial_operators_mod.F90:80-99), forms the Rusanov face fluxes
// (:101-149), the divergence / vorticity / tendencies (:151-179), applies the RK
// stage update (time_scheme_mod.F90:69-115) and the boundary correction
// (correct_bdy_ghost, :117-125): interior cells convert their new covariant wind
// to sphere components and back, and every cell within `halo` of a panel edge
// pushes its phiG and sphere wind into the halo cell that CubedSphereFillHalo
// (ghost_mod.f90:18-82) would fill from it, converting there with that cell's
// own metric.  The output slot never feeds the same launch, so one launch per
// stage is the whole grid-wide dependency.
#include "ccs_kernels.h"
#include "ccs_bounds.cuh"
#include "ccs_softfp.cuh"

namespace ccs {

namespace {

// arrays of single-cell products of a reconstructed field (see side)
constexpr int NSING = 6;

// A tile of TX x TY cells worked on by NT threads, CTAS of them resident on an SM; phase
// 3 maps one thread to one cell.  The tile is one of the PX / TX x PY / TY parts of a work
// item of PX x PY cells (the item itself unless a launch is split).  FACES: with the face
// phases and their shared memory; a tile without runs central-difference operators only.
template <int TX_, int TY_, int NT_, int CTAS_, int PX_ = TX_, int PY_ = TY_, bool FACES_ = true>
struct F64Tile {
  static constexpr bool FACES = FACES_;
  static constexpr int TX = TX_, TY = TY_, NC = TX * TY, NT = NT_, CTAS = CTAS_;
  static constexpr int SX = PX_ / TX, SY = PY_ / TY, PX = PX_, PY = PY_;
  static constexpr int RX = TX + 6, RY = TY + 6, RN = RX * RY;
  static constexpr int NFX = TY * (TX + 1), NFY = (TY + 1) * TX, NF = NFX + NFY;
  // cells of the lines through the tile: rows of RX cells, columns of RY
  static constexpr int NLX = TY * RX, NLY = RY * TX;
  static constexpr int NSCR_F = (NSING + 2) * (NLX + NLY), NSCR_E = NSING * RN + 2 * (NLX + NLY);
  static constexpr int NSCR = !FACES ? 3 * NC : NSCR_F > NSCR_E ? NSCR_F : NSCR_E;
  static constexpr int NREC = FACES ? NF : 1;
};
}  // namespace

// x / b for the constants 3, 6, 12 of the reference (x/3., x/6., A*A*13./12.) in tiles
// outside the integer arithmetic's window, correctly rounded: q0 = RN(x y) with
// y = RN(1/b), the remainder r = x - q0 b is exact in one FMA, and q0 + r y rounded once is
// RN(x / b) (Markstein's correction, IBM J. Res. Dev. 34(1), 1990) when the quotient does
// not underflow.  Where the correction does not apply, q0 is already the IEEE result: a
// zero dividend keeps its sign, an infinite one stays infinite (the remainder would
// be inf - inf = NaN) and a NaN stays NaN.  The GPU test suite checks this against
// IEEE division.
__device__ __forceinline__ double ccs_div_const(double x, double b, double y) {
  const double q0 = x * y;
  const double r = fma(-q0, b, x);
  const double q1 = fma(r, y, q0);
  // x = +-0, +-inf or NaN, tested on the bits (the FP64 pipe is the lane's
  // bottleneck): with the sign shifted out, 0 - 1 wraps to the top of the range and
  // an all-ones exponent field is at least 0xffe0...
  const unsigned long long t = (unsigned long long)__double_as_longlong(x) << 1;
  return t - 1ull >= 0xffe0000000000000ull - 1ull ? q0 : q1;
}

// a / b for a divisor b shared by several quotients, from y = RN(1 / b) computed
// once: q0 = RN(a y), the exact remainder r = a - q0 b in one FMA, and q0 + r y
// rounded once, which is RN(a / b) when the quotient is a normal number (Markstein's
// correction, as in ccs_div_const).  The GPU test suite checks it against IEEE
// division on random operands.
__device__ __forceinline__ double ccs_div_by(double a, double b, double y) {
  const double q0 = a * y;
  const double r = fma(-q0, b, a);
  return fma(r, y, q0);
}

namespace {

// Comparisons of non-negative doubles on the integer pipes: for +0 and positive
// finite or infinite values the IEEE order is the order of the bit patterns read
// as signed integers, so these give the FP64 comparisons' results without issuing
// on the FP64 pipe (GB300 runs FP64 at 1/64 of the FP32 rate).  |x| is the bit
// pattern with the sign cleared.
__device__ __forceinline__ long long abs_bits(double x) {
  return __double_as_longlong(x) & 0x7fffffffffffffffLL;
}

// WENO_limiter, spatial_operators_mod.F90:282-361: the "+" side.  The "-" side's formulas
// are these with the cells in mirrored order, operation for operation, so a caller passes
// them mirrored: the two sides of a face sit in neighbouring lanes, and with a routine each
// a warp runs both (a C384 tendency with every tile out of the window: 6.8 -> 3.7 ms).
__device__ __forceinline__ double weno5z(double Qim2, double Qim1, double Qi, double Qip1, double Qip2) {
  const double y3 = 1. / 3., y6 = 1. / 6., y12 = 1. / 12.;
  const double s0 = ccs_div_const(Qim2, 3., y3) - 7. / 6. * Qim1 + 11. / 6. * Qi;
  const double s1 = ccs_div_const(-Qim1, 6., y6) + 5. / 6. * Qi + 1. / 3. * Qip1;
  const double s2 = ccs_div_const(Qi, 3., y3) + 5. / 6. * Qip1 - 1. / 6. * Qip2;
  const double a0 = Qim2 - 2. * Qim1 + Qi;
  const double a1 = Qim1 - 2. * Qi + Qip1;
  const double a2 = Qi - 2. * Qip1 + Qip2;
  const double b0 = Qim2 - 4. * Qim1 + 3. * Qi;
  const double b1 = Qim1 - Qip1;
  const double b2 = 3. * Qi - 4. * Qip1 + Qip2;
  const double be0 = ccs_div_const(a0 * a0 * 13., 12., y12) + b0 * b0 * 0.25;
  const double be1 = ccs_div_const(a1 * a1 * 13., 12., y12) + b1 * b1 * 0.25;
  const double be2 = ccs_div_const(a2 * a2 * 13., 12., y12) + b2 * b2 * 0.25;
  // the betas are sums of squares (never -0 or negative), the taus absolute values
  const long long t40 = abs_bits(be0 - be1), t41 = abs_bits(be1 - be2);
  const double tau5 = fabs(be2 - be0);
  long long mn = __double_as_longlong(be0);
  if (__double_as_longlong(be1) < mn) mn = __double_as_longlong(be1);
  if (__double_as_longlong(be2) < mn) mn = __double_as_longlong(be2);
  // a comparison with a NaN (of betas that overflow, or of a cell that is not finite) is
  // false; with the taus numbers, the betas are
  const bool numbers = t40 <= 0x7ff0000000000000LL && t41 <= 0x7ff0000000000000LL;
  double w0, w1, w2;
  if (numbers && t40 <= mn && t41 > mn) {
    w0 = 1. / 3.; w1 = 2. / 3.; w2 = 0.;
  } else if (numbers && t40 > mn && t41 < mn) {
    w0 = 0.; w1 = 2. / 3.; w2 = 1. / 3.;
  } else {
    const double eps = 1.E-2;
    const double al0 = 0.1 * (1. + tau5 / (eps + be0));
    const double al1 = 0.6 * (1. + tau5 / (eps + be1));
    const double al2 = 0.3 * (1. + tau5 / (eps + be2));
    const double sum = ((0. + al0) + al1) + al2;
    // omega = alpha / sum(alpha): one IEEE reciprocal for the three quotients.  Each
    // alpha is at least its linear weight (0.1) and sum >= alpha, so the quotients lie
    // in (2^-1004, 1] whenever sum < 2^1000 (tested on the bits); a larger, infinite
    // or NaN sum takes IEEE division
    if (__double_as_longlong(sum) < 0x7e70000000000000LL) {
      const double ys = 1. / sum;
      w0 = ccs_div_by(al0, sum, ys); w1 = ccs_div_by(al1, sum, ys); w2 = ccs_div_by(al2, sum, ys);
    } else {
      w0 = al0 / sum; w1 = al1 / sum; w2 = al2 / sum;
    }
  }
  return ((0. + s0 * w0) + s1 * w1) + s2 * w2;
}

// Centred difference of cell values f[-3s .. 3s] around f[0], divided by the
// stencil's denominator times d: spatial_operators_mod_2nd.F90:54-59,
// spatial_operators_mod_4th.F90:58-63, spatial_operators_mod_6th.F90:62-67.
__device__ __forceinline__ double central_diff(int op, const double *f, int s, double d) {
  if (op == 2) return (f[s] - f[-s]) / (2. * d);
  if (op == 4) return (f[-2 * s] - 8. * f[-s] + 8. * f[s] - f[2 * s]) / (12. * d);
  return (-f[-3 * s] + 9. * f[-2 * s] - 45. * f[-s] + 45. * f[s] - 9. * f[2 * s] + f[3 * s]) / (60. * d);
}

// Sums and products as FMAs: a DADD or DMUL warp instruction holds the FP64 pipe for
// 19 cycles, a DFMA for 16 (measured, 4-16 warps per SM).  a 1 + b and a b + (-0) are
// the sum and the product to the last bit and sign; the two constants come from memory,
// where the compiler cannot see that the FMA could be an addition or a multiplication.
struct F64Ops {
  double one, neg0;
  __device__ __forceinline__ double add(double a, double b) const { return fma(a, one, b); }
  __device__ __forceinline__ double sub(double a, double b) const { return fma(-b, one, a); }
  __device__ __forceinline__ double mul(double a, double b) const { return fma(a, b, neg0); }
  // x / b from y = RN(1 / b), as ccs_div_const
  __device__ __forceinline__ double div_const(double x, double b, double y) const {
    const double q0 = mul(x, y);
    const double r = fma(-q0, b, x);
    const double q1 = fma(r, y, q0);
    const unsigned long long t = (unsigned long long)__double_as_longlong(x) << 1;
    return t - 1ull >= 0xffe0000000000000ull - 1ull ? q0 : q1;
  }
};

// phiG / sqrtG from the grid's reciprocals y = RN(1 / sqrtG), which are zero where sqrtG is
// not in [2^-400, 2^300); there, and for a phiG whose quotient might not be normal, IEEE
// division
__device__ __forceinline__ double div_depth(const F64Ops &f, double x, double b, double y) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  if ((e - 400u >= 1200u && x != 0.) || __double2hiint(y) == 0) return x / b;
  return f.div_const(x, b, y);
}

// x / b on the integer pipes, b prepared by the host (y zero: b not in [2^-400, 2^300));
// values whose quotient might leave the normal range (and zeros) take IEEE division
__device__ __forceinline__ double div_by(double x, const softfp::Divisor &d, double b) {
  const uint32_t h = (uint32_t)__double2hiint(x);
  if (((h >> 20) & 0x7ffu) - 400u >= 1200u || d.y == 0u) return x / b;
  const double q = softfp::round_double(softfp::div(softfp::unpack(x), d));
  return __hiloint2double((int)((uint32_t)__double2hiint(q) | (h & 0x80000000u)), __double2loint(q));
}
__device__ __forceinline__ double div_by6(double x) {
  const uint32_t h = (uint32_t)__double2hiint(x);
  if (((h >> 20) & 0x7ffu) - 400u >= 1200u) return x / 6.;
  softfp::Quot t = softfp::div3(softfp::unpack(x));
  t.e -= 1;
  const double q = softfp::round_double(t);
  return __hiloint2double((int)((uint32_t)__double2hiint(q) | (h & 0x80000000u)), __double2loint(q));
}

// -q(-3) + 9 q(-2) - 45 q(-1) + 45 q(1) - 9 q(2) + q(3), left to right
// (spatial_operators_mod.F90:165,169)
__device__ __forceinline__ double diff6(const F64Ops &f, const double *q, int s) {
  double t = f.add(-q[-3 * s], f.mul(9., q[-2 * s]));
  t = f.sub(t, f.mul(45., q[-s]));
  t = f.add(t, f.mul(45., q[s]));
  t = f.sub(t, f.mul(9., q[2 * s]));
  return f.add(t, q[3 * s]);
}

// x / 2 of a normal x by its exponent; zeros, infinities, NaNs and values at the
// bottom of the range take the FP64 multiplication
__device__ __forceinline__ double half_of(double x) {
  const uint32_t h = softfp::hi32(softfp::bits_of(x)), e = h & 0x7ff00000u;
  if (e - 0x00200000u < 0x7fc00000u) return __hiloint2double((int)(h - 0x00100000u), __double2loint(x));
  return 0.5 * x;
}

// x as RK4's doubled tendencies take it: where 2 x overflows an infinity, so that
// fma(2, x, a) is infinite where the reference's a + 2 x is
__device__ __forceinline__ double to_double(double x) {
  const uint32_t h = softfp::hi32(softfp::bits_of(x));
  const bool over = (h & 0x7ff00000u) == 0x7fe00000u;
  return __hiloint2double((int)(over ? (h & 0x80000000u) | 0x7ff00000u : h), over ? 0 : __double2loint(x));
}

// Whether the integer arithmetic of the reconstructions covers a field value: zero or
// of magnitude in [2^-200, 2^200).  Differences of such values are zero or at least
// 2^-253, so the smoothness indicators lie in {0} or [2^-510, 2^410], the weights in
// [2^-415, 1], and no product, sum or quotient of a reconstruction leaves the normal range.
__device__ __forceinline__ bool in_window(double x) {
  const unsigned long long t = (unsigned long long)__double_as_longlong(x) << 1;
  return t == 0ull || t - ((unsigned long long)(1023 - 200) << 53) < ((unsigned long long)400 << 53);
}

// The switches of spatial_operators_mod.F90:348-351 on tau40 = |be0 - be1|, tau41 =
// |be1 - be2| and mn = min(be): first = (tau40 <= mn && tau41 > mn), last = (tau40 > mn &&
// tau41 < mn), the differences rounded as FP64 rounds them.  Single precision decides
// them when both differences are further from mn than its error: the betas as floats
// relative to the largest exponent, cut to 20 bits (error 2^-20, the largest in [1, 2)), so
// tau - mn is off by less than 4e-6.  A lane with a closer call takes the FP64 differences.
__device__ __forceinline__ void switches(const F64Ops &f, double be0, double be1, double be2, long long mn,
                                         bool &first, bool &last) {
  const int h0 = __double2hiint(be0), h1 = __double2hiint(be1), h2 = __double2hiint(be2);
  const int base = (max(max(h0, h1), h2) & 0x7ff00000) - (127 << 20);
  const float f0 = __int_as_float(max(h0 - base, 0) << 3), f1 = __int_as_float(max(h1 - base, 0) << 3),
              f2 = __int_as_float(max(h2 - base, 0) << 3);
  const float fm = fminf(fminf(f0, f1), f2);
  const float d40 = fabsf(f0 - f1) - fm, d41 = fabsf(f1 - f2) - fm;
  first = d40 < 0.f && d41 > 0.f;
  last = d40 > 0.f && d41 < 0.f;
  if (!(fminf(fabsf(d40), fabsf(d41)) > 1e-5f)) {
    const long long t40 = abs_bits(f.sub(be0, be1)), t41 = abs_bits(f.sub(be1, be2));
    first = t40 <= mn && t41 > mn;
    last = t40 > mn && t41 < mn;
  }
}

// a w
__device__ __forceinline__ double times(double a, softfp::Unp w) {
  using namespace softfp;
  const unsigned long long bits = __double_as_longlong(a), sign = bits & 0x8000000000000000ull;
  const double r = round_double(mul(unpack(a), w));
  return __longlong_as_double((bits << 1 == 0 ? 0ull : (unsigned long long)__double_as_longlong(r)) | sign);
}

// One WENO-Z reconstruction (WENO_limiter, spatial_operators_mod.F90:282-361) of a
// cell's value at one of its two faces, in the reference's order of operations:
// Q at stride +s for the "+" side (face after the cell), -s for the "-" side, whose
// formulas are the mirrored ones.  What depends on a single cell, or on three cells
// alike in the neighbouring reconstructions, comes from shared memory:
//   G[0..5] at the cell, arrays SG apart: Q/3, 7/6 Q, 11/6 Q, 5/6 Q, 1/3 Q, 3 Q
//   ga at the cell: 13/12 (second difference centred there)^2, same orientation
// (Q/6 and 1/6 Q are exact halves of Q/3 and 1/3 Q; multiplications by 2, 4 and 1/4 are
// exact and fuse.)  The quotients run on the integer pipes (ccs_softfp.cuh).
__device__ __forceinline__ double side(const F64Ops &f, const double *Q, int s, const double *G, int SG, int gs,
                                       const double *ga, int as) {
  const double q3 = G[5 * SG];
  const double b0 = f.add(fma(-4., Q[-s], Q[-2 * s]), q3);
  const double b1 = f.sub(Q[-s], Q[s]);
  const double b2 = f.add(fma(-4., Q[s], q3), Q[2 * s]);
  const double be0 = fma(f.mul(b0, b0), 0.25, ga[-as]);
  const double be1 = fma(f.mul(b1, b1), 0.25, ga[0]);
  const double be2 = fma(f.mul(b2, b2), 0.25, ga[as]);
  const double tau5 = fabs(f.sub(be2, be0));
  long long mn = __double_as_longlong(be0);
  if (__double_as_longlong(be1) < mn) mn = __double_as_longlong(be1);
  if (__double_as_longlong(be2) < mn) mn = __double_as_longlong(be2);
  bool first, last;  // the reference's two switches to fixed weights
  switches(f, be0, be1, be2, mn, first, last);
  using namespace softfp;
  double w0 = first ? 1. / 3. : 0., w1 = 2. / 3., w2 = first ? 0. : 1. / 3.;
  const double s0 = f.add(f.sub(G[-2 * gs], G[SG - gs]), G[2 * SG]);
  const double s1 = f.add(fma(-0.5, G[-gs], G[3 * SG]), G[4 * SG + gs]);
  const double s2 = fma(-0.5, G[4 * SG + 2 * gs], f.add(G[0], G[3 * SG + gs]));
  if (!first && !last) {
    // eps + beta: beta itself from 2^48 on (eps is less than half its last place), which
    // is every beta of the fluxes and phitG
    double e0 = be0, e1 = be1, e2 = be2;
    if (mn < 0x42f0000000000000LL) {
      const double eps = 1.E-2;
      e0 = f.add(eps, be0); e1 = f.add(eps, be1); e2 = f.add(eps, be2);
    }
    constexpr Unp k01 = constant(0.1), k06 = constant(0.6), k03 = constant(0.3);
    const Unp t = unpack(tau5);  // tau5 = 0 reads as 2^-1023: 1 + tau5 / .. rounds to 1 either way
    const Unp p0 = round_unp(one_plus(div(t, divisor(unpack(e0)))));
    const Unp p1 = round_unp(one_plus(div(t, divisor(unpack(e1)))));
    const Unp p2 = round_unp(one_plus(div(t, divisor(unpack(e2)))));
    const Unp a0 = round_unp(mul(p0, k01)), a1 = round_unp(mul(p1, k06)), a2 = round_unp(mul(p2, k03));
    const Divisor d = divisor(round_unp(add(round_unp(add(a0, a1)), a2)));
    w0 = round_double(div(a0, d));
    w1 = round_double(div(a1, d));
    w2 = round_double(div(a2, d));
  }
  return f.add(f.add(fma(s0, w0, 0.), f.mul(s1, w1)), f.mul(s2, w2));
}

// 13/12 a^2 rounded as the reference does: ((a a) 13) / 12
__device__ __forceinline__ double curvature(double a) {
  using namespace softfp;
  const Unp u = unpack(a);
  Quot g = div3(round_unp(mul13(round_unp(mul(u, u)))));
  g.e -= 2;
  return __double_as_longlong(a) << 1 == 0 ? 0. : round_double(g);
}

template <class T>
struct Smem {
  // cell quantities on the halo'd tile (row-major [RY][RX])
  double phit[T::RN], phitG[T::RN], E[T::RN], Fx[T::RN], Fy[T::RN], uC[T::RN], vC[T::RN], u[T::RN], v[T::RN];
  // face values: sums of the two sides of the flux and E, difference of phitG's (and of
  // the wind's: E dissipation); then the Rusanov fluxes of phiG and E in the first two
  double rec[4][T::NREC];
  // per-cell products of the fields of one pass: either fields of their own on the rows
  // and columns, or one field on the halo'd tile with curvatures on rows and columns; then
  // the cells' new values for the push
  double scr[T::NSCR];
  F64Stage st;  // the work item's stage descriptor
};

__device__ __forceinline__ bool is_corner(int i, int j, int N) {
  return (i < 1 || i > N) && (j < 1 || j > N);
}

__device__ __forceinline__ void store_singles(const F64Ops &f, double *G, int SG, double q) {
  using namespace softfp;
  const double t = round_double(div3(unpack(q)));
  const double third = __longlong_as_double(
      __double_as_longlong(q) << 1 == 0 ? __double_as_longlong(q)
              : __double_as_longlong(t) | (__double_as_longlong(q) & (long long)0x8000000000000000ull));
  G[0] = third;
  constexpr Unp k76 = constant(7. / 6.), k116 = constant(11. / 6.), k56 = constant(5. / 6.), k13 = constant(1. / 3.);
  G[SG] = times(q, k76);
  G[2 * SG] = times(q, k116);
  G[3 * SG] = times(q, k56);
  G[4 * SG] = times(q, k13);
  G[5 * SG] = fma(2., q, q);
}

// Reconstructs one pass of fields at every face of the tile, both sides: QX along the
// rows and QY along the columns (the same array for E and phitG).  rec receives
// (+) + (-) or, with DIFF, (-) - (+).  nx, ny: the tile's cells inside the panel.
template <class T, bool SAME, bool DIFF>
__device__ __forceinline__ void reconstruct(Smem<T> &S, const F64Ops &f, const double *QX, const double *QY,
                                            double *rec, int nx, int ny, bool slow) {
  constexpr int TX = T::TX, TY = T::TY, RX = T::RX, RY = T::RY, RN = T::RN, NLX = T::NLX, NLY = T::NLY;
  constexpr int NFX = T::NFX, NF = T::NF, NT = T::NT;
  const int tid = threadIdx.x;
  // products: [NSING] arrays on the halo'd tile (SAME) or on the rows / columns, then
  // the curvatures of the "+" and "-" orientation on the rows and on the columns
  double *GX = S.scr, *GY = SAME ? S.scr : S.scr + NSING * NLX;
  constexpr int SGX = SAME ? RN : NLX, SGY = SAME ? RN : NLY;
  double *AX = S.scr + (SAME ? NSING * RN : NSING * (NLX + NLY)), *AY = AX + 2 * NLX;
  if (!slow) {
    if constexpr (SAME) {
      for (int r = tid; r < RN; r += NT) store_singles(f, GX + r, SGX, QX[r]);
    } else {
      for (int r = tid; r < NLX + NLY; r += NT) {
        if (r < NLX) {
          store_singles(f, GX + r, SGX, QX[3 * RX + r]);
        } else {
          const int q = r - NLX;
          store_singles(f, GY + q, SGY, QY[(q / TX) * RX + q % TX + 3]);
        }
      }
    }
    for (int r = tid; r < 2 * (NLX + NLY); r += NT) {
      const bool minus = r >= NLX + NLY;
      const int q = minus ? r - (NLX + NLY) : r;
      const double *z;
      double *o;
      int st;
      bool in;
      if (q < NLX) {
        const int ci = q % RX;
        in = ci >= 1 && ci < RX - 1;
        z = QX + 3 * RX + q;
        st = 1;
        o = AX + (minus ? NLX : 0) + q;
      } else {
        const int k = q - NLX, cj = k / TX;
        in = cj >= 1 && cj < RY - 1;
        z = QY + cj * RX + k % TX + 3;
        st = RX;
        o = AY + (minus ? NLY : 0) + k;
      }
      if (in) {
        const int d = minus ? -st : st;
        *o = curvature(f.add(fma(-2., z[0], z[-d]), z[d]));
      }
    }
    __syncthreads();
  }
  // lanes 2 k and 2 k + 1 take the two sides of one face; two rounds share one FP64
  // addition: the even lanes add the first round's faces, the odd lanes the second's
  double first = 0.;
  int first_face = -1;
  for (int t0 = tid & ~31; t0 < 2 * NF; t0 += NT) {
    const int t = t0 + (tid & 31), face = t >> 1, minus = t & 1;
    double val = 0.;
    if (t < 2 * NF) {
      bool in;
      int cell, lcell, st, ls;  // the cell in the halo'd tile and on its line's arrays
      const double *z, *G, *A;
      if (face < NFX) {
        const int lj = face / (TX + 1), ci = face % (TX + 1) + 2 + minus;
        in = lj < ny && ci - 2 - minus <= nx;
        cell = (lj + 3) * RX + ci;
        lcell = lj * RX + ci;
        st = ls = 1;
        z = QX;
        G = GX + (SAME ? cell : lcell);
        A = AX + (minus ? NLX : 0);
      } else {
        const int fy = face - NFX, li = fy % TX, cj = fy / TX + 2 + minus;
        in = li < nx && cj - 2 - minus <= ny;
        cell = cj * RX + li + 3;
        lcell = cj * TX + li;
        st = RX;
        ls = TX;
        z = QY;
        G = GY + (SAME ? cell : lcell);
        A = AY + (minus ? NLY : 0);
      }
      if (in && ccs_inb(cell - 2 * st, RN, 211) && ccs_inb(cell + 2 * st, RN, 212)) {
        z += cell;
        if (minus) { st = -st; ls = -ls; }
        if (slow)
          val = weno5z(z[-2 * st], z[-st], z[0], z[st], z[2 * st]);
        else
          val = side(f, z, st, G, face < NFX ? SGX : SGY, SAME ? st : ls, A + lcell, ls);
      }
    }
    if (t0 + NT < 2 * NF && first_face < 0) {
      first = val;
      first_face = face;
      continue;
    }
    const bool two = first_face >= 0;  // uniform in the warp
    const double o1 = __shfl_xor_sync(0xffffffffu, two ? first : val, 1), o2 = __shfl_xor_sync(0xffffffffu, val, 1);
    const double plus = minus ? o2 : two ? first : val, neg = minus ? val : o1;
    const double sum = DIFF ? f.sub(neg, plus) : f.add(plus, neg);
    const int dst = minus || !two ? face : first_face;
    if ((two || !minus) && dst < NF && ccs_inb(dst, NF, 213)) rec[dst] = sum;
    first_face = -1;
  }
  __syncthreads();
}

// Writes cell c of the stage's output from its phiG and sphere wind: the covariant and
// contravariant wind by the cell's own metric, and phi.
__device__ __forceinline__ void complete(const F64Ops &f, const F64Stage &st, int64_t c, double phiG, double zon,
                                         double mer) {
  const MeshF64 &m = st.m;
  const double g11 = __ldg(m.gia11 + c), g12 = __ldg(m.gia12 + c), g21 = __ldg(m.gia21 + c), g22 = __ldg(m.gia22 + c);
  const double i11 = __ldg(m.ig11 + c), i12 = __ldg(m.ig12 + c), i21 = __ldg(m.ig21 + c), i22 = __ldg(m.ig22 + c);
  const double sg = __ldg(m.sqrtG + c), rsg = __ldg(m.rsqrtG + c);
  const double u = f.add(f.mul(g11, zon), f.mul(g12, mer));
  const double v = f.add(f.mul(g21, zon), f.mul(g22, mer));
  const double uC = f.add(f.mul(i11, u), f.mul(i12, v));
  const double vC = f.add(f.mul(i21, u), f.mul(i22, v));
  const double phi = div_depth(f, phiG, sg, rsg);
  st.out.phiG[c] = phiG;
  st.out.u[c] = u;
  st.out.v[c] = v;
  st.out.uC[c] = uC;
  st.out.vC[c] = vC;
  st.out.phi[c] = phi;
  if (st.zonal) {
    st.zonal[c] = zon;
    st.merid[c] = mer;
  }
}

template <class T>
__global__ void __launch_bounds__(T::NT, T::CTAS)
f64_stage_kernel(const F64Stage *__restrict__ stages, const WorkItem *__restrict__ work, int nwork) {
  constexpr int TX = T::TX, TY = T::TY, RX = T::RX, RN = T::RN, NFX = T::NFX, NF = T::NF, NT = T::NT;
  constexpr int PARTS = T::SX * T::SY;
  static_assert(T::NC <= NT, "phase 3 maps one thread to one cell");
  extern __shared__ __align__(16) double smem_raw[];
  Smem<T> &S = *reinterpret_cast<Smem<T> *>(smem_raw);
  const int tid = threadIdx.x;

  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const WorkItem wi = work[w / PARTS];
    const F64Stage &st = S.st;
    {  // (the loop's last barrier is behind every thread's use of the previous one)
      const uint64_t *src = reinterpret_cast<const uint64_t *>(stages + wi.inst);
      uint64_t *dst = reinterpret_cast<uint64_t *>(&S.st);
      static_assert(sizeof(F64Stage) % sizeof(uint64_t) == 0, "copied in words");
      for (int k = tid; k < (int)(sizeof(F64Stage) / sizeof(uint64_t)); k += NT) dst[k] = __ldg(src + k);
    }
    __syncthreads();
    const Layout L = st.L;
    const int N = L.N, p = wi.panel;
    const int i0 = 1 + wi.tx * T::PX + w % T::SX * TX, j0 = 1 + wi.ty * T::PY + w / T::SX % T::SY * TY;
    if (i0 > N || j0 > N) {  // a part beyond the panel's edge
      __syncthreads();  // (every thread has read S.st before the next part's is written)
      continue;
    }
    const bool ediss = st.ediss != 0;
    const int op = st.op;  // uniform over the work item
    const F64Ops f{st.one, st.neg0};
#ifdef CCS_BOUNDS
    // poison the tile arrays: a read of a slot this tile never wrote shows up as NaN
    // in the result (checked build only)
    for (int k = tid; k < (int)((sizeof(S) - sizeof(S.st)) / sizeof(double)); k += NT)
      smem_raw[k] = __longlong_as_double(0x7ff8000000000000LL);
    __syncthreads();
#endif

    stage_wait();

    // ---- phase 1: cell quantities (spatial_operators_mod.F90:71-78) ----------
    // (cells outside the panel and its edge halos are set to zero: the faces that
    // would read them belong to no interior cell)
    bool odd = false;
    for (int r = tid; r < RN; r += NT) {
      const int li = r % RX, lj = r / RX;
      const int i = i0 - 3 + li, j = j0 - 3 + lj;
      double phit = 0., phitG = 0., E = 0., Fx = 0., Fy = 0., uC = 0., vC = 0., u = 0., v = 0.;
      const int64_t c = L.idx(i, j, p);
      if (i >= -2 && i <= N + 3 && j >= -2 && j <= N + 3 && !is_corner(i, j, N) && ccs_inb(c, L.field, 201)) {
        const double phiG = __ldcg(st.in.phiG + c), phi = __ldcg(st.in.phi + c);
        u = __ldcg(st.in.u + c);
        v = __ldcg(st.in.v + c);
        uC = __ldcg(st.in.uC + c);
        vC = __ldcg(st.in.vC + c);
        phit = f.add(phi, __ldg(st.m.phis + c));
        phitG = f.mul(phit, __ldg(st.m.sqrtG + c));
        const double K = half_of(f.add(f.mul(u, uC), f.mul(v, vC)));
        E = f.add(phit, K);
        Fx = f.mul(phiG, uC);
        Fy = f.mul(phiG, vC);
        odd = odd || __double_as_longlong(phit) <= 0 || !in_window(phitG) || !in_window(E) || !in_window(Fx) || !in_window(Fy) ||
              !in_window(u) || !in_window(v);
      }
      S.phit[r] = phit; S.phitG[r] = phitG; S.E[r] = E; S.Fx[r] = Fx; S.Fy[r] = Fy;
      S.uC[r] = uC; S.vC[r] = vC; S.u[r] = u; S.v[r] = v;
    }
    // a tile with values outside the window of the integer arithmetic (or without
    // positive depth) takes the FP64 instructions throughout
    const bool slow = __syncthreads_or(odd);
    const int nx = min(TX, N + 1 - i0), ny = min(TY, N + 1 - j0);

    // ---- phase 2: face reconstructions (weno, :183-277) ---------------------
    // (the central-difference operators have no faces: straight to phase 3)
    if constexpr (T::FACES) if (op == CCS_OP_WENO) {
    reconstruct<T, false, false>(S, f, S.Fx, S.Fy, S.rec[0], nx, ny, slow);
    reconstruct<T, true, false>(S, f, S.E, S.E, S.rec[1], nx, ny, slow);
    reconstruct<T, true, true>(S, f, S.phitG, S.phitG, S.rec[2], nx, ny, slow);
    if (ediss) reconstruct<T, false, true>(S, f, S.u, S.v, S.rec[3], nx, ny, slow);

    // ---- phase 2b: Rusanov fluxes at faces (:101-149) ------------------------
    for (int face = tid; face < NF; face += NT) {
      double a, b, pa, pb, lam;  // contravariant wind and phit at the two cells, mean IG diagonal
      if (face < NFX) {
        const int fi = face % (TX + 1), lj = face / (TX + 1);
        const int r = (lj + 3) * RX + fi + 2;  // cell f; cell f+1 is r + 1
        if (i0 - 1 + fi > N || j0 + lj > N || !ccs_inb(r + 1, RN, 214)) continue;
        a = S.uC[r + 1]; b = S.uC[r];
        pa = S.phit[r + 1]; pb = S.phit[r];
        lam = __ldg(st.m.lamx + L.idx(i0 - 1 + fi, j0 + lj, p));
      } else {
        const int fy = face - NFX;
        const int li = fy % TX, fj = fy / TX;
        const int r = (fj + 2) * RX + li + 3;  // cell g; cell g+1 is r + RX
        if (i0 + li > N || j0 - 1 + fj > N || !ccs_inb(r + RX, RN, 215)) continue;
        a = S.vC[r + RX]; b = S.vC[r];
        pa = S.phit[r + RX]; pb = S.phit[r];
        lam = __ldg(st.m.lamy + L.idx(i0 + li, j0 - 1 + fj, p));
      }
      const double uBdy = half_of(f.add(a, b));
      const double phitBdy = half_of(f.add(pa, pb));
      // max(|u - c|, |u + c|) = |u| + c, rounded alike
      const double c2 = f.mul(lam, phitBdy);
      const double cs = ((uint32_t)__double2hiint(c2) >> 20) - 400u < 1200u
                            ? softfp::square_root(softfp::unpack(c2))
                            : sqrt(c2);
      double mx = f.add(fabs(uBdy), cs);
      // a wave speed that is not finite (mx >= 0, or a NaN of either sign), and a cell that is
      // not, keep the reference's comparison and its E term
      const bool exact = slow || (uint32_t)__double2hiint(mx) >= 0x7ff00000u;
      if (exact) {
        const double e1 = uBdy - cs, e2 = uBdy + cs;
        mx = abs_bits(e2) > abs_bits(e1) ? fabs(e2) : fabs(e1);
      }
      const double FS = S.rec[0][face], PD = S.rec[2][face];
      double ES = S.rec[1][face];
      // the never-written u_ext / v_ext slots (CCS_EDISS_ZERO) contribute mx (0 - 0): zero
      // but for a wave speed that is not finite
      if (ediss || exact) ES = f.sub(ES, f.mul(mx, ediss ? S.rec[3][face] : 0.));
      S.rec[0][face] = half_of(f.sub(FS, f.mul(mx, PD)));
      S.rec[1][face] = half_of(ES);
    }
    __syncthreads();
    }  // op == CCS_OP_WENO

    // ---- phase 3: tendencies, stage update, boundary correction --------------
    double *new_phiG = S.scr, *new_zon = S.scr + T::NC, *new_mer = S.scr + 2 * T::NC;  // for the push
    {
      const int li = tid % TX, lj = tid / TX;
      const int i = i0 + li, j = j0 + lj;
      const int64_t c = L.idx(i, j, p);
      const int rc = (lj + 3) * RX + li + 3;
      if (tid < T::NC && i <= N && j <= N && ccs_inb(c, L.field, 221) && ccs_inb(rc + 3 * RX, RN, 222) &&
          ccs_inb(NFX + (lj + 1) * TX + li, NF, 223)) {
        // every global operand before the first store, so that the loads overlap
        const int kind = st.kind;
        const double sgf = __ldg(st.m.sqrtGf + c);
        double y0[3] = {0., 0., 0.}, ac[3] = {0., 0., 0.};
        if (kind != K_TEND) {
          y0[0] = __ldcg(st.y0phiG + c); y0[1] = __ldcg(st.y0u + c); y0[2] = __ldcg(st.y0v + c);
          if (kind == K_RK4_2 || kind == K_RK4_4) { ac[0] = __ldcg(st.accphiG + c); ac[1] = __ldcg(st.accu + c); ac[2] = __ldcg(st.accv + c); }
          if (kind == K_RK3_2 || kind == K_RK3_3) { ac[0] = __ldcg(st.in.phiG + c); ac[1] = S.u[rc]; ac[2] = S.v[rc]; }
        }
        const double a11 = __ldg(st.m.aig11 + c), a12 = __ldg(st.m.aig12 + c), a21 = __ldg(st.m.aig21 + c),
                     a22 = __ldg(st.m.aig22 + c);
        double dfluxdx, dEdx, dvdx, dfluxdy, dEdy, dudy;
        if (T::FACES && op == CCS_OP_WENO) {
          const double *FF = S.rec[0], *EF = S.rec[1];
          const int xl = lj * (TX + 1) + li, xr = xl + 1;
          const int yb = NFX + lj * TX + li, yt = yb + TX;
          // (spatial_operators_mod.F90:153-169)
          dfluxdx = div_by(f.sub(FF[xr], FF[xl]), st.by_dx, st.dx);
          dEdx = div_by(f.sub(EF[xr], EF[xl]), st.by_dx, st.dx);
          dvdx = div_by(diff6(f, S.v + rc, 1), st.by_dx60, st.dx60);
          dfluxdy = div_by(f.sub(FF[yt], FF[yb]), st.by_dy, st.dy);
          dEdy = div_by(f.sub(EF[yt], EF[yb]), st.by_dy, st.dy);
          dudy = div_by(diff6(f, S.u + rc, RX), st.by_dy60, st.dy60);
        } else {
          dfluxdx = central_diff(op, S.Fx + rc, 1, st.dx);
          dEdx = central_diff(op, S.E + rc, 1, st.dx);
          dvdx = central_diff(op, S.v + rc, 1, st.dx);
          dfluxdy = central_diff(op, S.Fy + rc, RX, st.dy);
          dEdy = central_diff(op, S.E + rc, RX, st.dy);
          dudy = central_diff(op, S.u + rc, RX, st.dy);
        }
        const double vort = f.add(f.sub(dvdx, dudy), sgf);
        const double uCc = S.uC[rc], vCc = S.vC[rc];
        const double t[3] = {-f.add(dfluxdx, dfluxdy), f.add(-dEdx, f.mul(vort, vCc)), f.sub(-dEdy, f.mul(vort, uCc))};

        if (kind == K_TEND) {
          st.tphiG[c] = t[0];
          st.tu[c] = t[1];
          st.tv[c] = t[2];
        } else {
          double n[3];
          if (kind == K_RK4_2)
#pragma unroll
            for (int q = 0; q < 3; q++) ac[q] = fma(2., to_double(t[q]), ac[q]);
#pragma unroll
          for (int q = 0; q < 3; q++) {
            if (kind == K_RK4_4)
              n[q] = f.add(y0[q], f.mul(st.c1, div_by6(f.add(ac[q], t[q]))));
            else if (kind == K_RK3_2)
              n[q] = f.add(f.add(f.mul(0.75, y0[q]), f.mul(0.25, ac[q])), f.mul(st.c1, t[q]));
            else if (kind == K_RK3_3)
              n[q] = f.add(f.add(f.div_const(y0[q], 3., 1. / 3.), f.mul(2. / 3., ac[q])), f.mul(st.c1, t[q]));
            else
              n[q] = f.add(y0[q], f.mul(st.c1, t[q]));
          }
          // correct_bdy_ghost: P2SP (interior), SP2P, cov2contrav, phi = phiG / sqrtG
          const double zon = f.add(f.mul(a11, n[1]), f.mul(a12, n[2]));
          const double mer = f.add(f.mul(a21, n[1]), f.mul(a22, n[2]));
          new_phiG[tid] = n[0]; new_zon[tid] = zon; new_mer[tid] = mer;
          if (kind == K_RK4_1) {
            st.accphiG[c] = t[0]; st.accu[c] = t[1]; st.accv[c] = t[2];
          } else if (kind == K_RK4_2) {
            st.accphiG[c] = ac[0]; st.accu[c] = ac[1]; st.accv[c] = ac[2];
          }
          complete(f, st, c, n[0], zon, mer);
        }
      }
    }
    __syncthreads();

    if (w + gridDim.x >= nwork) stage_release();  // this CTA's last item is all but done
    // ---- phase 4: ghost push of the part's edge strips ------------------------
    // A cell within `halo` of a panel edge lands in that edge's halo strip (two strips
    // near a panel corner).  The strip cells of the part, strip by strip (0 left, 1
    // right, 2 below, 3 above), are dealt out to all threads.
    if (st.kind != K_TEND) {
      const int h = L.h, ie = i0 + nx - 1, je = j0 + ny - 1;
      const int xlo1 = max(i0, N - h + 1), xlo3 = max(j0, N - h + 1);
      const int o1 = max(min(ie, h) - i0 + 1, 0) * ny;
      const int o2 = o1 + max(ie - xlo1 + 1, 0) * ny;
      const int o3 = o2 + max(min(je, h) - j0 + 1, 0) * nx;
      const int o4 = o3 + max(je - xlo3 + 1, 0) * nx;
      for (int t = tid; t < o4; t += NT) {
        const int sd = (t >= o1) + (t >= o2) + (t >= o3);
        const int q = t - (sd == 0 ? 0 : sd == 1 ? o1 : sd == 2 ? o2 : o3);
        const int na = sd < 2 ? ny : nx;
        const int x = (sd == 0 ? i0 : sd == 1 ? xlo1 : sd == 2 ? j0 : xlo3) + q / na, m = (sd < 2 ? j0 : i0) + q % na;
        const int k = (sd == 0 || sd == 2) ? x : N + 1 - x;
        const int i = sd < 2 ? x : m, j = sd < 2 ? m : x;
        const int64_t e = ((int64_t)p * 4 + sd) * h * N + (int64_t)(k - 1) * N + (m - 1);
        if (!ccs_inb(e, (long long)24 * h * N, 224)) continue;
        const int64_t d = __ldg(st.m.push + e);
        const int cell = (j - j0) * TX + i - i0;
        if (!ccs_inb(d, L.field, 225) || !ccs_inb(cell, T::NC, 226)) continue;
        complete(f, st, d, new_phiG[cell], new_zon[cell], new_mer[cell]);
      }
    }
    __syncthreads();
  }
}

}  // namespace

// test support: out[k] = ccs_div_const(x[k], b, 1/b) next to out[n + k] = x[k] / b
__global__ void div_const_check_kernel(const double *__restrict__ x, int64_t n, double b, double y,
                                       double *__restrict__ out) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    out[k] = ccs_div_const(x[k], b, y);
    out[n + k] = x[k] / b;
  }
}

// test support: out[k] = ccs_div_by(a[k], b[k], 1 / b[k]) next to out[n + k] = a[k] / b[k]
__global__ void div_pairs_check_kernel(const double *__restrict__ a, const double *__restrict__ b, int64_t n,
                                       double *__restrict__ out) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    out[k] = ccs_div_by(a[k], b[k], 1. / b[k]);
    out[n + k] = a[k] / b[k];
  }
}

cudaError_t launch_div_pairs_check(const double *a, const double *b, int64_t n, double *out, cudaStream_t s) {
  div_pairs_check_kernel<<<1024, 256, 0, s>>>(a, b, n, out);
  return cudaGetLastError();
}

// test support: out[k] = what the stage kernel computes with the integer routines, out[n + k]
// = the IEEE operations it stands for (CCS_CHECK_*)
__global__ void integer_check_kernel(int what, const double *__restrict__ a, const double *__restrict__ b, int64_t n,
                                     double *__restrict__ out) {
  using namespace softfp;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const double x = a[k], y = b[k];
    double fast = 0., ieee = 0.;
    switch (what) {
      case CCS_CHECK_MUL: fast = round_double(mul(unpack(x), unpack(y))); ieee = x * y; break;
      case CCS_CHECK_MUL_UNPACKED: fast = pack(round_unp(mul(unpack(x), unpack(y)))); ieee = x * y; break;
      case CCS_CHECK_DIV: fast = round_double(div(unpack(x), divisor(unpack(y)))); ieee = x / y; break;
      case CCS_CHECK_DIV_UNPACKED: fast = pack(round_unp(div(unpack(x), divisor(unpack(y))))); ieee = x / y; break;
      case CCS_CHECK_ONE_PLUS_DIV:
        fast = pack(round_unp(one_plus(div(unpack(x), divisor(unpack(y))))));
        ieee = 1. + x / y;
        break;
      case CCS_CHECK_ADD: fast = pack(round_unp(add(unpack(x), unpack(y)))); ieee = x + y; break;
      case CCS_CHECK_SQRT: fast = square_root(unpack(x)); ieee = sqrt(x); break;
      case CCS_CHECK_CURVATURE: fast = curvature(x); ieee = x * x * 13. / 12.; break;
      case CCS_CHECK_GRID_DIV: {
        Divisor d = divisor(unpack(y));
        if (!(y >= 0x1p-400 && y < 0x1p300)) d.y = 0u;  // (as the host prepares a grid's)
        fast = div_by(x, d, y);
        ieee = x / y;
        break;
      }
      case CCS_CHECK_DIV6: fast = div_by6(x); ieee = x / 6.; break;
      case CCS_CHECK_HALF: fast = half_of(x); ieee = 0.5 * x; break;
    }
    out[k] = fast;
    out[n + k] = ieee;
  }
}

// the same of one whole reconstruction: window k is a[5 k .. 5 k + 4]
__global__ void side_check_kernel(const double *__restrict__ a, int64_t n, F64Ops f, double *__restrict__ out) {
  const int64_t m = n / 5;
  for (int64_t k0 = blockIdx.x * (int64_t)blockDim.x; k0 < m; k0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = k0 + threadIdx.x, w = k < m ? k : m - 1;  // (whole warps, for the votes)
    double Q[5], G[NSING * 5], ga[3];
    for (int q = 0; q < 5; q++) Q[q] = a[5 * w + q];
    for (int q = 0; q < 5; q++) store_singles(f, G + q, 5, Q[q]);
    for (int q = 0; q < 3; q++) ga[q] = curvature(f.add(fma(-2., Q[q + 1], Q[q]), Q[q + 2]));
    const double fast = side(f, Q + 2, 1, G + 2, 5, 1, ga + 1, 1);
    const double ieee = weno5z(Q[0], Q[1], Q[2], Q[3], Q[4]);
    if (k < m) {
      out[k] = fast;
      out[n + k] = ieee;
    }
  }
}

cudaError_t launch_integer_check(int what, const double *a, const double *b, int64_t n, double *out, cudaStream_t s) {
  if (what == CCS_CHECK_RECONSTRUCTION)
    return launch_stage(side_check_kernel, 1024, 256, 0, s, false, a, n, F64Ops{1., -0.}, out);
  return launch_stage(integer_check_kernel, 1024, 256, 0, s, false, what, a, b, n, out);
}

unsigned long long f64_bounds_take() { return bounds_take_tu(); }

cudaError_t launch_div_const_check(const double *x, int64_t n, double b, double *out, cudaStream_t s) {
  div_const_check_kernel<<<1024, 256, 0, s>>>(x, n, b, 1. / b, out);
  return cudaGetLastError();
}

namespace {

// 12 warps and two CTAs an SM (80 registers): the FP64 pipe is shared by the whole SM,
// and a warp holds it for a fraction of its time (C384 stage: 8 warps 1023 us, 12 warps
// 989, 16 warps, which spill, 1032)
using F64T0 = F64Tile<32, 8, 384, 2>;
using F64T1 = F64Tile<16, 16, 384, 2>;
using F64T2 = F64Tile<64, 4, 384, 1>;
// 64 x 4 items of the central operators: the face phases' shared memory leaves room for one
// CTA an SM (the other tiles hold two); without it two fit (fourth-order operator: C384 306 ->
// 243 us a stage, C192 79 -> 67, C96 28.8 -> 24.5; three of 256 threads 256, 65, 26.1)
using F64C2 = F64Tile<64, 4, 384, 2, 64, 4, false>;
// parts of 16 x 8 cells, three CTAs an SM
using F64H0 = F64Tile<16, 8, 288, 3, 32, 8>;
using F64H1 = F64Tile<16, 8, 288, 3, 16, 16>;
// parts of 8 x 8 cells: nine warps hold all its face sides at once
using F64S0 = F64Tile<8, 8, 288, 2, 32, 8>;
using F64S1 = F64Tile<8, 8, 288, 2, 16, 16>;

template <class T>
constexpr int f64_smem_bytes() {
  return (int)sizeof(Smem<T>);
}

template <class T>
int f64_resident() {  // CTAs on an SM
  int per = 0;
  constexpr int smem = f64_smem_bytes<T>();
  cudaFuncSetAttribute(f64_stage_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f64_stage_kernel<T>, T::NT, smem);
  return per < 1 ? 1 : per;
}

template <class T>
int f64_grid_for(int device) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms * f64_resident<T>();
}

template <class T>
StageTile f64_tile_of() {
  return StageTile{T::TX, T::TY, f64_resident<T>()};
}

template <class T>
cudaError_t f64_launch(const F64Stage *d_stages, const WorkItem *d_work, int nwork, int grid, cudaStream_t s,
                       bool chained) {
  constexpr int smem = f64_smem_bytes<T>();
  static std::atomic<uint64_t> attr_done{0};
  const cudaError_t e = smem_attr_once((const void *)f64_stage_kernel<T>, smem, attr_done);
  if (e != cudaSuccess) return e;
  if (grid > nwork) grid = nwork;
  if (grid < 1) return cudaSuccess;
  // chained only with one item a CTA: CTAs that start early spread unevenly over the SMs,
  // which costs more than it saves when some have an item more than others (C384: 921 us a
  // stage unchained, 933 chained; C24 23.6 -> 23.1, C48 30.1 -> 29.5)
  return launch_stage(f64_stage_kernel<T>, grid, T::NT, smem, s, chained && grid == nwork, d_stages, d_work, nwork);
}

// the same work items in parts, one CTA each
template <class T>
cudaError_t f64_launch_parts(const F64Stage *d_stages, const WorkItem *d_work, int nwork, cudaStream_t s,
                             bool chained) {
  const int parts = nwork * T::SX * T::SY;
  return f64_launch<T>(d_stages, d_work, parts, parts, s, chained);
}

static_assert(F64T0::TX == kF64Tiles[0].tx && F64T0::TY == kF64Tiles[0].ty, "tile table");
static_assert(F64T1::TX == kF64Tiles[1].tx && F64T1::TY == kF64Tiles[1].ty, "tile table");
static_assert(F64T2::TX == kF64Tiles[2].tx && F64T2::TY == kF64Tiles[2].ty, "tile table");
static_assert(F64C2::TX == kF64Tiles[2].tx && F64C2::TY == kF64Tiles[2].ty, "tile table");

}  // namespace

int f64_max_grid(int var, bool central, int device) {
  switch (var) {
    case 1: return f64_grid_for<F64T1>(device);
    case 2: return central ? f64_grid_for<F64C2>(device) : f64_grid_for<F64T2>(device);
    default: return f64_grid_for<F64T0>(device);
  }
}

// The 256 cells of an item take one CTA 54 us alone on its SM, and two CTAs 84 us.  Small
// launches therefore run their items in parts, as long as all parts are resident:
//   in four (8 x 8 cells) when there are at most two an SM: C24 61 -> 23 us a stage, C48 61
//   -> 29.5 (C64, with 96 items: 58, in two 49, whole 54)
//   in two (16 x 8 cells) when there are at most three an SM: C64 54 -> 49, C96 84 -> 67
//   (larger grids lose by the halo cells of the parts: C192 245 -> 260, C384 921 -> 985)
// grid: the resident CTAs of whole items, two an SM.  64 x 4 items have no such parts.
static int f64_parts(int var, int nwork, int grid) {
  if (var == 2) return 1;
#ifdef CCS_BOUNDS  // (the checked build reaches all three on small grids)
  return nwork <= 12 ? 4 : nwork <= 24 ? 2 : 1;
#else
  return 4 * nwork <= grid ? 4 : 4 * nwork <= 3 * grid ? 2 : 1;
#endif
}

cudaError_t launch_f64_stage(int var, bool central, const F64Stage *d_stages, const WorkItem *d_work, int nwork,
                             int grid, cudaStream_t s, bool chained) {
  const int parts = f64_parts(var, nwork, grid);
  switch (var) {
    case 1:
      if (parts == 4) return f64_launch_parts<F64S1>(d_stages, d_work, nwork, s, chained);
      if (parts == 2) return f64_launch_parts<F64H1>(d_stages, d_work, nwork, s, chained);
      return f64_launch<F64T1>(d_stages, d_work, nwork, grid, s, chained);
    case 2:
      if (central) return f64_launch<F64C2>(d_stages, d_work, nwork, grid, s, chained);
      return f64_launch<F64T2>(d_stages, d_work, nwork, grid, s, chained);
    default:
      if (parts == 4) return f64_launch_parts<F64S0>(d_stages, d_work, nwork, s, chained);
      if (parts == 2) return f64_launch_parts<F64H0>(d_stages, d_work, nwork, s, chained);
      return f64_launch<F64T0>(d_stages, d_work, nwork, grid, s, chained);
  }
}

StageTile f64_stage_tile(int var, bool central, int nwork, int grid) {
  const int parts = f64_parts(var, nwork, grid);
  if (parts == 4) return f64_tile_of<F64S0>();  // (F64S1 alike; so F64H1)
  if (parts == 2) return f64_tile_of<F64H0>();
  if (var == 2) return central ? f64_tile_of<F64C2>() : f64_tile_of<F64T2>();
  return var == 1 ? f64_tile_of<F64T1>() : f64_tile_of<F64T0>();
}

// Products of static metric terms, each in the order the operator forms it: sqrtG f,
// 1 / sqrtG, and the face means of the wave-speed metric
// (spatial_operators_mod.F90:113-114, 138-139, 171).
__global__ void mesh_products_kernel(Layout L, MeshF64 m, double *__restrict__ out) {
  const int64_t n = (int64_t)L.nh * L.nh * 6;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int ia = (int)(q % L.nh), ja = (int)((q / L.nh) % L.nh), p = (int)(q / ((int64_t)L.nh * L.nh));
    const int64_t c = ia + (int64_t)L.pitch * ja + L.panel * p;
    out[c] = m.sqrtG[c] * m.f[c];
    // (for div_depth)
    const unsigned e = ((unsigned)__double2hiint(m.sqrtG[c]) >> 20) & 0x7ffu;
    out[L.field + c] = e - 623u < 700u ? 1. / m.sqrtG[c] : 0.;
    if (ia + 1 < L.nh) out[2 * L.field + c] = 0.5 * (m.ig11[c + 1] + m.ig11[c]);
    if (ja + 1 < L.nh) out[3 * L.field + c] = 0.5 * (m.ig22[c + L.pitch] + m.ig22[c]);
  }
}

cudaError_t launch_f64_mesh_products(const Layout &L, const MeshF64 &m, double *out, cudaStream_t s) {
  return launch_stage(mesh_products_kernel, 1024, 256, 0, s, false, L, m, out);
}

// ---- diagnostics: calc_total_mass / calc_total_energy (diag_mod.F90:10-53) ------
// Each block sums a contiguous range of interior cells in the reference's order
// (i fastest, then j, then panel); the host adds the block partials in order.
__global__ void f64_diag_kernel(Layout L, const double *__restrict__ phiG, const double *__restrict__ phi,
                                const double *__restrict__ u, const double *__restrict__ v,
                                const double *__restrict__ uC, const double *__restrict__ vC,
                                const double *__restrict__ sqrtG, const double *__restrict__ phis,
                                double *__restrict__ partials) {
  __shared__ double sm[2][256];
  const int64_t ncell = (int64_t)L.N * L.N * 6;
  const int64_t per = (ncell + gridDim.x - 1) / gridDim.x;
  const int64_t beg = blockIdx.x * per;
  int64_t end = beg + per;
  if (end > ncell) end = ncell;
  double m = 0., e = 0.;
  for (int64_t q = beg + threadIdx.x; q < end; q += blockDim.x) {
    const int i = 1 + (int)(q % L.N);
    const int j = 1 + (int)((q / L.N) % L.N);
    const int p = (int)(q / ((int64_t)L.N * L.N));
    const int64_t c = L.idx(i, j, p);
    m += phiG[c];
    const double KE = 0.5 * phi[c] * (u[c] * uC[c] + v[c] * vC[c]);
    const double t = phi[c] + phis[c];
    const double PE = 0.5 * (t * t);
    e += sqrtG[c] * (KE + PE);
  }
  sm[0][threadIdx.x] = m;
  sm[1][threadIdx.x] = e;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      sm[0][threadIdx.x] += sm[0][threadIdx.x + s];
      sm[1][threadIdx.x] += sm[1][threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = sm[0][0];
    partials[2 * blockIdx.x + 1] = sm[1][0];
  }
}

cudaError_t launch_f64_diag(const Layout &L, const double *phiG, const double *phi, const double *u,
                            const double *v, const double *uC, const double *vC, const double *sqrtG,
                            const double *phis, double *partials, int nblocks, cudaStream_t s) {
  f64_diag_kernel<<<nblocks, 256, 0, s>>>(L, phiG, phi, u, v, uC, vC, sqrtG, phis, partials);
  return cudaGetLastError();
}

}  // namespace ccs
