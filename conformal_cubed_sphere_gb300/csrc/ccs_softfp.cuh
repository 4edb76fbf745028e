// ccs_softfp.cuh -- IEEE double arithmetic on the integer pipes.
//
// GB300 retires two FP64 lanes per SM and cycle, so one FP64 warp instruction holds
// the FP64 pipe for 16 cycles, in which the SM can issue 64 other warp instructions.
// The FP64 lane is bound by that pipe, and a correctly rounded quotient costs it
// about eight instructions (128 cycles) but only some 45 integer ones (about 20
// cycles of the integer pipes).  The routines here compute the round-to-nearest-even
// results of IEEE operations on positive normal operands in integers, bit for bit.
//
// An unpacked number is m 2^(e - 1023 - 63): m has bit 63 set and its low 11 bits
// clear (53 significant bits), e is the biased exponent of the leading bit.  No
// routine handles overflow, underflow, infinities or NaNs: the caller keeps its
// operands in a window of exponents in which none can occur.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define SF_HD __host__ __device__ __forceinline__
#else
#define SF_HD inline
#endif

namespace ccs {
namespace softfp {

struct Unp {
  uint64_t m;
  int e;
};

SF_HD uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
SF_HD uint32_t lo32(uint64_t x) { return (uint32_t)x; }
SF_HD uint64_t mk64(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }
SF_HD uint64_t wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }  // one IMAD.WIDE
SF_HD uint32_t mulhi(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
SF_HD int32_t mulhi_s(int32_t a, int32_t b) {
#if defined(__CUDA_ARCH__)
  return __mulhi(a, b);
#else
  return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
SF_HD uint64_t bits_of(double x) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}
SF_HD double from_bits(uint64_t u) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)u);
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}
// an approximate reciprocal of the float with bits u (in [1, 2)), as its bits; the
// callers allow a relative error of 2^-22
SF_HD uint32_t rcp_bits(uint32_t u) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(u)));
  return __float_as_uint(r);
#else
  float f;
  std::memcpy(&f, &u, 4);
  f = 1.0f / f;
  std::memcpy(&u, &f, 4);
#ifdef SF_RCP_PERTURB  // host test: the worst approximations the device may return
  u += (uint32_t)(SF_RCP_PERTURB);
#endif
  return u;
#endif
}

// |x| of a normal x
SF_HD Unp unpack(double x) {
  const uint64_t b = bits_of(x);
  return Unp{(b << 11) | 0x8000000000000000ull, (int)((hi32(b) >> 20) & 0x7ff)};
}
SF_HD double pack(Unp a) {
  // the leading bit adds one to the exponent field
  return from_bits((a.m >> 11) + ((uint64_t)(uint32_t)(a.e - 1) << 52));
}

// Rounds x, whose leading bit is bit 63 - lead (lead = 0 or 1) and whose bits below
// the lowest are folded into it (sticky), to 53 bits.
SF_HD Unp round_top(uint64_t x, int e) {
  const bool low = (int64_t)x >= 0;
  if (low) x <<= 1;
  e -= low ? 1 : 0;
  const uint32_t odd = (lo32(x) >> 11) & 1u;
  const uint64_t r = x + (0x3ffu + odd);
  const bool carry = r < x;  // rounded up to the next power of two
  return Unp{carry ? 0x8000000000000000ull : (r & ~0x7ffull), e + (carry ? 1 : 0)};
}

// RN(a b), the exponent of a 2^63-scaled pair: e = ea + eb - 1023 (+ 1)
SF_HD Unp mul(Unp a, uint64_t bm, int be) {
  const uint32_t ah = hi32(a.m), al = lo32(a.m), bh = hi32(bm), bl = lo32(bm);
  const uint64_t p0 = wide(al, bl);
  const uint64_t p1 = wide(ah, bl) + hi32(p0);
  const uint64_t p2 = wide(al, bh) + lo32(p1);
  uint64_t x = wide(ah, bh) + hi32(p1) + hi32(p2);
  x |= (lo32(p2) | lo32(p0)) != 0u ? 1u : 0u;
  return round_top(x, a.e + be - 1022);
}
SF_HD Unp mul(Unp a, Unp b) { return mul(a, b.m, b.e); }

// x >> n (n >= 0) with the bits shifted out folded into the lowest bit
SF_HD uint64_t shift_jam(uint64_t x, int n) {
  const int k = n < 63 ? n : 63;
  const uint64_t y = x >> k;
  return y | ((y << k) != x ? 1u : 0u);
}

// RN(1 + a)
SF_HD Unp one_plus(Unp a) {
  const int d = a.e - 1023;
  const uint64_t one = 0x4000000000000000ull, am = a.m >> 1;  // scaled to bit 62
  const bool less = d < 0;
  const uint64_t big = less ? one : am, small = less ? am : one;
  return round_top(big + shift_jam(small, less ? -d : d), (less ? 1023 : a.e) + 1);
}

// RN(a + b) of two positive numbers
SF_HD Unp add(Unp a, Unp b) {
  const bool sw = b.e > a.e;
  const uint64_t big = (sw ? b.m : a.m) >> 1, small = (sw ? a.m : b.m) >> 1;
  const int d = sw ? b.e - a.e : a.e - b.e;
  return round_top(big + shift_jam(small, d), (sw ? b.e : a.e) + 1);
}

// A divisor b = B 2^.. prepared for several quotients: B = b.m >> 11 (53 bits),
// y <= 2^63 / (b.m 2^-32) its 32-bit reciprocal, below the true one by at most 8.
struct Divisor {
  uint64_t nB;  // -B
  uint32_t y;
  int e;
};

SF_HD Divisor divisor(Unp b) {
  Divisor d;
  const uint32_t bh = hi32(b.m);  // b / 2^e in [1, 2) is bh 2^-31 (cut to 32 bits)
  // y24 = y 2^24 < 2^24, y the reciprocal of the leading 24 bits plus two units (so
  // that y < 1 even for b = 1): relative error below 2^-20
  const uint32_t y24 = rcp_bits(0x3f800002u + ((bh >> 8) & 0x7fffffu)) - 0x3e800000u;
  // one Newton step: y32 = y24 2^8 (1 + (2^55 - bh y24) 2^-55)
  const int64_t dl = (int64_t)(0x0080000000000000ull - wide(bh, y24));  // |dl| < 2^35
  const int32_t t = mulhi_s((int32_t)(y24 << 7), (int32_t)(dl >> 4));   // y24 dl 2^-29
  d.y = (y24 << 8) + (uint32_t)(t >> 18) - 6u;
  d.nB = 0ull - (b.m >> 11);
  d.e = b.e;
  return d;
}

// RN(a / b).  Two quotient digits, each from the 32-bit reciprocal, which never
// exceeds the true one: the partial remainders stay non-negative, and the quotient
// cut to 54 binary places (q 2^54, q in (1/2, 2)) is at most one too small before the
// last comparison.  A quotient of two 53-bit numbers is never half-way between two
// 53-bit numbers, so adding half a unit and cutting rounds it to nearest.
SF_HD Unp div(Unp a, Divisor d) {
  const uint64_t A = a.m >> 11;
  const uint32_t nl = lo32(d.nB), nh = hi32(d.nB);
  const uint32_t q1 = mulhi(hi32(a.m), d.y);  // q 2^31, short by less than 32
  uint64_t r = (A << 31) + wide(q1, nl);
  r = mk64(hi32(r) + q1 * nh, lo32(r));  // A 2^31 - q1 B  (mod 2^64), in [0, 2^58)
  const uint32_t q2 = mulhi((uint32_t)(r >> 26), d.y) >> 3;  // r 2^23 / B, short by less than 2
  uint64_t s = (r << 23) + wide(q2, nl);
  s = mk64(hi32(s) + q2 * nh, lo32(s));  // r 2^23 - q2 B, in [0, 2 B)
  uint64_t q = wide(q1, 1u << 23) + q2;
  q += (int64_t)(s + d.nB) >= 0 ? 1u : 0u;
  const bool ge1 = (hi32(q) & (1u << 22)) != 0u;  // q >= 2^54
  const uint64_t x = ge1 ? q << 9 : q << 10;
  return Unp{(x + 0x400u) & ~0x7ffull, a.e - d.e + (ge1 ? 1023 : 1022)};
}

// RN(a / 3): 8 M / 3 (M = a.m >> 11) in two 28-bit digits, cut.  No a / 3 is half-way
// between two 53-bit numbers (3 (2 n + 1) is odd), so adding half a unit and cutting
// rounds it to nearest; it never reaches the next power of two.
SF_HD Unp div3(Unp a) {
  const uint32_t xh = hi32(a.m) >> 4, xl = lo32(a.m >> 8) & 0x0fffffffu;  // 8 M = xh 2^28 + xl
  const uint32_t qh = mulhi(xh, 0xaaaaaaabu) >> 1;
  const uint32_t ql = mulhi(((xh - 3u * qh) << 28) + xl, 0xaaaaaaabu) >> 1;
  const uint64_t q = wide(qh, 1u << 28) + ql;      // in [2^53, 2^55)
  const bool big = (hi32(q) & (1u << 22)) != 0u;   // M >= 3 2^51
  const uint64_t x = big ? q << 9 : q << 10;
  return Unp{(x + 0x400u) & ~0x7ffull, a.e - (big ? 1 : 2)};
}

// RN(13 a)
SF_HD Unp mul13(Unp a) { return round_top((a.m >> 11) * (13u << 7), a.e + 4); }

}  // namespace softfp
}  // namespace ccs
