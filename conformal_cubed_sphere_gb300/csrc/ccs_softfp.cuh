// ccs_softfp.cuh -- IEEE double arithmetic on the integer pipes.
//
// GB300 retires two FP64 lanes per SM and cycle, so one FP64 warp instruction holds
// the FP64 pipe for 16 cycles, in which the SM can issue 64 other warp instructions.
// The FP64 lane is bound by that pipe, and a correctly rounded quotient costs it
// about eight instructions (128 cycles) but only some 45 integer ones (about 20
// cycles of the integer pipes).  The routines here compute the round-to-nearest-even
// results of IEEE operations on positive normal operands in integers, bit for bit.
//
// An unpacked number is (h 2^21 + l) 2^(e - 1023 - 52): 53 significant bits, the upper
// 32 in h (bit 31 set) and the lower 21 in l, and the biased exponent e of the leading
// bit.  No routine handles overflow, underflow, infinities or NaNs: the caller keeps
// its operands in a window of exponents in which none can occur.
//
// An ALU and an IMAD warp instruction take half a cycle of an SM each, IMAD.HI a whole
// one, so the routines spread over both pipes: normalising shifts are multiplications.
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
  uint32_t h, l;
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

// an approximate reciprocal square root of the float with bits u (in [1, 4)), as its
// bits; the callers allow a relative error of 2^-21
SF_HD uint32_t rsqrt_bits(uint32_t u) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(u)));
  return __float_as_uint(r);
#else
  float f;
  std::memcpy(&f, &u, 4);
  f = (float)(1.0 / __builtin_sqrt((double)f));
  std::memcpy(&u, &f, 4);
#ifdef SF_RCP_PERTURB
  u += (uint32_t)(SF_RCP_PERTURB);
#endif
  return u;
#endif
}

// (lo, hi) >> n of a 64-bit pair, low word (0 < n < 32)
SF_HD uint32_t funnel_r(uint32_t lo, uint32_t hi, int n) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(lo, hi, n);
#else
  return (lo >> n) | (hi << (32 - n));
#endif
}
// a + b of 64-bit pairs: the sum's words and the carry out
SF_HD uint32_t add_carry(uint32_t &hi, uint32_t &lo, uint32_t bh, uint32_t bl) {
#if defined(__CUDA_ARCH__)
  uint32_t c;
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, 0, 0;"
      : "+r"(lo), "+r"(hi), "=r"(c)
      : "r"(bl), "r"(bh));
  return c;
#else
  const uint64_t x = mk64(hi, lo), y = x + mk64(bh, bl);
  hi = hi32(y);
  lo = lo32(y);
  return y < x ? 1u : 0u;
#endif
}

// q + 1 if x >= -nB (x < 2^63), else q
SF_HD uint32_t add_if_ge(uint32_t q, uint64_t x, uint64_t nB) {
#if defined(__CUDA_ARCH__)
  asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %1, %3;\n\taddc.cc.u32 t, %2, %4;\n\taddc.u32 %0, %0, 0;\n\t}"
      : "+r"(q)
      : "r"(lo32(x)), "r"(hi32(x)), "r"(lo32(nB)), "r"(hi32(nB)));
  return q;
#else
  return q + (x + nB < x ? 1u : 0u);
#endif
}

// |x| of a normal x
SF_HD Unp unpack(double x) {
  const uint64_t b = bits_of(x);
  return Unp{funnel_r(lo32(b), hi32(b), 21) | 0x80000000u, lo32(b) & 0x1fffffu, (int)((hi32(b) >> 20) & 0x7ffu)};
}
// the same of a constant, folded by the compiler
SF_HD constexpr Unp constant(double x) {
  int e = 1023;
  while (x >= 2.) { x *= 0.5; e++; }
  while (x < 1.) { x *= 2.; e--; }
  const uint64_t m = (uint64_t)(x * 4503599627370496.);
  return Unp{(uint32_t)(m >> 21), (uint32_t)m & 0x1fffffu, e};
}
SF_HD double pack(Unp a) {
  // the leading bit adds one to the exponent field
  return from_bits(mk64((a.h >> 11) + ((uint32_t)(a.e - 1) << 20), (a.h << 21) + a.l));
}

// A positive number before rounding: x 2^.. with its leading bit at bit 63 (its exponent
// is e) or at bit 62 (e - 1), and `tail` not zero where bits follow below x.
struct Wide {
  uint64_t x;
  uint32_t tail;
  int e;
};

// Moves the leading bit to bit 63 and adds half a unit of the 53rd bit (less one unit of
// x for an even number with no tail, so that a tie goes to even).  Returns the carry.
SF_HD uint32_t round_up(Wide &w, uint32_t &hi, uint32_t &lo, uint32_t top) {
  const uint32_t k = 2u - (hi32(w.x) >> 31);
  w.e -= (int)(k - 1u);
  const uint64_t r = wide(lo32(w.x), k);
  lo = lo32(r);
  hi = hi32(w.x) * k + hi32(r);
  const uint32_t half = ((lo & 0x800u) | w.tail) != 0u ? 0x400u : 0x3ffu;
  return add_carry(hi, lo, top, half);
}
SF_HD Unp round_unp(Wide w) {
  uint32_t hi, lo;
  const uint32_t c = round_up(w, hi, lo, 0u);  // a carry leaves zero: the next power of two
  return Unp{hi + (c << 31), lo >> 11, w.e + (int)c};
}
SF_HD double round_double(Wide w) {
  uint32_t hi, lo;
  // without its leading bit, so that a carry lands in the exponent field
  round_up(w, hi, lo, 0x80000000u);
  return from_bits(mk64((hi >> 11) + ((uint32_t)w.e << 20), funnel_r(lo, hi, 11)));
}

// a b
SF_HD Wide mul(Unp a, Unp b) {
  const uint64_t ll = wide(a.l, b.l);  // 42 bits
  const uint64_t c = wide(a.h, b.l) + (wide(a.l, b.h) + (uint32_t)(ll >> 21));
  return Wide{wide(a.h, b.h) + (c >> 21), (lo32(c) | lo32(ll)) & 0x1fffffu, a.e + b.e - 1022};
}
// 13 a: 2^7 13 (h 2^21 + l)
SF_HD Wide mul13(Unp a) { return Wide{wide(a.h, 13u << 28) + a.l * (13u << 7), 0u, a.e + 4}; }

// a + b of the numbers big 2^(e - 62) and small 2^(e - 62 - n), both with leading bit 62
SF_HD Wide add_aligned(uint64_t big, uint64_t small, int n, int e) {
  const int k = n < 63 ? n : 63;
  const uint64_t y = small >> k, back = (y << k) ^ small;
  return Wide{big + y, lo32(back) | hi32(back), e + 1};
}
SF_HD uint64_t at62(Unp a) { return mk64(a.h >> 1, (a.h << 31) + (a.l << 10)); }
// 1 + a
SF_HD Wide one_plus(Unp a) {
  const int d = a.e - 1023;
  const uint64_t one = 0x4000000000000000ull, m = at62(a);
  return d < 0 ? add_aligned(one, m, -d, 1023) : add_aligned(m, one, d, a.e);
}
// a + b
SF_HD Wide add(Unp a, Unp b) {
  const int d = a.e - b.e;
  const uint64_t ma = at62(a), mb = at62(b);
  return add_aligned(d < 0 ? mb : ma, d < 0 ? ma : mb, d < 0 ? -d : d, d < 0 ? b.e : a.e);
}

// A divisor B = h 2^21 + l (53 bits) prepared for several quotients: y its 32-bit
// reciprocal, 2^63 / h to the 32nd bit, never above 2^84 / B and below it by at most 9.
struct Divisor {
  uint64_t nB;  // -B
  uint32_t y;
  int e;
};

SF_HD Divisor divisor(Unp b) {
  Divisor d;
  // y24 = y 2^24 < 2^24, y the reciprocal of the leading 24 bits plus two units (so
  // that y < 1 even for b = 1): relative error below 2^-20
  const uint32_t y24 = rcp_bits(0x3f800002u + ((b.h >> 8) & 0x7fffffu)) - 0x3e800000u;
  // one Newton step: y = y24 2^8 (1 + (2^55 - h y24) 2^-55)
  const int64_t dl = (int64_t)(0x0080000000000000ull - wide(b.h, y24));  // |dl| < 2^35
  const int32_t t = mulhi_s((int32_t)(y24 << 7), (int32_t)(dl >> 4));    // y24 dl 2^-29
  d.y = (y24 << 8) + (uint32_t)(t >> 18) - 6u;
  d.nB = 0ull - (wide(b.h, 1u << 21) + b.l);
  d.e = b.e;
  return d;
}

// The quotient A / B of two 53-bit numbers, 2^54 times, cut: two digits, each from the
// 32-bit reciprocal, which never exceeds the true one, so the partial remainders stay
// non-negative, and one comparison (the digits are together at most one too small).
SF_HD uint64_t quotient54(Unp a, Divisor d) {
  const uint32_t nl = lo32(d.nB), nh = hi32(d.nB);
  const uint32_t q1 = mulhi(a.h, d.y);  // A / B 2^31, short by less than 20
  // A 2^31 - q1 B (mod 2^64), in [0, 2^58)
  uint64_t r = wide(q1, nl) + mk64((a.h << 20) + (a.l >> 1), a.l << 31);
  r = mk64(hi32(r) + q1 * nh, lo32(r));
  const uint32_t q2 = mulhi((uint32_t)(r >> 26), d.y) >> 3;  // r 2^23 / B, short by less than 2
  uint64_t s = wide(q2, nl) + (r << 23);
  s = mk64(hi32(s) + q2 * nh, lo32(s));  // r 2^23 - q2 B, in [0, 2 B)
  return wide(q1, 1u << 23) + add_if_ge(q2, s, d.nB);
}

// The 54- or 55-bit quotients above to 53 bits.  A quotient of two 53-bit numbers, or of
// one by 3, is never half-way between two 53-bit numbers, so adding half a unit of the
// last place and cutting rounds it to nearest; it never reaches the next power of two.
// e: the exponent of a 54-bit one.
struct Quot {
  uint64_t q;
  int e;
};
SF_HD Unp round_unp(Quot a) {
  const uint32_t one = hi32(a.q) >> 22;  // 55 bits
  const uint64_t x = a.q + (1u + one);
  const int n = 1 + (int)one;
  return Unp{(uint32_t)(x >> (21 + n)), (uint32_t)(x >> n) & 0x1fffffu, a.e + (int)one};
}
SF_HD double round_double(Quot a) {
  const uint32_t one = hi32(a.q) >> 22;
  const uint64_t x = (a.q + (1u + one)) >> (1 + one);
  return from_bits(mk64(hi32(x) + ((uint32_t)(a.e - 1) << 20) + (one << 20), lo32(x)));
}
// a / b
SF_HD Quot div(Unp a, Divisor d) { return Quot{quotient54(a, d), a.e - d.e + 1022}; }

// a / 3: 8 A / 3 in two 28-bit digits
SF_HD Quot div3(Unp a) {
  const uint32_t xh = a.h >> 4, xl = ((a.h & 15u) << 24) + (a.l << 3);  // 8 A = xh 2^28 + xl
  const uint32_t qh = mulhi(xh, 0xaaaaaaabu) >> 1;
  const uint32_t ql = mulhi(((xh - 3u * qh) << 28) + xl, 0xaaaaaaabu) >> 1;
  return Quot{wide(qh, 1u << 28) + ql, a.e - 2};
}

// 1 + a, a rounded first
SF_HD Wide one_plus(Quot a) {
  const uint32_t one = hi32(a.q) >> 22;
  const uint64_t x = a.q + (1u + one);
  const uint32_t k = 512u - 256u * one;  // the leading bit to bit 62
  const uint64_t lo = wide(lo32(x), k);
  const uint64_t m = mk64(hi32(x) * k + hi32(lo), lo32(lo) & ~0x3ffu);
  const int e = a.e + (int)one, d = e - 1023;
  const uint64_t unit = 0x4000000000000000ull;
  return d < 0 ? add_aligned(unit, m, -d, 1023) : add_aligned(m, unit, d, e);
}

// RN(sqrt(a)), x = a 2^-2k in [1, 4): the first 32 bits from a 32-bit reciprocal square
// root (off by at most 20), the other 22 from the remainder, and one comparison.  No
// square root of a 53-bit number is half-way between two, so adding half a unit and
// cutting rounds it to nearest.
SF_HD double square_root(Unp a) {
  const uint32_t odd = (uint32_t)(a.e & 1) ^ 1u;  // e - 1023 odd
  const uint64_t X = mk64(a.h, a.l << 11) >> (1u - odd);  // x 2^62
  const uint32_t xh = hi32(X);                            // x 2^30, cut
  // y24 = 2^24 / sqrt(x) < 2^24 from the leading 24 bits plus six units, relative error
  // below 2^-20; one Newton step y (1 + (1 - x y^2) / 2)
  const uint32_t y24 = rsqrt_bits(0x3f800006u + ((odd << 23) + ((a.h >> 8) & 0x7fffffu))) - 0x3e800000u;
  const uint32_t u = mulhi(xh, (uint32_t)(wide(y24, y24) >> 16));                   // x y^2 2^30
  const int32_t t = mulhi_s((int32_t)(y24 << 7), (int32_t)((0x40000000u - u) << 8));  // y (1 - x y^2) 2^37
  const uint32_t y = (y24 << 8) + (uint32_t)(t >> 6) - 6u;                          // 2^32 / sqrt(x)
  const uint32_t s1 = mulhi(xh, y) << 1;                                            // sqrt(x) 2^31
  const int64_t r = (int64_t)(X - wide(s1, s1));                                    // |x 2^62 - s1^2| < 2^38
  const int32_t s2 = (mulhi_s((int32_t)(r >> 7), (int32_t)(y >> 1)) - 2) >> 2;      // r y 2^-10 less a half
  uint64_t s = wide(s1, 1u << 22) + (uint64_t)(int64_t)s2;  // sqrt(x) 2^53, cut, or one less
  const uint64_t sq = wide(lo32(s), lo32(s));
  // x 2^106 - s^2 (mod 2^64) against 2 s + 1, the distance of the next square
  const uint64_t rem = (X << 44) - mk64(hi32(sq) + 2u * lo32(s) * hi32(s), lo32(sq));
  s = (s + 1u + (rem >= 2u * s + 1u ? 1u : 0u)) >> 1;
  return from_bits(s + ((uint64_t)(uint32_t)(((a.e - (int)odd - 1023) >> 1) + 1022) << 52));
}

}  // namespace softfp
}  // namespace ccs
