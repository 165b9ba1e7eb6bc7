// FP64 sums, differences and products on the integer pipes, bit for bit what
// the FP64 unit gives (round to nearest even).
//
// Why: GB300 issues one FP64 instruction per warp and scheduler every 65 to
// 70 cycles, an integer instruction every 2.1, and the two overlap.  Measured
// at 2070 MHz, cycles a warp and scheduler: an FP64 FMA 69.5; add() 90,
// addp() 77, addsub() (sum and difference of one pair) 130, mul() 57; three
// FMAs with one addsub() 210 and three with one add() 209, against 208 for
// the three FMAs alone: integer forms are free as long as their cycles stay
// below those of the FP64 instructions beside them.  So a kernel that the
// FP64 unit bounds hands about half of its sums and products to these (never
// its FMAs, whose 106-bit alignment costs more than the FMA).
//
// How: the significands are aligned in 64-bit integers with 10 bits below
// the last place.  The smaller operand is shifted right by the exponents'
// difference d and truncated (floor); bits are lost only when d > 10, and
// matter only if the sum then ends in a rounding tie, so that case is left to
// the FP64 unit, as are denormal, infinite and NaN operands, exponents near
// the ends of the range and cancellations of more than 31 bits.  Each form
// reports those in `bad` (its result is then meaningless) and the caller
// recomputes its cell in FP64: one branch a cell.  A branch at each operation
// would not do: the compiler predicates a lone FP64 instruction, and a
// predicated-off one costs as much as one that runs.  Exact zeros (no-slip
// walls, fluid at rest) stay on the integer path.
//
// Plain C++ apart from the marked instructions, so that a host build of this
// file can be compared with the host's own arithmetic.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SBFS_IF __device__ __forceinline__
#else
#define SBFS_IF inline
#endif

namespace sbfs {

namespace intfp {

using u32 = uint32_t;
using u64 = uint64_t;
using i64 = int64_t;

constexpr u32 kMag = 0x7fffffffu, kSign = 0x80000000u;
constexpr u64 kLead = 0x4000000000000000ull, kFrac = 0x3fffffffffffffffull;

// the words are taken with mov, not through a 64-bit bit cast: the compiler
// turns a masked bit cast into an FP64 |x|
SBFS_IF u64 bits(double x) {
#ifdef __CUDA_ARCH__
  u32 lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
  return ((u64)hi << 32) | lo;
#else
  u64 r;
  std::memcpy(&r, &x, 8);
  return r;
#endif
}
SBFS_IF double from_words(u32 hi, u32 lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const u64 b = ((u64)hi << 32) | lo;
  double r;
  std::memcpy(&r, &b, 8);
  return r;
#endif
}
SBFS_IF u32 high(u64 x) { return (u32)(x >> 32); }
SBFS_IF u32 low(u64 x) { return (u32)x; }

// x >> n and (signed) x >> n for any n: 0 or the sign once n reaches 64
SBFS_IF u64 shr(u64 x, u32 n) {
#ifdef __CUDA_ARCH__
  u64 r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));
  return r;
#else
  return n > 63 ? 0 : x >> n;
#endif
}
SBFS_IF i64 sar(i64 x, u32 n) {
#ifdef __CUDA_ARCH__
  i64 r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));
  return r;
#else
  return x >> (n > 63 ? 63 : n);
#endif
}
SBFS_IF u64 shl(u64 x, u32 n) {
#ifdef __CUDA_ARCH__
  u64 r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));
  return r;
#else
  return n > 63 ? 0 : x << n;
#endif
}
// leading zeros of x != 0
SBFS_IF u32 lead_zeros(u32 x) {
#ifdef __CUDA_ARCH__
  u32 r;
  asm("bfind.shiftamt.u32 %0, %1;" : "=r"(r) : "r"(x));
  return r;
#else
  return (u32)__builtin_clz(x | 1u);
#endif
}
SBFS_IF u64 mul_high(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}

// Significand s with its leading bit at 63 - lz, rounded to 53 bits; head is
// the sign and exponent word of a significand whose leading bit is at 62.
SBFS_IF double round_pack(u64 s, u32 lz, u32 head) {
  const u64 n = shl(s, lz);
  const u64 r = n >> 11;
  const u32 rest = low(n) << 21, inc = 0x7fffffffu + (low(r) & 1u);  // a carry of rest + inc rounds up
  const u32 e = head - (lz << 20);
#ifdef __CUDA_ARCH__
  u32 lo, hi;
  asm("{.reg .u32 x; add.cc.u32 x, %2, %3; addc.cc.u32 %0, %4, 0; addc.u32 %1, %5, %6;}"
      : "=r"(lo), "=r"(hi)
      : "r"(rest), "r"(inc), "r"(low(r)), "r"(high(r)), "r"(e));
  return from_words(hi, lo);
#else
  const u64 q = r + (((u64)rest + inc) >> 32) + ((u64)e << 32);
  return from_words(high(q), low(q));
#endif
}

SBFS_IF u64 significand(u64 x) { return ((x << 10) & kFrac) | kLead; }
SBFS_IF u32 exponent(u32 hi) { return (hi >> 20) & 0x7ffu; }
SBFS_IF u32 exponent_field(u32 hi) { return hi & 0x7ff00000u; }
// exponent fields without room for every shift and carry of a sum
SBFS_IF u32 wide(u32 e) { return e - (70u << 20) >= (1900u << 20); }
// bits of the smaller operand were lost and the sum may end in a tie
SBFS_IF u32 tie(u32 d, u32 lo) { return (u32)(d - 11u < 46u) & (u32)((lo & 0xffu) == 0u); }

// a + b.  ZERO: both may be zero at once
template <bool ZERO>
SBFS_IF double add(double a, double b, u32 &bad) {
  const u64 ua = bits(a), ub = bits(b);
  const u64 kM = 0x7fffffffffffffffull;
  const bool sw = (ua & kM) < (ub & kM);
  const u64 x = sw ? ub : ua, y = sw ? ua : ub;  // |x| >= |y|
  const u32 xh = high(x), yh = high(y);
  const u32 ex = exponent_field(xh), d = (ex - exponent_field(yh)) >> 20;
  i64 Y = (i64)significand(y);
  if ((int32_t)(xh ^ yh) < 0) Y = -Y;
  const i64 Ys = sar(Y, d);
  const u64 S = significand(x) + (u64)Ys;
  const u32 sh = high(S);
  bool zero = S == 0;
  u32 range = wide(ex);
  if (ZERO) {
    const bool none = ((xh & kMag) | low(x)) == 0;
    zero |= none;
    range = none ? 0u : range;
  }
  bad |= range | ((u32)(sh == 0) & (u32)(S != 0)) | tie(d, low((u64)Ys));
  const u64 r = bits(round_pack(S, lead_zeros(sh), xh & 0xfff00000u));
  // a zero sum is -0 only of two -0 (x = -y has one sign of each)
  return from_words(zero ? xh & yh & kSign : high(r), zero ? 0u : low(r));
}
SBFS_IF double negate(double a) {
  const u64 u = bits(a);
  return from_words(high(u) ^ kSign, low(u));
}
template <bool ZERO>
SBFS_IF double sub(double a, double b, u32 &bad) {
  return add<ZERO>(a, negate(b), bad);
}

// a + b of positive normal numbers
SBFS_IF double addp(double a, double b, u32 &bad) {
  const u64 ua = bits(a), ub = bits(b);
  const bool sw = ua < ub;
  const u64 x = sw ? ub : ua, y = sw ? ua : ub;
  const u32 xh = high(x), ex = xh & 0xfff00000u, d = (ex - (high(y) & 0xfff00000u)) >> 20;
  const u64 Ys = shr(significand(y), d);
  const u64 S = significand(x) + Ys;
  bad |= wide(ex);  // also any negative operand: its word is the larger
  bad |= tie(d, low(Ys));
  return round_pack(S, 1u - (high(S) >> 31), ex);
}

// s = a + b and t = a - b.  ZERO: both may be zero at once.  STICKY: the lost
// bits are kept as one bit that breaks ties, three instructions more than
// giving those sums up, for operands whose magnitudes are often far apart
// (a transform's: one pair in 256 of those would be given up)
template <bool ZERO, bool STICKY = false>
SBFS_IF void addsub(double a, double b, double &s, double &t, u32 &bad) {
  const u64 ua = bits(a), ub = bits(b);
  const u64 kM = 0x7fffffffffffffffull;
  const bool sw = (ua & kM) < (ub & kM);
  const u64 x = sw ? ub : ua, y = sw ? ua : ub;  // |x| >= |y|
  const u32 xh = high(x), yh = high(y);
  const u32 ex = exponent_field(xh), d = (ex - exponent_field(yh)) >> 20;
  const u64 X = significand(x), Y = significand(y);
  u64 Ys = shr(Y, d);
  if (STICKY) {
    const u64 lost = shl(Y, 64u - d);  // none when d = 0, and any does when d > 63
    Ys |= (low(lost) | high(lost)) != 0 ? 1u : 0u;
  }
  const u64 S = X + Ys, D = X - Ys;
  const u32 dh = high(D);
  const bool none = ZERO && ((xh & kMag) | low(x)) == 0;
  const u32 range = none ? (xh | yh) >> 31 : wide(ex);  // of zeros only two +0
  bad |= range | ((u32)(dh == 0) & (u32)(D != 0));
  if (!STICKY) bad |= tie(d, low(Ys));
  const u32 head = xh & 0xfff00000u;
  const u64 p = bits(round_pack(S, 1u - (high(S) >> 31), head));    // the sum of the magnitudes
  const u64 q = bits(round_pack(D, lead_zeros(dh), head));          // their difference
  const u32 ph = none ? 0u : high(p), pl = none ? 0u : low(p);
  const bool qz = D == 0;
  const bool same = (int32_t)(xh ^ yh) >= 0;
  // a - b = -(b - a) where they were swapped; an exact zero difference is +0
  const u32 flip = sw ? kSign : 0u;
  const u32 qh = qz ? 0u : high(q), ql = qz ? 0u : low(q);
  s = from_words(same ? ph : qh, same ? pl : ql);
  t = from_words(same ? (qz ? 0u : qh ^ flip) : ph ^ flip, same ? ql : pl);
}

// a b; |a| lies between 2^-256 and 2^256, and so does |b|, or (ZERO) |b|
// between 2^-763 and 2^737 and either may be zero
template <bool ZERO>
SBFS_IF double mul(double a, double b, u32 &bad) {
  const u64 ua = bits(a), ub = bits(b);
  const u32 ah = high(ua), bh = high(ub);
  const u32 ea = exponent(ah), eb = exponent(bh);
  const u64 A = (ua << 11) | 0x8000000000000000ull, B = (ub << 11) | 0x8000000000000000ull;
  u64 h = mul_high(A, B);
  h |= (u64)(A * B != 0);  // what is below only breaks ties
  const u32 head = ((ah ^ bh) & kSign) + ((ea + eb - 1023u) << 20);
  const u64 r = bits(round_pack(h, 1u - (high(h) >> 31), head));
  if (!ZERO) {
    bad |= (u32)(((ea - 767u) | (eb - 767u)) >= 512u);
    return from_words(high(r), low(r));
  }
  const bool za = ((ah & kMag) | low(ua)) == 0, zb = ((bh & kMag) | low(ub)) == 0;
  bad |= ((u32)!za & (u32)(ea - 767u >= 512u)) | ((u32)!zb & (u32)(eb - 260u >= 1500u));
  const bool z = za | zb;
  return from_words(z ? (ah ^ bh) & kSign : high(r), z ? 0u : low(r));
}

}  // namespace intfp

}  // namespace sbfs
