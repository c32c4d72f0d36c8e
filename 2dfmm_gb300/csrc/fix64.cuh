// FP64-grade arithmetic on the integer pipes.
//
// An FP64 warp instruction takes a GB300 SM sub-partition 64 cycles, a
// 32 x 32 -> 64-bit multiply-add or a 64-bit add 2 (measured with independent
// chains, 8 warps per sub-partition).  The plain treecode's two inner terms,
// the multipole sum and the regularised pair, are therefore formed in 64-bit
// fixed point with explicit exponents: about 58 significant bits through
// every step (FP64 has 53), and their sums held in 96.  FP64 stays for the two
// coordinate differences, which are exact for close pairs, and for what the
// fixed units would not hold as well: cells whose leading coefficients cancel
// or leave FP64's normal range, targets far outside the blobs.
//
// A mantissa "with its leading one at bit b" lies in [2^b, 2^(b+1)); biased
// exponents are a double's exponent field.  mulhi() leaves out the product of
// the low halves and truncates (an error below 2 units of its result).  The
// host compiles the same code (the tests compare it with exact arithmetic);
// only the reciprocal's FP32 seed differs there.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define T2D_HD __host__ __device__ __forceinline__
#else
#define T2D_HD inline
#endif

namespace t2d {
namespace fix {

T2D_HD uint64_t bits(double d) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(d);
#else
  uint64_t u;
  std::memcpy(&u, &d, 8);
  return u;
#endif
}
T2D_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double d;
  std::memcpy(&d, &u, 8);
  return d;
#endif
}
// v >> s for any s >= 0 (0 from 64 on)
T2D_HD uint64_t shr(uint64_t v, int s) {
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
#else
  return s > 63 ? 0 : v >> s;
#endif
}
T2D_HD int clz(uint64_t v) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}
T2D_HD int clz32(uint32_t v) {
#ifdef __CUDA_ARCH__
  return __clz((int)v);
#else
  return v ? __builtin_clz(v) : 32;
#endif
}
// a b and a b + c with 32-bit factors and a 64-bit result, unsigned and
// signed: one instruction each on the device (left to itself the compiler
// may widen the factors first and multiply 64 by 64 bits).
T2D_HD uint64_t wide(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("mul.wide.u32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
#else
  return (uint64_t)a * b;
#endif
}
T2D_HD uint64_t wide(uint32_t a, uint32_t b, uint64_t c) {
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (uint64_t)a * b + c;
#endif
}
T2D_HD int64_t swide(int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
#else
  return (int64_t)a * b;
#endif
}
T2D_HD int64_t swide(int32_t a, int32_t b, int64_t c) {
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (int64_t)a * b + c;
#endif
}
T2D_HD uint32_t hi32(uint64_t v) { return (uint32_t)(v >> 32); }

// The number 1 where the compiler cannot see it: hi32(c) times it plus a
// 64-bit number is one instruction, where a sum of a zero- or sign-extended
// half takes two or three.
struct One {
  int32_t v = 1;
};

// High 64 bits of a b for a, b < 2^63.
T2D_HD uint64_t mulhi(uint64_t a, uint64_t b, One one) {
  const uint64_t c = wide(hi32(a), (uint32_t)b, wide((uint32_t)a, hi32(b)));
  return wide(hi32(c), (uint32_t)one.v, wide(hi32(a), hi32(b)));
}

// A signed 64-bit number as hi 2^32 + lo with both halves signed.
struct Limbs {
  int32_t h, l;
};
T2D_HD Limbs limbs(int64_t v) {
  Limbs r;
  r.l = (int32_t)v;
  r.h = (int32_t)hi32((uint64_t)v) + (int32_t)((uint32_t)v >> 31);
  return r;
}

// (dx, dy) as mantissas of one exponent, |dx| = mx 2^(e - 1085), the larger
// with its leading one at bit 62 (for |d|^2: the smaller one loses bits), and
// their bits.  A zero's mantissa is the implicit bit of exponent field 0, far
// below any other value.
struct Vec {
  uint64_t mx, my;
  int e;
  uint64_t ux, uy;
};
T2D_HD Vec vec(double dx, double dy) {
  const uint64_t ux = bits(dx), uy = bits(dy);
  const int ex = (int)(ux >> 52) & 0x7ff, ey = (int)(uy >> 52) & 0x7ff;
  Vec v;
  v.e = ex > ey ? ex : ey;
  v.mx = shr(((ux << 10) & 0x3fffffffffffffffull) | 0x4000000000000000ull, v.e - ex);
  v.my = shr(((uy << 10) & 0x3fffffffffffffffull) | 0x4000000000000000ull, v.e - ey);
  v.ux = ux;
  v.uy = uy;
  return v;
}

// |d|^2 = norm2(v) 2^(2 e - 2106), in [2^60, 2^63).
T2D_HD uint64_t norm2(const Vec &v, One one) {
  const uint32_t xh = hi32(v.mx), yh = hi32(v.my);
  const uint64_t c = wide(xh, (uint32_t)v.mx, wide(yh, (uint32_t)v.my));
  return wide(hi32(c), 2u * (uint32_t)one.v, wide(xh, xh, wide(yh, yh)));
}

// 2^123 / m for m in [2^60, 2^63), below 2^63: an FP32 reciprocal of the
// upper half, then one third-order Newton step (y <- y + y (e + e^2), e the
// residual 1 - m y) in fixed point.
T2D_HD uint64_t recip(uint64_t m, One one) {
  const uint32_t h = hi32(m);
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint2float_rn(h)));
  const uint32_t y0 = __float2uint_rz(y * 0x1.fffffep58f);  // below 2^31
#else
  const uint32_t y0 = (uint32_t)(1.0f / (float)h * 0x1.fffffep58f);
#endif
  // m y0 / 2^32 = 2^59 (1 - e), |e| < 2^-21; r = e + e^2 in units of 2^-59
  const uint64_t p = wide(hi32(wide((uint32_t)m, y0)), (uint32_t)one.v, wide(h, y0));
  int64_t r = (int64_t)((1ull << 59) - 2 - p);  // 2: below 2^123 / m for sure
  const int32_t s = (int32_t)(r >> 7);
  r = swide((int32_t)(hi32((uint64_t)swide(s, s)) >> 13), one.v, r);
  // y0 2^32 (1 + r 2^-59): y0 (r 2^25) as a signed high and an unsigned low half
  const uint64_t q = (uint64_t)r << 25;
  const int64_t c = swide((int32_t)hi32(q), (int32_t)y0, (int64_t)hi32(wide((uint32_t)q, y0)));
  return ((uint64_t)y0 << 32) + (uint64_t)(c >> 20);
}

// m 2^(e - 1075 - 10) to the nearest double (ties up), for m < 2^63 and e the
// exponent field of a double with its leading one at m's bit 62; `sign` is
// its sign bit.  Infinity on overflow.
T2D_HD double pack(uint64_t m, int e, uint64_t sign) {
  const int z = clz(m);
  e += 1 - z;
  m = m << (z & 63);  // leading one at bit 63
  uint64_t u = ((uint64_t)(uint32_t)(e - 1) << 52) + (m >> 11) + ((m >> 10) & 1);
  if (e <= 0) {  // subnormal
    const uint64_t h = shr(m, 11 - e);
    u = (h >> 1) + (h & 1);
  }
  if (z == 64) u = 0;
  if (e > 0x7fe && z < 64) u = 0x7ff0000000000000ull;
  return from_bits(u | sign);
}

// A double as a mantissa with its leading one at bit 62 and the exponent
// field that goes with it (subnormals normalised, the field then <= 0; zero
// gives a zero mantissa).  Infinities keep field 0x7ff.
T2D_HD uint64_t mantissa(double d, int &e) {
  const uint64_t u = bits(d) & 0x7fffffffffffffffull;
  e = (int)(u >> 52);
  if (e) return ((u << 10) & 0x3fffffffffffffffull) | 0x4000000000000000ull;
  if (!u) return 0;
  const int z = clz(u);
  e = 12 - z;
  return u << (z - 1);
}

// ------------------------------------------------------------------ sums
// A running sum of two components, (x + xl 2^-32, y + yl 2^-32) 2^e, and its
// terms m 2^et (|m| < 2^62).  The unit 2^e is set 2^8 above the largest
// term's so far and moves when a term's comes within 2^5 of it; settle(),
// called at least once in 32 terms, moves it when the sum leaves 62 bits.  A
// term whose unit is no more than 2^31 below the sum's is added exactly, a
// smaller one rounded to that.  Integer instructions only.
struct Sum2 {
  int64_t x = 0, y = 0;
  uint32_t xl = 0, yl = 0;
  int e = -(1 << 28);
};
// (v + l 2^-32) >> s
T2D_HD void sar96(int64_t &v, uint32_t &l, int s) {
  for (int k = 0; k < 3 && s >= 32; k++, s -= 32) {
    l = (uint32_t)v;
    v >>= 32;
  }
  s = s > 31 ? 31 : s;
  if (s > 0) {
    l = (l >> s) | ((uint32_t)v << (32 - s));
    v >>= s;
  }
}
// (v + l 2^-32) += m 2^-d, 1 <= d <= 63, exactly up to 32 and rounded down to
// 2^-32 beyond
T2D_HD void add96(int64_t &v, uint32_t &l, int64_t m, int d) {
  const uint32_t w = hi32((uint64_t)m << (64 - d));
#ifdef __CUDA_ARCH__
  const int64_t h = m >> d;
  uint32_t v0 = (uint32_t)v, v1 = hi32((uint64_t)v);
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
      : "+r"(l), "+r"(v0), "+r"(v1)
      : "r"(w), "r"((uint32_t)h), "r"(hi32((uint64_t)h)));
  v = (int64_t)(((uint64_t)v1 << 32) | v0);
#else
  l += w;
  v += (m >> d) + (l < w);
#endif
}
T2D_HD void raise(Sum2 &a, int e) {
  sar96(a.x, a.xl, e - a.e);
  sar96(a.y, a.yl, e - a.e);
  a.e = e;
}
T2D_HD void settle(Sum2 &a) {
  const uint32_t xh = hi32((uint64_t)a.x), yh = hi32((uint64_t)a.y);
  if ((int32_t)((xh ^ (xh << 1)) | (yh ^ (yh << 1))) < 0) raise(a, a.e + 4);
}
T2D_HD void add(Sum2 &a, int64_t mx, int64_t my, int et) {
  int d = a.e - et;
  if ((unsigned)(d - 5) > 26u) {
    if (d < 5) {
      raise(a, et + 8);
      d = 8;
    } else {
      const int s = d - 31 > 63 ? 63 : d - 31;
      mx = ((mx >> (s - 1)) + 1) >> 1;
      my = ((my >> (s - 1)) + 1) >> 1;
      d = 31;
    }
  }
  add96(a.x, a.xl, mx, d);
  add96(a.y, a.yl, my, d);
}
// The term (mx 2^ex, my 2^ey), the component of the smaller unit rounded to the
// other's.
template <class Low>
T2D_HD void add(Sum2 &a, int64_t mx, int ex, int64_t my, int ey, Low) {
  const int e = ex > ey ? ex : ey, sx = e - ex > 63 ? 63 : e - ex, sy = e - ey > 63 ? 63 : e - ey;
  if (sx) mx = ((mx >> (sx - 1)) + 1) >> 1;
  if (sy) my = ((my >> (sy - 1)) + 1) >> 1;
  add(a, mx, my, e);
}

// The same sum with a unit for each component, so that a component is summed
// to the accuracy of its own terms however small they are beside the other's.
struct Sum1 {
  int64_t v = 0;
  uint32_t l = 0;
  int e = -(1 << 28);
};
struct SumXY {
  Sum1 x, y;
};
T2D_HD void raise(Sum1 &a, int e) {
  sar96(a.v, a.l, e - a.e);
  a.e = e;
}
T2D_HD void settle(SumXY &a) {
  const uint32_t xh = hi32((uint64_t)a.x.v), yh = hi32((uint64_t)a.y.v);
  if ((int32_t)(xh ^ (xh << 1)) < 0) raise(a.x, a.x.e + 4);
  if ((int32_t)(yh ^ (yh << 1)) < 0) raise(a.y, a.y.e + 4);
}
// A term m 2^e of any size.
T2D_HD void add(Sum1 &a, int64_t m, int e) {
  if (m == 0) return;
  if (a.e - e < 5) raise(a, e + 8);
  const int d = a.e - e, over = d < 63 ? 0 : d > 126 ? 63 : d - 63;
  add96(a.v, a.l, m >> over, d < 63 ? d : 63);
}
// The term (mx 2^ex, my 2^ey).  low(second component, m, e) corrects one whose
// m stands for less than it says (see add_pair).
template <class Low>
T2D_HD void add(SumXY &a, int64_t mx, int ex, int64_t my, int ey, Low low) {
  const int dx = a.x.e - ex, dy = a.y.e - ey;
  if ((unsigned)(dx - 5) <= 58u && (unsigned)(dy - 5) <= 58u) {
    add96(a.x.v, a.x.l, mx, dx);
    add96(a.y.v, a.y.l, my, dy);
  } else {
    low(false, mx, ex);
    low(true, my, ey);
    add(a.x, mx, ex);
    add(a.y, my, ey);
  }
}
// v + l 2^-32 as a double times 2^e
T2D_HD double to_double(int64_t v, uint32_t l, int e) {
  // up to 31 bits further left while the top bits are clear
  const int64_t m = v < 0 ? ~v : v;
  int z = clz((uint64_t)m) - 2;
  z = z < 0 ? 0 : z > 31 ? 31 : z;
  const int64_t w = (int64_t)((uint64_t)v << z) + (z ? l >> (32 - z) : 0);
  return pack((uint64_t)(w < 0 ? -w : w), e - z + 1085, (uint64_t)w & 0x8000000000000000ull);
}

// ------------------------------------------------------ regularised pair
// r > 1e-10 (fmm.c:131), decided on r^2 > 1e-20 in FP64 where the exponent
// leaves it open: a component of 2^-33 or more decides it (field 990), none of
// 2^-34 or more rules it out.  The call keeps the FP64 products out of the
// pairs that do not need them (the compiler would predicate them into all).
#ifdef __CUDACC__
static __device__ __noinline__ bool apart64(double dx, double dy) {
  return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)) > 1.0e-20;
}
// a - b, once: opaque to the compiler, which would otherwise subtract again
// where it needs the sign (it takes FP64 additions to be cheap)
static __device__ __forceinline__ double minus(double a, double b) {
  double d = __dsub_rn(a, b);
  asm volatile("" : "+d"(d));
  return d;
}
static __device__ __forceinline__ bool apart(const Vec &v, double dx, double dy) {
  return v.e >= 990 || (v.e == 989 && apart64(dx, dy));
}
#endif

// e^-x = kExpInt[floor(x)] kExpFrac[next 11 bits] e^-r, r < 2^-11: a
// table-driven exponential (P. T. P. Tang, ACM TOMS 15, 1989) with both
// tables in units of 2^-62.
constexpr int kExpInts = 40;  // e^-40 < 2^-57: 1 - e^-x is 1 from there on
constexpr int kExpFracs = 2048;
struct ExpTables {
  uint64_t ints[kExpInts], fracs[kExpFracs];
};
typedef unsigned __int128 u128;
// e^-(j / 2048) in units of 2^-100 by its Taylor series in integers
constexpr u128 exp_series(int j) {
  u128 t = (u128)1 << 100, pos = t, neg = 0;
  for (int k = 1; t; k++) {
    t = (t * (unsigned)j >> 11) / (unsigned)k;
    if (k & 1)
      neg += t;
    else
      pos += t;
  }
  return pos - neg;
}
// high 128 bits of a product
constexpr u128 mul128(u128 a, u128 b) {
  const uint64_t ah = (uint64_t)(a >> 64), al = (uint64_t)a, bh = (uint64_t)(b >> 64), bl = (uint64_t)b;
  const u128 m1 = (u128)ah * bl, m2 = (u128)al * bh, l = (u128)al * bl;
  const u128 mid = (l >> 64) + (uint64_t)m1 + (uint64_t)m2;
  return (u128)ah * bh + (m1 >> 64) + (m2 >> 64) + (mid >> 64);
}
constexpr ExpTables make_exp_tables() {
  ExpTables r{};
  for (int j = 0; j < kExpFracs; j++) r.fracs[j] = (uint64_t)((exp_series(j) + ((u128)1 << 37)) >> 38);
  const u128 e1 = exp_series(kExpFracs) << 27;  // e^-1, units of 2^-127
  u128 v = (u128)1 << 127;
  for (int n = 0; n < kExpInts; n++) {
    r.ints[n] = (uint64_t)((v + ((u128)1 << 64)) >> 65);
    v = mul128(v, e1) << 1;
  }
  return r;
}

// Adds G (1 - exp(-r^2 / sigma^2)) / r^2 times (-dy, dx) to `sum`, for the
// offset (dx, dy) = v whose upper words are hx, hy: |G| = gm 2^(ge - 1085),
// 1/sigma^2 = cm 2^(ce - 1085), mantissas as mantissa() gives them, hg the
// upper word of G.  Each component's relative error is below 2^-52, besides
// an absolute 2^-55 in the bracket: the products take the components' own
// mantissas and exponents, so that this holds for offsets along an axis too.
// (A unit for each component costs 16,384 targets x 262,144 sources 26.2
// against 25.5 ms; with a common one a component at 2^-r of the other had 58 -
// r bits.)
template <class Sum>
T2D_HD void add_pair(Sum &sum, const Vec &v, uint32_t hx, uint32_t hy, uint64_t gm, int ge, uint32_t hg, uint64_t cm,
                     int ce, const uint64_t *exp_int, const uint64_t *exp_frac, One one) {
  if (gm == 0) return;
  const uint64_t m2 = norm2(v, one);
  // f 2^z = (1 - e^-x) / r^2; where e^-x is nothing, the reciprocal
  uint64_t f = recip(m2, one);
  int z = 4;
  // x = r^2 / sigma^2 in units of 2^-55, below 64; a product of 2^60 or more
  // with a left shift would be x >= 64
  const int s = 3074 - 2 * v.e - ce;
  if (s >= 0) {
    const uint64_t x = shr(mulhi(m2, cm, one) << 2, s);
    const uint32_t n = hi32(x) >> 23;
    if (n < kExpInts) {
      if (x == 0) return;  // below 2^-55
      const uint64_t t = mulhi(exp_int[n], exp_frac[(hi32(x) >> 12) & (kExpFracs - 1)], one);
      // u = 1 - e^-r = r - r^2/2 + r^2/2 r/3 (1 - r/4) in units of 2^-64, from
      // r = a 2^-43 + b 2^-55
      const uint64_t r = x & ((1ull << 44) - 1);
      const uint32_t a = (uint32_t)(r >> 12), b = (uint32_t)r & 4095u;
      const uint32_t p = hi32(wide(hi32(wide(a, 0x55555555u)), ~(a >> 13)));  // r/3 (1 - r/4), 2^-43
      const uint64_t rr = wide(a, a, wide(a, b) >> 11);                       // r^2, 2^-86
      // x was truncated: half a unit on average
      const uint64_t u = wide(hi32(wide(hi32(rr), p)) >> 2, (uint32_t)one.v, ((r << 9) | 256) - (rr >> 23));
      const uint64_t d = (1ull << 60) - t + mulhi(t, u, one);  // 1 - e^-x in units of 2^-60
      // leading one to bit 62 (to bit 31 or above where 1 - e^-x < 2^-28 has
      // fewer than 30 significant bits anyway)
      z = clz32(hi32(d) | 1u) - 1;
      f = mulhi(d << z, f, one);
    }
  }
  f = mulhi(f, gm, one);
  const uint64_t nx = ((v.ux << 10) & 0x3fffffffffffffffull) | 0x4000000000000000ull;
  const uint64_t ny = ((v.uy << 10) & 0x3fffffffffffffffull) | 0x4000000000000000ull;
  const uint64_t px = mulhi(f, nx, one), py = mulhi(f, ny, one);
  const int64_t sx = (int32_t)(hg ^ hx) >> 31, sy = ~((int32_t)(hg ^ hy) >> 31);
  const int ex = (int)(v.ux >> 52) & 0x7ff, ey = (int)(v.uy >> 52) & 0x7ff, et = ge - 2 * v.e - z - 55;
  add(sum, ((int64_t)py ^ sy) - sy, et + ey, ((int64_t)px ^ sx) - sx, et + ex, [&](bool second, int64_t &m, int &e) {
    if (second ? ex : ey) return;  // else no implicit bit, and the exponent of field 1
    const int64_t s = second ? sx : sy;
    m -= ((int64_t)(f >> 2) ^ s) - s;
    e++;
  });
}

// ------------------------------------------------------- multipole sums
// A cell's coefficients a_k (k < K) as integers b_k = a_k 2^(61 - eb - k es):
// es scales the polynomial's variable, eb the values, so that every partial
// sum of the Horner scheme stays below 2^61.  At every target that accepts
// the cell |w| 2^es < 1/2 (kHalf) or < 1.
struct Coef {
  long long re, im;
};
struct CellScale {
  int es, eb;
};
constexpr int kLeave = -(1 << 21);  // es of a cell left to FP64
// kHalf up to this opening angle: es can then reach the farthest blob's
// log2(0.71 R) whatever R (the full form up to twice that).
constexpr double kHalfTheta = 0.35;

// The terms k >= k0 are summed in FP32 pairs, about 46 bits: they reach the
// result times (w 2^es)^k0, and first_pair_term() sets k0 by the opening
// angle.  An FP32 instruction issues in one cycle where an integer one takes
// two, and a step needs 28 of them against 25.  For these k the entry holds
// (kAnchor + h, l) per component, h the multiple of 2^-22 nearest to
// b_k 2^-61 and l the rest.
T2D_HD int first_pair_term(double theta) {
  return theta <= 0.3 ? 5 : theta <= 0.4 ? 6 : theta <= 0.5 ? 7 : theta <= 0.6 ? 10 : 64;
}
constexpr float kAnchor = 3.0f;  // kAnchor + v, |v| < 1, is v rounded to a multiple of 2^-22
struct PairCoef {
  float re, rl, im, il;
};
T2D_HD float fma32(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}
T2D_HD float add32(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(a, b);
#else
  return a + b;
#endif
}
T2D_HD int32_t float_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_int(f);
#else
  int32_t i;
  std::memcpy(&i, &f, 4);
  return i;
#endif
}
T2D_HD int32_t to_int(float f) {
#ifdef __CUDA_ARCH__
  return __float2int_rn(f);
#else
  return (int32_t)std::lrintf(f);
#endif
}

// x = u - kAnchor + l; one real component of acc <- acc w + c:
// a w + b v + c for the FP32 pairs a, b (acc's components) and w, v.  The
// anchored sum takes the products' parts above 2^-22 exactly, their rests go
// to the low word.
struct PairReal {
  float h, l, f;  // the two parts and their rounded sum
};
T2D_HD float pair_step(const PairReal &a, float wh, float wl, const PairReal &b, float vh, float vl, float cu, float cl,
                       float &lo) {
  const float u2 = fma32(b.h, vh, cu), d2 = add32(u2, -cu), l2 = fma32(b.h, vh, -d2);
  const float u3 = fma32(a.h, wh, u2), d3 = add32(u3, -u2), l3 = fma32(a.h, wh, -d3);
  float t = add32(add32(cl, l2), l3);
  t = fma32(b.l, vh, t);
  t = fma32(a.l, wh, t);
  t = fma32(b.f, vl, t);
  lo = fma32(a.f, wl, t);
  return u3;
}
T2D_HD PairReal pair_real(float u, float l) {
  PairReal r;
  r.h = add32(u, -kAnchor);
  r.l = l;
  r.f = add32(r.h, l);
  return r;
}
// (u - kAnchor + l) 2^61
T2D_HD int64_t pair_fix(float u, float l, One one) {
  return swide(to_int(l * 0x1p51f), 1024 * one.v, (int64_t)((uint64_t)(uint32_t)((float_bits(u) - 0x40400000) << 7) << 32));
}
// w as an FP32 pair for w in units of unit 2^-42, the upper part a multiple
// of unit, the lower one to 2^-32 of it
T2D_HD void pair_of(int64_t w, float unit, float &h, float &l) {
  const int32_t g = ((int32_t)hi32((uint64_t)w) + (1 << 9)) >> 10;
  h = (float)g * unit;
  // bits 41..10 of the rest w - g 2^42, as a signed number
  l = (float)(int32_t)(uint32_t)((uint64_t)w >> 10) * (unit * 0x1p-32f);
}

// Adds sum_k a_k w^(k+1), w = 1/(dx + i dy), to `sum`.  With `may_leave`,
// false and nothing added for a target so far out (|w| 2^es below about 2^-5,
// which no target that opened the cell's parent reaches) that the fixed units
// would cost accuracy where the leading coefficients cancel.  False also for
// a cell left to FP64 altogether.
constexpr int kFarShift = 4;
template <bool kHalf, class Load, class LoadPair>
T2D_HD bool add_multipole(Sum2 &sum, double dx, double dy, CellScale sc, int K, int k0, Load load,
                          LoadPair load_pair, bool may_leave, One one) {
  const Vec v = vec(dx, dy);
  // w 2^es in units of 2^-64 or 2^-63 is W4 2^(1 - s) below (s >= 0 within
  // the bound)
  const int s = v.e - sc.es - (kHalf ? 1023 : 1022);
  if (s > (may_leave ? kFarShift : -kLeave / 2)) return false;
  const uint64_t y = recip(norm2(v, one), one);
  // |w| = W 2^(960 - e), W4 = 4 W < 2^63
  const uint64_t ux = mulhi(v.mx, y, one) << 2, uy = mulhi(v.my, y, one) << 2;
  const int64_t sx = (int64_t)bits(dx) >> 63, sy = ~((int64_t)bits(dy) >> 63);  // w = (dx - i dy) / |d|^2
  const int64_t vx = ((int64_t)shr(ux << 1, s) ^ sx) - sx, vy = ((int64_t)shr(uy << 1, s) ^ sy) - sy;
  int64_t ar, ai;
  int k;
  if (K > k0) {
    float xh, xl, yh, yl;
    pair_of(vx, kHalf ? 0x1p-22f : 0x1p-21f, xh, xl);
    pair_of(vy, kHalf ? 0x1p-22f : 0x1p-21f, yh, yl);
    PairCoef c = load_pair(K - 1);
    float ur = c.re, lr = c.rl, ui = c.im, li = c.il;
    for (k = K - 2; k >= k0; k--) {
      c = load_pair(k);
      const PairReal r = pair_real(ur, lr), i = pair_real(ui, li);
      ur = pair_step(r, xh, xl, i, -yh, -yl, c.re, c.rl, lr);
      ui = pair_step(r, yh, yl, i, xh, xl, c.im, c.il, li);
    }
    ar = pair_fix(ur, lr, one);
    ai = pair_fix(ui, li, one);
  } else {
    const Coef c = load(K - 1);
    ar = c.re;
    ai = c.im;
    k = K - 2;
  }
  const Limbs wx = limbs(vx), wy = limbs(vy);
  const int32_t mh = -wy.h, ml = -wy.l;
  for (; k >= 0; k--) {
    const Coef c = load(k);
    const Limbs r = limbs(kHalf ? ar : ar + ar), i = limbs(kHalf ? ai : ai + ai);
    const int64_t cr = swide(r.h, wx.l, swide(r.l, wx.h, swide(i.h, ml, swide(i.l, mh))));
    const int64_t ci = swide(r.h, wy.l, swide(r.l, wy.h, swide(i.h, wx.l, swide(i.l, wx.h))));
    ar = swide(r.h, wx.h, swide(i.h, mh, swide((int32_t)hi32((uint64_t)cr), one.v, (int64_t)c.re)));
    ai = swide(r.h, wy.h, swide(i.h, wx.h, swide((int32_t)hi32((uint64_t)ci), one.v, (int64_t)c.im)));
  }
  // the last factor w in full, not in the units of a far target's w 2^es
  const Limbs r = limbs(ar), i = limbs(ai);
  const Limbs zx = limbs(((int64_t)ux ^ sx) - sx), zy = limbs(((int64_t)uy ^ sy) - sy);
  const int32_t nh = -zy.h, nl = -zy.l;
  const int64_t cr = swide(r.h, zx.l, swide(r.l, zx.h, swide(i.h, nl, swide(i.l, nh))));
  const int64_t ci = swide(r.h, zy.l, swide(r.l, zy.h, swide(i.h, zx.l, swide(i.l, zx.h))));
  const int64_t vr = swide(r.h, zx.h, swide(i.h, nh, cr >> 32));
  const int64_t vi = swide(r.h, zy.h, swide(i.h, zx.h, ci >> 32));
  if (vr | vi) add(sum, vr, vi, 963 + sc.eb - v.e);
  return true;
}

// floor(log2 |v|) of a normal v; kNoLog for zero and subnormals
constexpr int kNoLog = -100000;
T2D_HD int ilog2(double v) {
  const int e = (int)(bits(v) >> 52) & 0x7ff;
  return e ? e - 1023 : kNoLog;
}
// v is an infinity, a NaN or subnormal
T2D_HD bool beyond(double v) {
  const uint32_t e = (uint32_t)(bits(v) >> 52) & 0x7ffu;
  return e == 0x7ffu || (e == 0 && (bits(v) << 1) != 0);
}
// 2^e |m| in FP32 for m = v 2^-ilog2(v), 0 below 2^-120, 2^120 above that
T2D_HD float mag32(double v, int e) {
  if (ilog2(v) == kNoLog || e < -120) return 0.0f;
  const uint32_t f = ((uint32_t)((e > 120 ? 120 : e) + 127) << 23) | ((uint32_t)(bits(v) >> 29) & 0x7fffffu);
  float r;
#ifdef __CUDA_ARCH__
  r = __uint_as_float(f);
#else
  std::memcpy(&r, &f, 4);
#endif
  return r;
}

// v 2^-ilog2(v)
T2D_HD double scale_frac(double v) { return from_bits((bits(v) & 0x800fffffffffffffull) | 0x3ff0000000000000ull); }

// The scale of a cell with coefficients a_k (k < K, load(k, re, im)), side R,
// for opening angle theta (a target accepts the cell only at R <= theta |d|).
// es is the smallest with |a_k| within a factor of 2 of the leading ones
// times 2^(k es), so that the b_k neither grow (the sums' headroom) nor fall
// below the units, within a factor of 2 of the largest that the bound on
// |w| 2^es allows (so that w keeps its digits).  The leading ones are a_0 to
// a_2, in units of (R/2)^k, or all if those are zero (moments that cancel
// exactly, as those of symmetric arrangements do).
// eb covers every partial sum |b_k| + wmax |b_k+1| + ..., wmax the largest
// |w| 2^es.  Exponent and FP32 arithmetic only: FP64 is slow.
//
// A cell whose leading coefficients are weak against the later ones is left
// to FP64 (es = kLeave).  In units of 2^eb the sums' rounding is about 2^-59,
// and that of the FP32 pairs 2^-46 x^k0, x = |w| 2^es, whatever the sum
// itself: where sum |b_k| x^k is too small for that, FP64, whose rounding
// goes with the terms, is better.  The line is drawn at an estimate of 2^-50
// of the terms' magnitudes, taken at the nearest target and four times
// farther out, where the sums' measured mean error passes FP64's (2^-51.7
// against 2^-51.7; at 2^-49: 2^-49.5 against 2^-51.6).  Ordinary cells (1 to
// 64 random blobs of random signs) stay below 2^-50.8; moments 0 and 1
// cancelled to about 2^-8 pass it.  So is a cell with an infinity, a NaN or a
// subnormal number among its coefficients (circulations or coordinates near
// the ends of FP64's range).
template <class Load>
T2D_HD CellScale cell_scale(int K, double R, double theta, Load load) {
  const int er = ilog2(R);
  auto log_of = [&](int k) {
    double re, im;
    load(k, re, im);
    const int a = ilog2(re), b = ilog2(im);
    return a > b ? a : b;
  };
  CellScale sc;
  int lead = kNoLog;
  for (int k = 0; k < K; k++) {
    double re, im;
    load(k, re, im);
    if (beyond(re) || beyond(im)) {
      sc.es = kLeave;
      sc.eb = 0;
      return sc;
    }
    const int a = log_of(k), l = a - k * (er - 1);
    if ((k < 3 || lead == kNoLog) && a > kNoLog && l > lead) lead = l;
  }
  const int cap = theta > 0.0 ? ilog2(R / (theta <= kHalfTheta ? 2.0 * theta : theta) * (1.0 - 0x1p-20)) : er;
  sc.es = cap - 1;
  sc.eb = 0;
  if (lead == kNoLog) return sc;
  int es = cap - 1;
  for (int k = 1; k < K; k++) {
    const int over = log_of(k) - lead - 1;  // needed: over <= k es
    if (over > kNoLog / 2 && over > k * es) es = over >= 0 ? (over + k - 1) / k : -((-over) / k);
  }
  sc.es = es = es > cap ? cap : es;
  // the partial sums in units of the largest |a_k| 2^(-k es)
  int top = kNoLog;
  for (int k = 0; k < K; k++) {
    const int l = log_of(k) - k * es;
    if (l > top) top = l;
  }
  const float wmax = theta > 0.0 ? (float)(theta / scale_frac(R)) * mag32(1.0, es - er) * 1.00001f : 1.0f;
  float beta = 0.0f, out4 = 0.0f, most = 0.0f;  // sum |b_k| x^k at x = wmax and wmax / 4
  for (int k = K - 1; k >= 0; k--) {
    double re, im;
    load(k, re, im);
    const float b = mag32(re, ilog2(re) - top - k * es) + mag32(im, ilog2(im) - top - k * es);
    beta = b + wmax * beta;
    out4 = b + 0.25f * wmax * out4;
    most = beta > most ? beta : most;
  }
  const int up = ilog2((double)(most * 1.00001f)) + 1;
  sc.eb = top + up;
  const int k0 = first_pair_term(theta);
  float x = 16.0f, x4 = 16.0f;
  for (int k = 0; k < k0 && K > k0; k++) x *= wmax, x4 *= 0.25f * wmax;
  if (K <= k0) x = x4 = 0.0f;
  const float unit = mag32(1.0, up);
  if (unit * (0x1p-9f + x) > beta || unit * (0x1p-9f + x4) > out4) sc.es = kLeave;
  return sc;
}
// a_k to the units of b_k, rounded to nearest
T2D_HD long long fix_coef(double a, int k, const CellScale &sc) {
  const int m = ilog2(a);
  if (m == kNoLog) return 0;
  const uint64_t v = ((bits(a) << 10) & 0x3fffffffffffffffull) | 0x4000000000000000ull;
  const int s = 1 + sc.eb + k * sc.es - m;  // >= 1 below the bound of eb
  const uint64_t r = (shr(v, s - 1) + 1) >> 1;
  return bits(a) >> 63 ? -(long long)r : (long long)r;
}

T2D_HD void pair_coef(double a, int k, const CellScale &sc, float &u, float &l) {
  const long long b = fix_coef(a, k, sc);  // units of 2^-61
  const int32_t g = (int32_t)((b + (1ll << 38)) >> 39);
  u = kAnchor + (float)g * 0x1p-22f;
  l = (float)(b - ((long long)g << 39)) * 0x1p-61f;
}

}  // namespace fix
}  // namespace t2d
