// fixed64.hpp -- the sampled functions of the plain FP64 walks in 64-bit fixed point.
//
// GB300 runs one FP64 instruction of a warp in the time of about 76 issue slots (1.06 TFLOP/s
// measured), so a 64-bit product out of four integer multiplies costs a tenth of an FP64 one.
// The sine and cosine of the azimuth, the logarithm of the free path, the factor of the deposit,
// the scattering angle and the rotation are functions of integers or of numbers below 2: here
// they are evaluated on the integer pipe, by Taylor series (and, for the logarithm, Tang's table of reciprocals,
// ACM Trans. Math. Softw. 16, 1990) whose truncation lies below 2^-57, and rounded to double
// once.  The first four's errors are at most 1.1 units in the last place of a result in [0.5, 1),
// absolute; the Henyey-Greenstein cosine's is 7e-17 at g = 0.9 and 7e-16 at 0.99 (the same formula
// in FP64: 4.5e-15 and 3.9e-14).  The CPU tests hold them to their bounds against wider arithmetic.
// Host and device code (the host form is what the tests call).
#pragma once
#include <stdint.h>
#include <string.h>

#include "vmc_types.hpp"

#if !defined(__CUDACC__)
#include <math.h>
#endif

namespace vmc {

VMC_HD inline uint64_t mulhi_u64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
VMC_HD inline int64_t mulhi_s64(int64_t a, int64_t b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return (int64_t)(((__int128)a * b) >> 64);
#endif
}
VMC_HD inline uint32_t mulhi_u32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
VMC_HD inline int32_t mulhi_s32(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }
VMC_HD inline int clz_u64(uint64_t x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}
VMC_HD inline double double_of_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double d;
  memcpy(&d, &b, 8);
  return d;
#endif
}
VMC_HD inline uint64_t bits_of_double(double d) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(d);
#else
  uint64_t b;
  memcpy(&b, &d, 8);
  return b;
#endif
}

// v 2^(exp - 64), rounded to nearest
VMC_HD inline double double_of_fixed(uint64_t v, int exp) {
  if (v == 0) return 0.0;
  const int z = clz_u64(v);
  const uint64_t m = v << z;
  return double_of_bits(((uint64_t)(1021 + exp - z) << 52) + (m >> 11) + ((m >> 10) & 1u));
}

// x 2^64 of 0 <= x < 1 (the fraction of x when it is larger), rounded down
VMC_HD inline uint64_t fixed_of_double(double x) {
  const uint64_t b = bits_of_double(x);
  const int s = (int)(b >> 52) - 1011;  // mantissa << s
  const uint64_t m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
  return s >= 0 ? (s < 64 ? m << s : 0) : (s > -64 ? m >> -s : 0);
}

// sine and cosine of turn 2^-64 of a full turn, within an eighth of one of its quarters: of that
// angle |sine| 2^63 and (1 - cosine) 2^63
struct TurnParts {
  int quadrant;
  bool neg;
  uint64_t sf, cf;
};
VMC_HD inline TurnParts turn_parts(uint64_t turn) {
  const uint64_t t = turn + 0x2000000000000000ull;
  const int quadrant = (int)(t >> 62);
  const int64_t y = (int64_t)((t << 2) - 0x8000000000000000ull);  // y 2^-64 quadrants, |.| <= 1/2
  const uint64_t a = y < 0 ? (uint64_t)0 - (uint64_t)y : (uint64_t)y;
  const uint64_t z = mulhi_u64(a, a);
  const uint32_t z5 = (uint32_t)(z >> 32);
  // sin(a pi/2) = a P(z), cos = 1 - z S(z); the small terms in 32 bits of finer scales
  uint32_t p = 0xb7d6dcf9u - (mulhi_u32(z5, 0xd5761958u) >> 7);  // 2^-62
  p = 0xf47a1a68u - (mulhi_u32(z5, p) >> 6);                      // 2^-56
  p = 0xf183a7efu - (mulhi_u32(z5, p) >> 6);                      // 2^-50
  uint64_t P = 0x000a83c1a43f73c1ull - (((uint64_t)z5 * p) >> 18);
  P = 0x0132d2cce62bd85cull - mulhi_u64(z, P);
  P = 0x1466bc6775aae1d2ull - mulhi_u64(z, P);
  P = 0xa55de7312df295f5ull - mulhi_u64(z, P);
  P = 0xc90fdaa22168c235ull - (mulhi_u64(z, P) >> 1);  // 2^-63
  const uint64_t sf = mulhi_u64(a, P);                 // 2^-63
  uint32_t s = 0x90631618u - (mulhi_u32(z5, 0x95062c8du) >> 7);  // 2^-65
  s = 0xdb7127a2u - (mulhi_u32(z5, s) >> 6);                      // 2^-59
  s = 0xfce9c51cu - (mulhi_u32(z5, s) >> 6);                      // 2^-53
  s = 0xd368f951u - (mulhi_u32(z5, s) >> 6);                      // 2^-47
  uint64_t S = 0x003c3ea0d1237576ull - (((uint64_t)z5 * s) >> 15);
  S = 0x05574f1f8f2ffe7full - mulhi_u64(z, S);
  S = 0x40f07c206d6b0ecdull - mulhi_u64(z, S);
  S = 0x9de9e64df22ef2d2ull - (mulhi_u64(z, S) >> 1);  // 2^-63
  const uint64_t cf = mulhi_u64(z, S);                 // (1 - cos) 2^63
  return TurnParts{quadrant, y < 0, sf, cf};
}
VMC_HD inline void sincos_turn(uint64_t turn, double &sn, double &cs) {
  const TurnParts p = turn_parts(turn);
  double sv = double_of_fixed(p.sf, 1);
  const double cv = p.cf == 0 ? 1.0 : double_of_fixed((uint64_t)0 - (p.cf << 1), 0);
  sv = p.neg ? -sv : sv;
  const double u = p.quadrant & 1 ? cv : sv, v = p.quadrant & 1 ? sv : cv;
  sn = p.quadrant & 2 ? -u : u;
  cs = (p.quadrant + 1) & 2 ? -v : v;
}
// the same in units of 2^-62
VMC_HD inline void sincos_turn_fixed(uint64_t turn, int64_t &sn, int64_t &cs) {
  const TurnParts p = turn_parts(turn);
  const int64_t s = (int64_t)(p.sf >> 1), sv = p.neg ? -s : s, cv = (int64_t)((0x8000000000000000ull - p.cf) >> 1);
  const int64_t u = p.quadrant & 1 ? cv : sv, v = p.quadrant & 1 ? sv : cv;
  sn = p.quadrant & 2 ? -u : u;
  cs = (p.quadrant + 1) & 2 ? -v : v;
}

// ---- directions and scattering angles: signed numbers in units of 2^-60, below 2 ----
// A product of two takes three 32-bit multiplies (of the lower halves' product the units are
// lost) and may come out two units low; sums of products share the shift.
constexpr int64_t kOne60 = 1ll << 60;
struct Split60 {
  int32_t h, l;  // h 2^30 + l
};
VMC_HD inline Split60 split60(int64_t x) { return Split60{(int32_t)(x >> 30), (int32_t)(x & 0x3fffffff)}; }
VMC_HD inline Split60 neg60(Split60 a) { return Split60{-a.h, -a.l}; }
VMC_HD inline int64_t wide(int32_t a, int32_t b) { return (int64_t)a * b; }
VMC_HD inline int64_t mul60(Split60 a, Split60 b) { return wide(a.h, b.h) + ((wide(a.h, b.l) + wide(a.l, b.h)) >> 30); }
VMC_HD inline int64_t dot60(Split60 a, Split60 b, Split60 c, Split60 d) {  // a b + c d
  return wide(a.h, b.h) + wide(c.h, d.h) + ((wide(a.h, b.l) + wide(a.l, b.h) + wide(c.h, d.l) + wide(c.l, d.h)) >> 30);
}
VMC_HD inline double double_of_60(int64_t v) {
  const uint64_t a = v < 0 ? (uint64_t)0 - (uint64_t)v : (uint64_t)v;
  const uint64_t d = bits_of_double(double_of_fixed(a, 4));
  return double_of_bits(d | ((uint64_t)v & 0x8000000000000000ull));
}
// |x| < 2, cut off below a unit
VMC_HD inline int64_t fixed60_of(double x) {
  const uint64_t b = bits_of_double(x);
  const int e = 1023 - (int)((b >> 52) & 0x7ffu);
  const int64_t v = (int64_t)((((b & 0xfffffffffffffull) | 0x10000000000000ull) << 8) >> (e < 63 ? e : 63));
  return (int64_t)b < 0 ? -v : v;
}
// upper half of |x|'s bits: orders magnitudes to 2^-20
VMC_HD inline uint32_t mag_of(double x) { return (uint32_t)(bits_of_double(x) >> 32) & 0x7fffffffu; }

#ifdef __CUDA_ARCH__
__device__ __forceinline__ float near_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float near_rsqrt(float x) { return rsqrtf(x); }
#else
inline float near_rcp(float x) { return 1.0f / x; }
inline float near_rsqrt(float x) { return 1.0f / sqrtf(x); }
#endif

// 1 / (d 2^-64) in units of 2^-61, d >= 2^63: an FP32 quotient y of d's upper half and what
// 1 - d y = e leaves of it, y (1 + e + e^2).  |e| < 2^-21 by the conversion of the upper half
// (2^-24) and the quotient's documented error of an ulp; the shift leaves room for 2^-21.
VMC_HD inline uint64_t rcp_refined(uint64_t d, float y) {
  const int32_t y0 = (int32_t)(y * 2305843009213693952.0f);  // 2^-29
  const uint64_t p = (d >> 32) * (uint32_t)y0 + (((uint64_t)(uint32_t)d * (uint32_t)y0) >> 32);
  const int64_t e = (int64_t)(0x2000000000000000ull - p);  // 2^-61
  const int32_t e5 = (int32_t)(e >> 9);                    // 2^-52
  const int64_t t = e + (wide(e5, e5) >> 43);
  return ((uint64_t)y0 << 32) + (uint64_t)((wide(y0, (int32_t)(t >> 15)) >> 14) + (wide(y0, (int32_t)(t & 0x7fff)) >> 29));
}
VMC_HD inline float rcp_first(uint64_t d) { return near_rcp((float)(uint32_t)(d >> 32)); }
VMC_HD inline uint64_t rcp_fixed(uint64_t d) { return rcp_refined(d, rcp_first(d)); }

// sqrt(s) 2^-k and 2^k / sqrt(s), s > 0, both in [1/2, 2]: h = t y from t = s 4^k, brought to
// [1/4, 1] or less than a unit above, and an FP32 y = 1 / sqrt(t); then with e = 1 - h y both
// times 1 + e / 2 + 3 e^2 / 8.  Two ulps of the root's documented error, t's conversion and the
// cut of y to 2^-29 make |e| < 5.5e-7; the shift leaves room for 2^-20.
struct Root60 {
  int64_t r, y;
  int k;
};
VMC_HD inline int root_shift(int64_t s) {
  return (clz_u64((uint64_t)s | 1u) - (s >> 60 ? 3 : 4)) >> 1;  // s = 1 is 2^60: none
}
VMC_HD inline float root_first(int64_t t) { return near_rsqrt((float)(uint32_t)(t >> 29) * 4.656612873077393e-10f); }
VMC_HD inline Root60 root_refined(int64_t t, int k, float y) {
  const int32_t y0 = (int32_t)(y * 536870912.0f);  // 2^-29
  const Split60 ts = split60(t);
  const int64_t h = (wide(ts.h, y0) << 1) + (wide(ts.l, y0) >> 29);
  const Split60 hs = split60(h);
  const int64_t e = kOne60 - ((wide(hs.h, y0) << 1) + (wide(hs.l, y0) >> 29));
  const int32_t e5 = (int32_t)(e >> 9);  // 2^-51
  const int64_t u = (e >> 1) + ((3 * (wide(e5, e5) >> 42)) >> 3);
  Root60 q;
  q.r = h + mul60(hs, split60(u));
  q.y = ((int64_t)y0 << 31) + (wide(y0, (int32_t)(u >> 15)) >> 14) + (wide(y0, (int32_t)(u & 0x7fff)) >> 29);
  q.k = k;
  return q;
}
VMC_HD inline Root60 sqrt60(int64_t s) {
  const int k = root_shift(s);
  const int64_t t = s << (2 * k);
  return root_refined(t, k, root_first(t));
}

// The Henyey-Greenstein cosine of the closed uniform's word u: with c = 2 xi - 1 and
// q = (1 - g^2) / (1 + g c) it is (1 + g^2 - q^2) / (2 g), c when g = 0.  inv = hg_inverse(g),
// 1 / (2 |g|) brought to [1/2, 1] by a power of two: as a double its rounding would be every
// event's, and walks added that up to more than all their other errors.
// kNoCosine for |g| above 0.999 or below 2^-30, which these units do not hold to a double's last
// place.
constexpr int64_t kNoCosine = INT64_MIN;
VMC_HD inline uint64_t hg_inverse(double g) {
  return (rcp_fixed(((bits_of_double(g) & 0xfffffffffffffull) | 0x10000000000000ull) << 11) + 2) >> 2;
}
VMC_HD inline int64_t hg_cosine(uint32_t u, double g, uint64_t inv) {
  const int64_t c = (int64_t)((((uint64_t)u << 32) | u) ^ 0x8000000000000000ull) >> 3;
  if (u == 0u || u == 0xffffffffu) return u == 0u ? -kOne60 : kOne60;
  if ((bits_of_double(g) << 1) == 0) return c;
  const uint32_t mag = mag_of(g);
  if (mag > 0x3feff7ceu || mag < 0x3e100000u) return kNoCosine;  // 0.999, 2^-30
  const uint64_t ga = fixed_of_double(double_of_bits(bits_of_double(g) & 0x7fffffffffffffffull));  // |g| 2^64
  const int64_t g6 = (int64_t)(ga >> 4);
  const uint64_t a = (uint64_t)0 - mulhi_u64(ga, ga);  // (1 - g^2) 2^64
  const uint64_t d = (uint64_t)(kOne60 + mul60(split60((int64_t)bits_of_double(g) < 0 ? -g6 : g6), split60(c)));
  const int z = clz_u64(d);
  const uint64_t q = ((mulhi_u64(a, rcp_fixed(d << z) << 1)) << (z - 3)) >> 3;
  const Split60 qs = split60((int64_t)q);
  const int64_t m = 2 * kOne60 - (int64_t)(a >> 4) - mul60(qs, qs);
  const int64_t ct = mul60(split60(m << (1022 - (int)(mag >> 20))), split60((int64_t)inv));
  return (int64_t)bits_of_double(g) < 0 ? -ct : ct;
}

// Cosine and sine of the 2D scattering angle 2 atan(h), h = tan(pi xi) (1 - g) / (1 + g), xi =
// u 2^-32, in units of 2^-60; k = turn_ratio(g), (1 - |g|) / (1 + |g|) 2^64, or 0 for |g| above
// 0.999 or below 2^-30.  With x = cos(pi xi) and y = sin(pi xi),
// the one that k belongs to times it (x when g < 0), they are (x^2 - y^2) / (x^2 + y^2) and
// 2 x y / (x^2 + y^2).  False when k = 0 and g is not.
VMC_HD inline uint64_t turn_ratio(double g) {
  const uint32_t mag = mag_of(g);
  if (mag > 0x3feff7ceu || mag < 0x3e100000u) return 0;  // 0.999, 2^-30
  const uint64_t ga = fixed_of_double(double_of_bits(bits_of_double(g) & 0x7fffffffffffffffull));
  return mulhi_u64((uint64_t)0 - ga, rcp_fixed(0x8000000000000000ull + (ga >> 1)) << 2);
}
VMC_HD inline bool turn_2d(uint32_t u, double g, uint64_t k, int64_t &c, int64_t &s) {
  const bool iso = (bits_of_double(g) << 1) == 0;  // then the angle is 2 pi xi itself
  int64_t s0, c0;
  sincos_turn_fixed((uint64_t)u << (iso ? 32 : 31), s0, c0);
  uint64_t x = (uint64_t)(c0 < 0 ? -c0 : c0), y = (uint64_t)s0;
  const bool back = (int64_t)bits_of_double(g) < 0;
  const uint64_t cut = mulhi_u64(back ? x : y, k);
  x = back ? cut : x;
  y = back ? y : cut;
  const int z = clz_u64(x > y ? x : y);
  const Split60 xs = split60((int64_t)((x << z) >> 4)), ys = split60((int64_t)((y << z) >> 4));
  const int64_t a = mul60(xs, xs), b = mul60(ys, ys), d = a + b;  // [1/4, 2)
  const int zd = clz_u64((uint64_t)d);
  const Split60 inv = split60((int64_t)(rcp_fixed((uint64_t)d << zd) >> 2));
  const int64_t cs = mul60(split60(a - b), inv) << (zd - 3), sn = mul60(split60(mul60(xs, ys)), inv) << (zd - 2);
  c = iso ? c0 >> 2 : cs;
  s = iso ? s0 >> 2 : c0 < 0 ? -sn : sn;
  return iso || k != 0;
}

// v brought back to length 1 when it is there to 2^-30 already
VMC_HD inline bool unit60(int64_t *v, int n) {
  int64_t hh = 0, hl = 0;
  for (int i = 0; i < n; i++) {
    const Split60 s = split60(v[i]);
    hh += wide(s.h, s.h);
    hl += wide(s.h, s.l);
  }
  const int64_t d = hh + ((2 * hl) >> 30) - kOne60;
  if (d >= 1 << 30 || d <= -(1 << 30)) return false;
  for (int i = 0; i < n; i++) v[i] -= wide((int32_t)(v[i] >> 30), (int32_t)d) >> 31;
  return true;
}

// 1 - x / 2! + x^2 / 3! - ..., so that 1 - exp(-x) = x times it, for 0 <= x < 1/16
VMC_HD inline double one_minus_exp_over_x(double x) {
  const uint64_t X = fixed_of_double(x);
  const uint32_t x5 = (uint32_t)(X >> 32);
  uint32_t h = 0xd00d00d0u - (mulhi_u32(x5, 0xb8ef1d2bu) >> 3);  // 2^-47
  h = 0xd00d00d0u - (mulhi_u32(x5, h) >> 3);                      // 2^-44
  h = 0xb60b60b6u - (mulhi_u32(x5, h) >> 3);                      // 2^-41
  uint64_t H = 0x0222222222222222ull - (((uint64_t)x5 * h) >> 9);
  H = 0x0aaaaaaaaaaaaaabull - mulhi_u64(X, H);
  H = 0x2aaaaaaaaaaaaaabull - mulhi_u64(X, H);
  H = 0x8000000000000000ull - mulhi_u64(X, H);
  const uint64_t e = mulhi_u64(X, H);
  return e == 0 ? 1.0 : double_of_fixed((uint64_t)0 - e, 0);
}

struct alignas(16) LogEntry {  // read by one 16-byte load
  uint64_t log_r;  // log(r / 256) 2^63
  uint64_t r;      // 256 / (the interval's middle), rounded: 256 at the end, where log is 0
};
static_assert(alignof(LogEntry) == 16 && sizeof(LogEntry) == 16, "LogEntry is loaded as 16 bytes");
#ifdef __CUDACC__
__device__
#endif
static const LogEntry kLogTable[128] = {
    {0x5838cbd11e23632aull, 510u}, {0x5736c771b05d9234ull, 506u}, {0x5632b6d735e624c2ull, 502u}, {0x552c919e66525ea4ull, 498u},
    {0x54669302e8d1199bull, 495u}, {0x535cb4e8e7f4011dull, 491u}, {0x5250aa0e8bf01dedull, 487u}, {0x51862f08717b09f4ull, 484u},
    {0x50763fa119cab992ull, 480u}, {0x4fa8ce4dacbd6e0full, 477u}, {0x4e94dcf9faf7e632ull, 473u}, {0x4dc45ed51d1ed717ull, 470u},
    {0x4cac4ce44875c4c8ull, 466u}, {0x4bd8aa65425518b6ull, 463u}, {0x4b03a7b5123a2ee6ull, 460u}, {0x4a2d4037d81e0abcull, 457u},
    {0x49556f3a63df2cf0ull, 454u}, {0x483373464aadb64dull, 450u}, {0x475843f99dc00c21ull, 447u}, {0x467b9ad19f25bb31ull, 444u},
    {0x459d72aeae98380eull, 441u}, {0x44bdc6564fbef14cull, 438u}, {0x43dc90726d25f53bull, 435u}, {0x43458f32e75adf82ull, 433u},
    {0x4261bd3d5cd482e4ull, 430u}, {0x417c52f49916702aull, 427u}, {0x40954a969743fb1aull, 424u}, {0x3fac9e41ec2ae395ull, 421u},
    {0x3f10946dfd3d8459ull, 419u}, {0x3e251ebf5e0dd967ull, 416u}, {0x3d37f4cb30c3eac9ull, 413u}, {0x3c98e350d0ee085aull, 411u},
    {0x3ba8d4098389417eull, 408u}, {0x3b07ce4b145e7ca1ull, 406u}, {0x3a14c75ce43cc84bull, 403u}, {0x3971c0e89af593fbull, 401u},
    {0x387baf4f9b5a9ae7ull, 398u}, {0x37d69b3b4e36f7efull, 396u}, {0x3730b12d2621f6b3ull, 394u}, {0x36363c1d7bf8b6d2ull, 391u},
    {0x358e3184b161c818ull, 389u}, {0x34e5492cd7b3d42dull, 387u}, {0x33e647d97f3097e5ull, 384u}, {0x333b2b022fc11597ull, 382u},
    {0x328f2838422df575ull, 380u}, {0x31e23d0e6cc58efcull, 378u}, {0x3134670d8284b56bull, 376u}, {0x302de83b41a92b6bull, 373u},
    {0x2f7dbc146f5f7f3cull, 371u}, {0x2ecc9c2473b79d82ull, 369u}, {0x2e1a85c4f1246babull, 367u}, {0x2d6776446b287b13ull, 365u},
    {0x2cb36ae607c3e504ull, 363u}, {0x2bfe60e14f27a791ull, 361u}, {0x2b485561e99fc339ull, 359u}, {0x2a9145875ba4c5a0ull, 357u},
    {0x29d92e64c004d35full, 355u}, {0x29200d008013a198ull, 353u}, {0x2865de5409d0276bull, 351u}, {0x2808610d0d4fc77aull, 350u},
    {0x274c98aad28bd38eull, 348u}, {0x268fbb3530faa9adull, 346u}, {0x25d1c575c23a6138ull, 344u}, {0x2512b427bd0d46bdull, 342u},
    {0x245283f79ef2cb45ull, 340u}, {0x23f1ff3c9145e51bull, 339u}, {0x23301a5ba846decfull, 337u}, {0x226d0e05275160beull, 335u},
    {0x220b17f35c95aa31ull, 334u}, {0x214649c4e721c6bfull, 332u}, {0x20804b2969a081b6ull, 330u}, {0x201cd88b5aa0398dull, 329u},
    {0x1f550a564b7b3707ull, 327u}, {0x1e8c0252aa5a5fe9ull, 325u}, {0x1e27076e2af2e5eaull, 324u}, {0x1d5c216b4fbb915cull, 322u},
    {0x1c8ff7c79a9a21acull, 320u}, {0x1c2968558c18c0a3ull, 319u}, {0x1b5b519e8fb5a46full, 317u}, {0x1af3c94e80bff2d9ull, 316u},
    {0x1a23bc1fe2b56319ull, 314u}, {0x19bb362e7dfb8356ull, 313u}, {0x18e928de886d40aaull, 311u}, {0x187fa06520c91090ull, 310u},
    {0x17ab890210d9091cull, 308u}, {0x1740f8f54037a4caull, 307u}, {0x16d60fe719d21c8dull, 306u}, {0x15ff3070a793d3c8ull, 304u},
    {0x159338d9982085d3ull, 303u}, {0x14ba36f39a55e55aull, 301u}, {0x144d2b6ccb7d1e68ull, 300u}, {0x13dfc2b0ecc629cbull, 299u},
    {0x1303d718e47fd2ffull, 297u}, {0x129552f81ff5234cull, 296u}, {0x12266f190a5acb7dull, 295u}, {0x114785846742ac69ull, 293u},
    {0x10d77e7cd08e5967ull, 292u}, {0x10671512ca596e2aull, 291u}, {0x0f85186008b15331ull, 289u}, {0x0f1383b7157972f5ull, 288u},
    {0x0ea189eb3659aeafull, 287u}, {0x0e2f2a47ade3a18bull, 286u}, {0x0d49369d256ab1b3ull, 284u}, {0x0cd5a1231019d66eull, 283u},
    {0x0c61a2eb18cd907bull, 282u}, {0x0bed3b36bd896642ull, 281u}, {0x0b032c549ba861d9ull, 279u}, {0x0a8d839f830c1fb5ull, 278u},
    {0x0a176e5f5323781eull, 277u}, {0x09a0ebcb0de8e849ull, 276u}, {0x0929fb17850a0b7cull, 275u}, {0x08b29b7751bd7074ull, 274u},
    {0x07c28c300458a998ull, 272u}, {0x0749dae2b6c2d484ull, 271u}, {0x06d0b75c465c6fb1ull, 270u}, {0x065720c3b238fadfull, 269u},
    {0x05dd163d8cb73f12ull, 268u}, {0x056296ebf2393523ull, 267u}, {0x04e7a1ee7faf57eaull, 266u}, {0x046c366248f65ff1ull, 265u},
    {0x03f05361cf06600aull, 264u}, {0x0373f804f5f232ffull, 263u}, {0x02f72360fab62355ull, 262u}, {0x0279d48868d4ae9eull, 261u},
    {0x01fc0a8b0fc03e3dull, 260u}, {0x017dc475f810a76eull, 259u}, {0x00ff015358833c48ull, 258u}, {0x0000000000000000ull, 256u},
};

// -log((w + 1/2) 2^-32), the exponential sample of the open uniform's word w
VMC_HD inline double neg_log_open(uint32_t w) {
  const uint64_t N = 2 * (uint64_t)w + 1;  // (w + 1/2) 2^-32 = N 2^-33
  const int k = clz_u64(N) - 31;           // = x 2^-k, x = (N << k) 2^-33 in [0.5, 1)
  const uint64_t M = N << k;
  const int i = (int)(M >> 25) & 127;
#ifdef __CUDA_ARCH__
  const ulonglong2 t = __ldg(reinterpret_cast<const ulonglong2 *>(kLogTable) + i);
  const uint64_t log_r = t.x, r = t.y;
#else
  const uint64_t log_r = kLogTable[i].log_r, r = kLogTable[i].r;
#endif
  // v = x r / 256 - 1 exactly, |v| < 0.0046: log(x) = log(1 + v) - log(r / 256)
  const int64_t V = (int64_t)(M * r) - (1ll << 41);  // v 2^41
  const int32_t v5 = (int32_t)(V >> 9);              // 2^-32
  const int64_t v = (int64_t)((uint64_t)V << 22);    // 2^-63
  int32_t u = 0x12492492 - mulhi_s32(v5, 0x10000000);  // 1/7 - v/8, 2^-31
  u = 0x15555555 - mulhi_s32(v5, u);
  u = 0x1999999a - mulhi_s32(v5, u);
  u = 0x20000000 - mulhi_s32(v5, u);
  int64_t W = 0x1555555555555555ll - 2 * mulhi_s64(v, (int64_t)u << 31);  // 2^-62
  W = 0x2000000000000000ll - 2 * mulhi_s64(v, W);
  W = 0x4000000000000000ll - 2 * mulhi_s64(v, W);
  if (log_r == 0 && k == 0) {  // x next to 1: -v W from the normalised v, to the last bit
    const uint64_t a = (uint64_t)-V;
    const int z = clz_u64(a);
    return double_of_fixed(mulhi_u64(a << z, (uint64_t)W << 1), 24 - z);
  }
  const int64_t lv = mulhi_s64(v, W);  // log(1 + v) 2^61
  if (k == 0) return double_of_fixed(log_r - (uint64_t)(lv << 2), 1);
  return double_of_fixed((uint64_t)k * 0x058b90bfbe8e7bcdull + (log_r >> 4) - (uint64_t)(lv >> 2), 5);
}

}  // namespace vmc
