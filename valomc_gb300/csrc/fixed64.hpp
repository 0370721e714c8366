// fixed64.hpp -- the sampled functions of the plain FP64 walks in 64-bit fixed point.
//
// GB300 runs one FP64 instruction of a warp in the time of about 76 issue slots (1.06 TFLOP/s
// measured), so a 64-bit product out of four integer multiplies costs a tenth of an FP64 one.
// The sine and cosine of the azimuth, the logarithm of the free path and the factor of the
// deposit are functions of integers or of small numbers in [0, 1): here they are evaluated on
// the integer pipe, by Taylor series (and, for the logarithm, Tang's table of reciprocals,
// ACM Trans. Math. Softw. 16, 1990) whose truncation lies below 2^-57, and rounded to double
// once.  Each function's error is at most 1.1 units in the last place of a result in [0.5, 1),
// absolute; the CPU tests hold them to that against wider arithmetic.
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

// sine and cosine of turn 2^-64 of a full turn
VMC_HD inline void sincos_turn(uint64_t turn, double &sn, double &cs) {
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
  double sv = double_of_fixed(sf, 1);
  const double cv = cf == 0 ? 1.0 : double_of_fixed((uint64_t)0 - (cf << 1), 0);
  sv = y < 0 ? -sv : sv;
  const double u = quadrant & 1 ? cv : sv, v = quadrant & 1 ? sv : cv;
  sn = quadrant & 2 ? -u : u;
  cs = (quadrant + 1) & 2 ? -v : v;
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

struct LogEntry {
  uint64_t log_r;  // log(r / 256) 2^63
  uint64_t r;      // 256 / (the interval's middle), rounded: 256 at the end, where log is 0
};
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
