// walk3d.cuh -- the tetrahedral photon walk, one element step per call.
//
// Walk3D64: plain form.  Follows PropagatePhoton (cpp/3d/MC3D.hpp:1450-1638) with the state
//   in FP64: the exit face that the reference's Moller-Trumbore test over the faces in order,
//   skipping the entry face, finds (WhichFace :1006-1057), Henyey-Greenstein ScatterPhoton
//   (:1297-1340; the polar cosine used as drawn, without acos / cos), FresnelPhoton
//   (:1365-1447), MirrorPhoton (:1343-1351), roulette and the reverse-face lookup
//   (:1573-1631).  Draw order is the reference's, so a tape replay visits the same elements.
// Walk3D32: tracking form.  Position, direction and weight in FP32; the exit face is the
//   nearest of the faces the direction points out of, from precomputed outward planes
//   (the barycentric coordinate of the opposite vertex reaching zero), with the distance
//   clamped at 0 -- a photon cannot be lost to rounding.  Fluence is still accumulated
//   into FP64 arrays.
// Both merge consecutive deposits in one element in a register and flush them with one
// FP64 atomic when the photon leaves the element or dies.
#pragma once
#include "walk_common.cuh"

namespace vmc {

enum StepResult { kAlive = 0, kScattered = 1, kAliveMax = kScattered, kDied = 2 };

// Moller-Trumbore (RayTriangleIntersects, cpp/3d/MC3D.hpp:1825-1869)
__device__ __forceinline__ bool ray_tri(const double O[3], const double D[3], const double *V0, const double *V1,
                                        const double *V2, double &t) {
  double e1[3] = {V1[0] - V0[0], V1[1] - V0[1], V1[2] - V0[2]};
  double e2[3] = {V2[0] - V0[0], V2[1] - V0[1], V2[2] - V0[2]};
  double pv[3] = {D[1] * e2[2] - D[2] * e2[1], D[2] * e2[0] - D[0] * e2[2], D[0] * e2[1] - D[1] * e2[0]};
  double det = e1[0] * pv[0] + e1[1] * pv[1] + e1[2] * pv[2];
  if ((-kDblEps < det) && (det < kDblEps)) return false;
  double tv[3] = {O[0] - V0[0], O[1] - V0[1], O[2] - V0[2]};
  double inv = 1.0 / det;
  double u = (tv[0] * pv[0] + tv[1] * pv[1] + tv[2] * pv[2]) * inv;
  if ((u < 0.0) || (u > 1.0)) return false;
  double qv[3] = {tv[1] * e1[2] - tv[2] * e1[1], tv[2] * e1[0] - tv[0] * e1[2], tv[0] * e1[1] - tv[1] * e1[0]};
  double v = (D[0] * qv[0] + D[1] * qv[1] + D[2] * qv[2]) * inv;
  if ((v < 0.0) || (u + v > 1.0)) return false;
  t = (e2[0] * qv[0] + e2[1] * qv[1] + e2[2] * qv[2]) * inv;
  return true;
}

// Fresnel reflect-or-transmit decision in FP64 (cpp/3d/MC3D.hpp:1397-1430).  Returns true
// when reflected.  costht is the transmitted cosine when false is returned.  R from the closed
// forms rs = (eta ci - ct) / (eta ci + ct), rp = (ci - eta ct) / (ci + eta ct) over one division:
// the reference's R = (sin^2(thi - tht) / sin^2(thi + tht) + tan^2 / tan^2) / 2 to a few ulps,
// without its seven angles and their functions.
//
// Where FP32 is certain of the choice it is made there, and the photon that leaves the body or is
// reflected needs no root and no quotient in FP64: eta = n1 / n2 and ci = |cos| in FP32 have
// errors of 3e-7, so 1 - ct^2 = eta^2 (1 - ci^2) one of 1e-6 (1 + eta^2), and R, from ct >= 0.1,
// one of 1e-4 (1 + eta^2); twice the last and ten times the other are allowed for.  word: what
// has been drawn, if anything.  With the launches' directions (create_photon_2d) 7.6 -> 5.8 ms
// for 1e6 photons on the 2D square, which launch, and meet the boundary, every 30 steps.
struct Choice {
  enum What { kPass, kReflect, kUnsure } what;
  bool drawn;
  uint32_t word;
};
template <class R>
__device__ __forceinline__ Choice fresnel_choice(R &rng, float eta, float dn, float nn) {
  const float ci = fabsf(dn) * rsqrtf(nn), e2 = eta * eta, s2 = e2 * fmaf(-ci, ci, 1.0f), wide = 1.0f + e2;
  if (!(eta > 0.25f && eta < 4.0f && nn > 1e-30f && nn < 1e30f && ci < 1.00001f)) return Choice{Choice::kUnsure, false, 0u};
  if (s2 > 1.0f + 1e-5f * wide) return Choice{Choice::kReflect, false, 0u};
  if (!(s2 < 0.99f)) return Choice{Choice::kUnsure, false, 0u};
  const uint32_t w = rng.next();
  const float ct = sqrtf(1.0f - s2);
  const float rs = __fdividef(fmaf(eta, ci, -ct), fmaf(eta, ci, ct)), rp = __fdividef(fmaf(-eta, ct, ci), fmaf(eta, ct, ci));
  const float m = (float)w * 2.3283064365386963e-10f - 0.5f * fmaf(rs, rs, rp * rp);
  const bool near1 = ci > 0.999999f;  // above 1 the photon passes (below)
  return Choice{m > 2e-4f * wide ? Choice::kPass : m < -2e-4f * wide && !near1 ? Choice::kReflect : Choice::kUnsure, true, w};
}
template <class R>
__device__ __forceinline__ bool fresnel_reflects_d(R &rng, const Choice &choice, double nipnt, double costhi, double &costht) {
  const double s = 1.0 - nipnt * nipnt * (1.0 - costhi * costhi);
  if (s <= 0.0) return true;
  costht = fast_sqrt(s);
  if (choice.what == Choice::kPass) return false;
  const double ci = fabs(costhi);
  const double u = word_d(choice.drawn ? choice.word : rng.next()) * (1.0 / 4294967295.0);  // unif_closed
  if (!(ci <= 1.0)) return false;  // acos is NaN there in the reference, and so is R
  const double a = fma(nipnt, ci, -costht), b = fma(nipnt, ci, costht);
  const double c = fma(-nipnt, costht, ci), d = fma(nipnt, costht, ci);
  const double q = b * d, rs = a * d, rp = c * b;
  return u <= 0.5 * fast_div(fma(rs, rs, rp * rp), q * q);
}

// The same in the reference's angles, for the literal walks (cpp/3d/MC3D.hpp:1397-1430).  Returns true
// when reflected.  costht is the transmitted cosine when false is returned.
template <class R>
__device__ __forceinline__ bool fresnel_reflects_angles(R &rng, double nipnt, double costhi, double &costht) {
  double s = 1.0 - nipnt * nipnt * (1.0 - costhi * costhi);
  if (s <= 0.0) return true;
  costht = sqrt(s);
  double thi = acos(costhi > 0.0 ? costhi : -costhi);
  double tht = acos(costht);
  double refl;
  double sp = sin(thi + tht);
  if (!(sp > kDblEps)) {
    double q = (nipnt - 1.0) / (nipnt + 1.0);
    refl = q * q;
  } else {
    double a = sin(thi - tht) / sp, b = tan(thi - tht) / tan(thi + tht);
    refl = 0.5 * (a * a + b * b);
  }
  return unif_closed(rng) <= refl;
}

// Fresnel in FP32 from the closed forms rs = (eta ci - ct)/(eta ci + ct),
// rp = (ci - eta ct)/(ci + eta ct), R = (rs^2 + rp^2)/2 (same R as the reference's angle form).
template <class R>
__device__ __forceinline__ bool fresnel_reflects_f(R &rng, float eta, float ci, float &ct) {
  // fused multiply-adds written out: one rounding whatever kernel this is inlined into
  float s = fmaf(-__fmul_rn(eta, eta), fmaf(-ci, ci, 1.0f), 1.0f);
  if (s <= 0.0f) return true;
  ct = sqrtf(s);
  // a launch direction that is not unit length (3D BCLNormal of direction type 'a'/'r' is
  // not normalised, MC3D.hpp:679-683) can give |cos| > 1: acos is then NaN in the
  // reference, R is NaN and the photon is transmitted
  if (!(ci <= 1.0f)) return false;
  float rs = fmaf(eta, ci, -ct) / fmaf(eta, ci, ct);
  float rp = fmaf(-eta, ct, ci) / fmaf(eta, ct, ci);
  float Rf = 0.5f * fmaf(rs, rs, __fmul_rn(rp, rp));
  return unif_closed_f(rng) <= Rf;
}

__device__ __forceinline__ bool is_mirror(uint8_t bt) { return bt == 'm' || bt == 'L' || bt == 'I' || bt == 'C'; }

// 1 - exp(-x) for x >= 0 in FP32 without cancellation: below 0.1 the series to x^5
// (truncation x^6/720, relative x^5/720 < 1.4e-8); above, 1 - exp(-x) from the fast
// exponential (relative error < 2^-22 / (1 - e^-0.1) ~ 1.3e-6 at the cut, falling beyond).
__device__ __forceinline__ float one_minus_exp_neg(float x) {
  const float s = x * (1.0f + x * (-0.5f + x * (1.0f / 6.0f + x * (-1.0f / 24.0f + x * (1.0f / 120.0f)))));
  const float e = 1.0f - __expf(-x);
  return x < 0.1f ? s : e;  // a select, not a branch
}

// sin(t) for the per-step phase increments of the frequency-domain walk (|t| ~ 1e-3): the
// series to t^5 below 0.1 (relative error < t^6 / 5040 < 2e-10), the fast sine above.
__device__ __forceinline__ float sin_small(float t) {
  if (fabsf(t) < 0.1f) {
    const float t2 = t * t;
    return t * (1.0f + t2 * (-1.0f / 6.0f + t2 * (1.0f / 120.0f)));
  }
  return __sinf(t);
}

// The FP32 walks carry the phase reduced to [0, 2 pi) so that the fast sine and cosine
// keep their absolute accuracy (cos and sin of the reduced angle are those of the phase).
constexpr float kTwoPiF = 6.28318530717958647692f;
__device__ __forceinline__ float wrap_phase(float p) { return p >= kTwoPiF ? p - kTwoPiF : p; }

// The tetrahedral tracking kernel flushes subnormals (its unit's -ftz flag): right for its
// reciprocals, roots, logarithms and exponentials, whose arguments and results of that size
// contribute nothing, and not for the deposits.  With an absorption coefficient down to 1e-38 the
// depth mua ds of a step is subnormal, and so may the coefficient itself be, while their sum over a
// visit to an element is what the normalisation divides by it.  These operations, and the test of
// the coefficient, keep subnormals at the price of the flushing ones (1e7 photons on the 648k-tet
// phantom 181.7 and 181.8 ms, frequency domain at 1e6 30.9 and 31.2).
__device__ __forceinline__ float keep_mul(float a, float b) {
  float r;
  asm("mul.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float keep_add(float a, float b) {
  float r;
  asm("add.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float keep_fma(float a, float b, float c) {
  float r;
  asm("fma.rn.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// (a path left of 1e37 mm in an element that hardly scatters, times 1e-38 on entering one that does)
__device__ __forceinline__ float keep_div(float a, float b) {
  float r;
  asm("div.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ bool keep_positive(float x) { return __float_as_uint(x) - 1u < 0x7f800000u; }  // x > 0
__device__ __forceinline__ float one_minus_exp_neg_keep(float x) {
  const float s = keep_mul(x, 1.0f + x * (-0.5f + x * (1.0f / 6.0f + x * (-1.0f / 24.0f + x * (1.0f / 120.0f)))));
  const float e = 1.0f - __expf(-x);
  return x < 0.1f ? s : e;
}
__device__ __forceinline__ float sin_small_keep(float t) {
  if (fabsf(t) < 0.1f) {
    const float t2 = t * t;
    return keep_mul(t, 1.0f + t2 * (-1.0f / 6.0f + t2 * (1.0f / 120.0f)));
  }
  return __sinf(t);
}

// distance to the next interaction, -log(U) / mus, with U in (0, 1).  The fast logarithm's
// absolute error (~1e-7) can make -log(U) of a U within 1e-7 of 1 come out at or just
// below zero; such a draw is an interaction at once, as it nearly is exactly.  The floor is
// 1e-30 rather than 0 so that a vacuum element (mus = 0) still gets an infinite path, as
// the reference's -log(U) / 0 does, and never 0 / 0.
__device__ __forceinline__ float free_path_f(float u, float mus) {
  return __fdividef(fmaxf(-__logf(u), 1e-30f), mus);
}

// =====================================================================================
// plain FP64 form
// =====================================================================================
// Bound by the FP64 pipe, which starts one warp instruction in about 19 cycles of the SM; with
// the reference's operation sequence taken literally a warp's step needed about 450 of them
// (Moller-Trumbore face by face, the library's exp, log, sin, cos, sqrt and divisions).  Here
// FP64 is spent where the state is: 25 operations for a step of which 1 belongs to the scatter.
//   exit face  picked in FP32 from planes about vertex 0, when it is certain by margins above
//              every FP32 rounding; else (2e-4 of the steps) by Moller-Trumbore, face by face as
//              in the reference.  Its distance is one FP64 quotient n . (v - p) / n . d, with no
//              more rounding than Moller-Trumbore's.
//   samples    log, sine, cosine, the deposit's factor, the scattering angle and the turned
//              direction on the integer pipe (fixed64.hpp); the last two by 48 FP64 operations of
//              3D before (23 in 2D), with errors 3 to 100 times as large.
//   quotients and roots from FP32 first values.
// 1e5 photons on the phantom 313 -> 102 -> 72 ms (571 before lanes were packed as well), 1e3 there
// 46.8 -> 31.7, 20 000 in the 48k-tet cube 33.7 -> 25.9 (102, 46.8 and 33.7 with the scatter in
// FP64).  The phantom's run ends in walks of 14 000 steps, with the issue slots 20 % and the FP64
// pipe 19 % busy: the latency of some 1000 instructions a step.  Against 80-bit arithmetic the
// elements' median error in the cube is 5e-14; with the library's functions it was 2.6e-13.
template <bool FD, class R>
struct Walk3D64 {
  static constexpr bool kBuffered = false;  // a block's words are drawn again rather than carried
  static constexpr bool kPack = true;
  static constexpr bool kCap32 = true;
  static constexpr bool kDefer = true;
  __device__ __forceinline__ bool pending() const { return pend != 0; }
  static constexpr int kMinBlocks = 2;
  static constexpr bool kStaged = false;
  static constexpr bool kLaunchLoss = false;
  Stage stage;
  using Tr = typename TraceFor<R>::type;
  double pos[3], dir[3];
  double w, prop, cph, sph;
  double mua, mus, g, nidx, imus;  // imus = 1 / mus
  uint64_t ig;                     // hg_inverse(g)
  double acc, accI;
  uint64_t turn;  // phase in 2^-64 turns
  int el, curface;
  int32_t nsteps;
  int pend;  // event to come: 1 + the face crossed, 0 none
  Tr tr;

  // moves the photon's state between lanes (Packer)
  template <class F> __device__ __forceinline__ void move(const F &f) {
    if constexpr (FD) f(pos[0], pos[1], pos[2], dir[0], dir[1], dir[2], w, prop, mua, mus, g, nidx, imus, ig, acc, turn, cph, sph, accI, el, curface, nsteps, pend);
    else f(pos[0], pos[1], pos[2], dir[0], dir[1], dir[2], w, prop, mua, mus, g, nidx, imus, ig, acc, el, curface, nsteps, pend);
  }

  __device__ __forceinline__ static const TetRec *recs(const JobDev &J) { return reinterpret_cast<const TetRec *>(J.geom); }
  __device__ __forceinline__ static const Tet64 *verts(const JobDev &J) { return reinterpret_cast<const Tet64 *>(recs(J) + J.Ne); }

  __device__ __forceinline__ void optics(const JobDev &J, int e, double &a, double &s, double &gg, double &nn) const {
    const double2 *o = reinterpret_cast<const double2 *>(J.optics) + 2 * (int64_t)(e & J.opt_mask);
    const double2 o0 = __ldg(o), o1 = __ldg(o + 1);
    a = o0.x; s = o0.y; gg = o1.x; nn = o1.y;
  }

  __device__ void launch(const JobDev &J, R &rng, int64_t q) {
    tr.begin(J, q);
    create_photon_3d<false>(J, rng, pos, dir, el, curface);
    w = 1.0;
    if (FD) {
      turn = J.turn0;
      sincos_turn(turn, sph, cph);
    }
    optics(J, el, mua, mus, g, nidx);
    nidx = index_at_launch(nidx);
    imus = fast_rcp(mus);
    ig = hg_inverse(g);
    prop = neg_log_open(rng.next()) * imus;  // the outer loop's first draw, MC3D.hpp:1458
    acc = accI = 0.0;
    nsteps = 0;
    pend = 0;
  }

  __device__ __forceinline__ void flush(const JobDev &J) {
    add_d(J, J.ER + el, acc);
    if (FD) add_d(J, J.EI + el, accI);
    acc = accI = 0.0;
  }

  __device__ __forceinline__ bool die(const JobDev &J, int64_t ev) {
    flush(J);
    tr.put(ev);
    tr.end();
    return false;
  }

  // What a scatter event draws: the polar cosine and sine, the azimuth's (in units of 2^-60), the
  // free path after it.
  struct Event { int64_t ct, st, cp, sp; double path; };

  // ScatterPhoton, MC3D.hpp:1297-1315, from the words u, without the round trip through the
  // angle: the reference draws theta = acos(c) from the HG inverse CDF c and takes sin and cos
  // of it; here cos theta is c itself and sin theta = sqrt(1 - c^2) (|c| > 1 from rounding at
  // the CDF's ends gives a NaN sine, as acos gives a NaN angle).
  __device__ __forceinline__ Event draw_event(uint3 u) const {
    Event e;
    e.ct = hg_cosine(u.x, g, ig);
    const Split60 c = split60(e.ct);
    const int64_t s2 = kOne60 - mul60(c, c);
    const Root60 s = sqrt60(s2);
    e.st = s2 > 0 ? s.r >> s.k : 0;
    if (s2 < 0) e.ct = kNoCosine;
    // the azimuth 2 pi u / (2^32 - 1): u 2^32 + u in 2^-64 turns, to one of them
    sincos_turn_fixed(((uint64_t)u.y << 32) | u.y, e.sp, e.cp);
    e.sp >>= 2;
    e.cp >>= 2;
    e.path = neg_log_open(u.z) * imus;
    return e;
  }

  // the rotation of ScatterPhoton, MC3D.hpp:1316-1340; false: not for fixed point
  __device__ __forceinline__ bool rotate(const Event &e) {
    const uint32_t top = max(mag_of(dir[0]), max(mag_of(dir[1]), mag_of(dir[2])));
    if (e.ct == kNoCosine || top > 0x3ff00000u) return false;
    const int64_t z6 = fixed60_of(dir[2]);
    const Split60 ct = split60(e.ct), st = split60(e.st), cp = split60(e.cp), sp = split60(e.sp), dz = split60(z6);
    int64_t v[3];
    if ((__double_as_longlong(dir[2]) & 0x7fffffffffffffffll) > __double_as_longlong(0.999)) {
      v[0] = mul60(st, cp);
      v[1] = mul60(st, sp);
      v[2] = z6 > 0 ? e.ct : -e.ct;
    } else {
      const Split60 dx = split60(fixed60_of(dir[0])), dy = split60(fixed60_of(dir[1]));
      const Root60 q = sqrt60(kOne60 - mul60(dz, dz));  // sqrt(1 - z^2), k <= 4
      const Split60 isq = split60(q.y), zc = split60(mul60(dz, cp));
      const Split60 ux = split60(mul60(dx, isq) << q.k), uy = split60(mul60(dy, isq) << q.k);
      v[0] = dot60(st, split60(dot60(ux, zc, neg60(uy), sp)), dx, ct);
      v[1] = dot60(st, split60(dot60(uy, zc, ux, sp)), dy, ct);
      v[2] = dot60(dz, ct, split60(-mul60(st, cp)), split60(q.r >> q.k));
    }
    if (!unit60(v, 3)) return false;
    dir[0] = double_of_60(v[0]); dir[1] = double_of_60(v[1]); dir[2] = double_of_60(v[2]);
    curface = -1;
    return true;
  }

  // Both in FP64, for what fixed point does not hold: |g| near 1 or nearly 0, a direction that is
  // not a unit vector yet, a cosine beyond 1.
  struct Dir { double x, y, z; };
  __device__ __noinline__ static Dir scatter_d(uint32_t ux, uint32_t uy, double g, double dx, double dy, double dz) {
    const double c0 = fma(word_d(ux), 2.0 / 4294967295.0, -1.0);  // 2 xi - 1, the isotropic cosine
    const double D = fma(g, c0, 1.0);                              // 1 - g (1 - 2 xi)
    const double q = div_near(fma(-g, g, 1.0), D, f32_of(D));
    double ct = fma(-q, q, fma(g, g, 1.0)) * (0.5 * fast_rcp(g));
    ct = ux == 0u ? -1.0 : ux == 0xffffffffu ? 1.0 : ct;  // theta = (1 - xi) pi at xi in {0, 1}
    ct = (__double_as_longlong(g) << 1) == 0 ? c0 : ct;
    const double t2 = fma(-ct, ct, 1.0);
    const float t2f = f32_of(t2);
    double st, y, sp, cp;
    sqrt_near(t2, t2f, st, y);
    st = t2f > 0.0f ? st : t2f == 0.0f ? 0.0 : __longlong_as_double(0x7ff8000000000000ll);
    sincos_turn(((uint64_t)uy << 32) | uy, sp, cp);
    double nx, ny, nz;
    if (fabs(dz) > 0.999) {
      nx = st * cp;
      ny = st * sp;
      nz = dz > 0.0 ? ct : -ct;
    } else {
      double sq, isq;
      const double s2 = fma(-dz, dz, 1.0);
      sqrt_near(s2, f32_of(s2), sq, isq);
      const double a = st * isq, zc = dz * cp;
      nx = fma(a, fma(dx, zc, -(dy * sp)), dx * ct);
      ny = fma(a, fma(dy, zc, dx * sp), dy * ct);
      nz = fma(-st * cp, sq, dz * ct);
    }
    const double s = unit_scale(fma(nx, nx, fma(ny, ny, nz * nz)));
    return Dir{nx * s, ny * s, nz * s};
  }

  // FresnelPhoton at a face with normal nor, of either orientation and any length
  // (MC3D.hpp:1365-1447); true if reflected
  __device__ __forceinline__ bool fresnel(R &rng, const double *nor, double nout, int nf, bool inside) {
    double n0 = __ldg(nor), n1 = __ldg(nor + 1), n2 = __ldg(nor + 2);
    const float f0 = f32_of(n0), f1 = f32_of(n1), f2 = f32_of(n2);
    const Choice choice = fresnel_choice(rng, __fdividef(f32_of(nidx), f32_of(nout)),
                                         f0 * f32_of(dir[0]) + f1 * f32_of(dir[1]) + f2 * f32_of(dir[2]),
                                         f0 * f0 + f1 * f1 + f2 * f2);
    if (choice.what == Choice::kPass && !inside) return false;
    const double nn = fma(n0, n0, fma(n1, n1, n2 * n2)), dn = fma(dir[0], n0, fma(dir[1], n1, dir[2] * n2));
    if (choice.what == Choice::kReflect) {
      const double k = -2.0 * div_near(dn, nn, f32_of(nn));
      dir[0] = fma(k, n0, dir[0]); dir[1] = fma(k, n1, dir[1]); dir[2] = fma(k, n2, dir[2]);
      curface = nf;
      return true;
    }
    const double nipnt = fast_div(nidx, nout);
    double len, inv;
    fast_sqrt(nn, len, inv);
    n0 *= inv; n1 *= inv; n2 *= inv;
    const double costhi = -dn * inv;
    double costht = 0.0;
    if (fresnel_reflects_d(rng, choice, nipnt, costhi, costht)) {
      const double k = 2.0 * costhi;
      dir[0] = fma(k, n0, dir[0]); dir[1] = fma(k, n1, dir[1]); dir[2] = fma(k, n2, dir[2]);
      curface = nf;
      return true;
    }
    const double m = (costhi > 0.0) ? (nipnt * costhi - costht) : (nipnt * costhi + costht);
    dir[0] = fma(nipnt, dir[0], m * n0); dir[1] = fma(nipnt, dir[1], m * n1); dir[2] = fma(nipnt, dir[2], m * n2);
    return false;
  }

  // WhichFace, MC3D.hpp:1006-1057: faces (0,1,2), (0,1,3), (0,2,3), (1,2,3) in order, skipping curface
  struct Exit { double dist; int nf; };
  __device__ __noinline__ static Exit which_face(const Tet64 *T, double px, double py, double pz, double dx, double dy,
                                                 double dz, int curface) {
    const double *v = &T->v[0][0];
    const double pos[3] = {px, py, pz}, dir[3] = {dx, dy, dz};
    double dist = 0.0;
    if (curface != 0 && ray_tri(pos, dir, v, v + 3, v + 6, dist) && dist > 0.0) return Exit{dist, 0};
    if (curface != 1 && ray_tri(pos, dir, v, v + 3, v + 9, dist) && dist > 0.0) return Exit{dist, 1};
    if (curface != 2 && ray_tri(pos, dir, v, v + 6, v + 9, dist) && dist > 0.0) return Exit{dist, 2};
    if (curface != 3 && ray_tri(pos, dir, v + 3, v + 6, v + 9, dist) && dist > 0.0) return Exit{dist, 3};
    return Exit{0.0, -1};
  }

  // The exit face and the distance to it; nbr: the record's neighbours.
  //
  // With r = p - v0 in FP64, FP32 has num_f = off_f - n_f . r (the distance to plane f) within
  // en = 1e-6 |r|_1 (5e-7 from the roundings of n, r and the sum) and nd_f = n_f . d within
  // ed = 1e-6 |d|_1.  The face that the ray leaves through is certain when num > en and
  // nd > 8 ed there, every other face's plane is met later by a margin, num_g nd - num nd_g >
  // 4e-6 |r|_1 |d|_1, and the ray starts clearly inside every other plane but the one it
  // entered by (which the reference does not test): then Moller-Trumbore finds u and v well
  // inside that face, and well outside the others or behind the photon.
  __device__ __forceinline__ int exit_face(const JobDev &J, double &dist, int4 &nbr) const {
    const TetRec *T = recs(J) + el;
    const double2 a0 = __ldg(reinterpret_cast<const double2 *>(T->v0));
    const double2 a1 = __ldg(reinterpret_cast<const double2 *>(T->v0) + 1);
    const float4 q0 = __ldg(reinterpret_cast<const float4 *>(T->nf)), q1 = __ldg(reinterpret_cast<const float4 *>(T->nf) + 1),
                 q2 = __ldg(reinterpret_cast<const float4 *>(T->nf) + 2);
    nbr = __ldg(reinterpret_cast<const int4 *>(T->nbr));
    const double rx = pos[0] - a0.x, ry = pos[1] - a0.y, rz = pos[2] - a1.x;
    const float fx = f32_of(rx), fy = f32_of(ry), fz = f32_of(rz), off = __ldg(&T->off_size);
    const float dx = f32_of(dir[0]), dy = f32_of(dir[1]), dz = f32_of(dir[2]);
    const float n[4][3] = {{q0.x, q0.y, q0.z}, {q0.w, q1.x, q1.y}, {q1.z, q1.w, q2.x}, {q2.y, q2.z, q2.w}};
    const float rs = fabsf(fx) + fabsf(fy) + fabsf(fz) + fabsf(off), ds = fabsf(dx) + fabsf(dy) + fabsf(dz);
    const float en = 1e-6f * rs, ed = 8e-6f * ds, margin = 4e-6f * rs * ds;
    float num[4], nd[4], bnum = 1.0f, bnd = 0.0f;
    int nf = -1;
#pragma unroll
    for (int f = 0; f < 4; f++) {
      num[f] = (f == 3 ? off : 0.0f) - (n[f][0] * fx + n[f][1] * fy + n[f][2] * fz);
      nd[f] = n[f][0] * dx + n[f][1] * dy + n[f][2] * dz;
      const bool better = f != curface && nd[f] > ed && num[f] * bnd < bnum * nd[f];
      bnum = better ? num[f] : bnum;
      bnd = better ? nd[f] : bnd;
      nf = better ? f : nf;
    }
    bool sure = nf >= 0 && bnum > en;
#pragma unroll
    for (int f = 0; f < 4; f++)
      sure = sure && (f == nf || (num[f] * bnd - bnum * nd[f] > margin && (f == curface || num[f] > en)));
    const double *m = T->n[nf < 0 ? 0 : nf];
    const double m0 = __ldg(m), m1 = __ldg(m + 1), m2 = __ldg(m + 2);
    const double dn = fma(m2, dir[2], fma(m1, dir[1], m0 * dir[0]));
    const double nr = fma(m2, rz, fma(m1, ry, m0 * rx));
    const float dnf = f32_of(dn);
    dist = div_near((nf == 3 ? a1.y : 0.0) - nr, dn, dnf);
    if (sure && f32_safe(dnf)) return nf;
    const Exit e = which_face(verts(J) + el, pos[0], pos[1], pos[2], dir[0], dir[1], dir[2], curface);
    dist = e.dist;
    return e.nf;
  }

  __device__ __forceinline__ bool step(const JobDev &J, R &rng, int32_t cap, uint32_t &n_scat) {
    if (rng.exhausted()) { job_count(J, kJcTapeEnd); return die(J, kEvTapeEnd); }
    double dist;
    int4 nb;
    const int nf = exit_face(J, dist, nb);
    if (nf < 0) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, w);
      return die(J, kEvLost);
    }
    nsteps++;
    // both lengths are positive, so their bits compare as they do (a NaN path never ends here)
    const bool ends = __double_as_longlong(prop) <= __double_as_longlong(dist);
    const double ds = ends ? prop : dist;
#pragma unroll
    for (int c = 0; c < 3; c++) pos[c] = fma(dir[c], ds, pos[c]);
    tr.put(el);
    // element fluence, MC3D.hpp:1479-1526
    if (!FD) {
      if (positive(mua)) {
        const double dep = absorbed_part(mua, ds) * w;
        acc += dep;
        w -= dep;
      } else {
        acc = fma(w, ds, acc);
        if (mua != 0.0) w *= exp(-mua * ds);
      }
    } else {
      const double att = positive(mua) ? 1.0 - absorbed_part(mua, ds) : exp(-mua * ds);
      turn += fixed_of_double(J.k_turn * nidx * ds);
      double sn, cn;
      sincos_turn(turn, sn, cn);
      acc = fma(w, fma(-cn, att, cph), acc);
      accI = fma(w, fma(sn, att, -sph), accI);
      cph = cn; sph = sn;
      w *= att;
    }
    if (ends) {
      if (positive(mus)) {
        const Event ev = draw_event(rng.peek3());
        if (!rotate(ev)) {
          const uint3 u = rng.peek3();
          const Dir d = scatter_d(u.x, u.y, g, dir[0], dir[1], dir[2]);
          dir[0] = d.x; dir[1] = d.y; dir[2] = d.z;
          curface = -1;
        }
        rng.take(3);
        prop = ev.path;
        n_scat++;
      } else {
        rng.align();
        prop = neg_log_open(rng.next()) * imus;
      }
    } else {
      prop -= dist;
      const int nextel = nf == 0 ? nb.x : nf == 1 ? nb.y : nf == 2 ? nb.z : nb.w;
      if (!cross_on(J, nextel)) {
        pend = 1 + nf;
        return true;
      }
    }
    if (nsteps >= cap && !rng.exhausted()) {  // a tape that ends here is reported as that
      job_count(J, kJcCapped); job_ledger(J, kLgLost, w);
      return die(J, kEvCapped);
    }
    return true;
  }

  // The common crossing: into an element that scatters, no index jump, weight above the roulette
  // threshold.
  __device__ __forceinline__ bool cross_on(const JobDev &J, int nextel) {
    if ((unsigned)nextel >= (unsigned)J.Ne) return false;
    double mua2, mus2, g2, n2;
    optics(J, nextel, mua2, mus2, g2, n2);
    if (!positive(mus) || differ(nidx, n2) || below(w, kWeight0)) return false;
    const int4 nb2 = __ldg(reinterpret_cast<const int4 *>((recs(J) + nextel)->nbr));
    const int f2 = nb2.x == el ? 0 : nb2.y == el ? 1 : nb2.z == el ? 2 : nb2.w == el ? 3 : -1;
    if (f2 < 0) return false;
    if (differ(mus2, mus)) {
      prop *= mus / mus2;  // x (mus / mus) == x
      imus = fast_rcp(mus2);
    }
    if (differ(g2, g)) ig = hg_inverse(g2);
    flush(J);
    curface = f2;
    el = nextel;
    mua = mua2; mus = mus2; g = g2; nidx = n2;
    return true;
  }

  // What else lies behind face pend - 1, for several lanes of a warp together.
  __device__ __forceinline__ bool event(const JobDev &J, R &rng, int32_t cap, uint32_t &) {
    const int nf = pend - 1;
    pend = 0;
    const bool on = cross(J, rng, nf, __ldg((recs(J) + el)->nbr + nf));
    if (on && nsteps >= cap && !rng.exhausted()) {  // a tape that ends here is reported as that
      job_count(J, kJcCapped); job_ledger(J, kLgLost, w);
      return die(J, kEvCapped);
    }
    return on;
  }

  // the boundary, or the next element, behind face nf
  __device__ __forceinline__ bool cross(const JobDev &J, R &rng, int nf, int nextel) {
    const double *nor = (recs(J) + el)->n[nf];
    if (nextel >= J.Ne) {  // open face: the reference would index past its arrays here
      job_count(J, kJcLoss); job_ledger(J, kLgLost, w);
      return die(J, kEvLost);
    }
    const bool inside = nextel >= 0;
    const int ib = -1 - nextel;
    double mua2 = 0.0, mus2 = 0.0, g2 = 0.0, n2;
    if (inside) {
      optics(J, nextel, mua2, mus2, g2, n2);
    } else {
      if (is_mirror(__ldg(J.bctype + ib))) {  // MirrorPhoton(ib) with Normal(ib)
        const double *bn = J.bnorm + 4 * (int64_t)ib;
        const double cdot = bn[0] * dir[0] + bn[1] * dir[1] + bn[2] * dir[2];
#pragma unroll
        for (int c = 0; c < 3; c++) dir[c] -= 2.0 * cdot * bn[c];
        curface = nf;
        return true;
      }
      n2 = __ldg(J.bcn + ib);
    }
    const bool vacuum = inside && at_most_zero(mus) && positive(mus2);
    const bool jump = inside ? differ(nidx, n2) : positive(n2);
    const bool light = inside && below(w, kWeight0);
    if (vacuum || jump || light) {
      rng.reload();
      if (vacuum) prop = neg_log_open(rng.next()) / mus2;
      if (light) {
        if (!closed_at_most(rng, kChance)) {
          job_count(J, kJcRoulette); job_ledger(J, kLgRouletteKill, w);
          return die(J, kEvRoulette);
        }
        const double up = w / kChance;
        job_ledger(J, kLgRouletteGain, up - w);
        w = up;
      }
      if (jump && fresnel(rng, nor, n2, nf, inside)) return true;
    }
    if (!inside) {
      flush(J);
      if (!FD) add_d(J, J.EBR + ib, w);
      else { add_d(J, J.EBR + ib, w * cph); add_d(J, J.EBI + ib, -(w * sph)); }
      tr.put(-1 - (int64_t)ib);
      tr.end();
      return false;
    }
    // reverse-face lookup, MC3D.hpp:1616-1628
    const int4 nb2 = __ldg(reinterpret_cast<const int4 *>((recs(J) + nextel)->nbr));
    const int f2 = nb2.x == el ? 0 : nb2.y == el ? 1 : nb2.z == el ? 2 : nb2.w == el ? 3 : -1;
    if (differ(mus2, mus)) {
      if (!vacuum) prop *= mus / mus2;  // x (mus / mus) == x
      imus = fast_rcp(mus2);
    }
    if (f2 < 0) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, w);
      return die(J, kEvLost);
    }
    if (differ(g2, g)) ig = hg_inverse(g2);
    flush(J);
    curface = f2;
    el = nextel;
    mua = mua2; mus = mus2; g = g2; nidx = n2;
    return true;
  }
};

// The plain form with the reference's operation sequence taken literally, for jobs whose
// scattering or index changes across most faces (rough_optics): there a photon's remaining path
// is rescaled at nearly every crossing, rounding differences grow from crossing to crossing, and
// walks of thousands of steps keep the reference's steps only with the reference's operations.
template <bool FD, class R>
struct Walk3D64L {
  static constexpr bool kBuffered = true;  // words left in a block are carried from step to step
  static constexpr bool kPack = true;
  static constexpr bool kCap32 = false;
  static constexpr bool kDefer = false;
  static constexpr int kMinBlocks = 2;  // ~125 registers: 2 CTAs of 256 per SM
  static constexpr bool kStaged = false;
  static constexpr bool kLaunchLoss = false;
  Stage stage;
  using Tr = typename TraceFor<R>::type;
  double pos[3], dir[3];
  double w, prop, phase, cph, sph;
  double mua, mus, g, nidx;
  double acc, accI;
  int el, curface;
  int64_t nsteps;
  Tr tr;

  // moves the photon's state between lanes (Packer)
  template <class F> __device__ __forceinline__ void move(const F &f) {
    if constexpr (FD) f(pos[0], pos[1], pos[2], dir[0], dir[1], dir[2], w, prop, mua, mus, g, nidx, acc, phase, cph, sph, accI, el, curface, nsteps);
    else f(pos[0], pos[1], pos[2], dir[0], dir[1], dir[2], w, prop, mua, mus, g, nidx, acc, el, curface, nsteps);
  }

  __device__ __forceinline__ static const Tet64 *tets(const JobDev &J) { return reinterpret_cast<const Tet64 *>(J.geom); }
  __device__ __forceinline__ void optics(const JobDev &J, int e, double &a, double &s, double &gg, double &nn) const {
    const double2 *o = reinterpret_cast<const double2 *>(J.optics) + 2 * (int64_t)(e & J.opt_mask);
    const double2 o0 = __ldg(o), o1 = __ldg(o + 1);
    a = o0.x; s = o0.y; gg = o1.x; nn = o1.y;
  }

  __device__ void launch(const JobDev &J, R &rng, int64_t q) {
    tr.begin(J, q);
    create_photon_3d<true>(J, rng, pos, dir, el, curface);
    w = 1.0;
    phase = J.phase0;
    if (FD) sincos(phase, &sph, &cph);
    optics(J, el, mua, mus, g, nidx);
    prop = -log(unif_open(rng)) / mus;  // the outer loop's first draw, MC3D.hpp:1458
    acc = accI = 0.0;
    nsteps = 0;
  }

  __device__ __forceinline__ void flush(const JobDev &J) {
    add_d(J, J.ER + el, acc);
    if (FD) add_d(J, J.EI + el, accI);
    acc = accI = 0.0;
  }

  __device__ __forceinline__ int die(const JobDev &J, int64_t ev) {
    flush(J);
    tr.put(ev);
    tr.end();
    return kDied;
  }

  __device__ void scatter(const JobDev &J, R &rng) {
    // ScatterPhoton, MC3D.hpp:1297-1340, without the round trip through the angle: the
    // reference draws theta = acos(c) from the HG inverse CDF c and takes sin and cos of it;
    // here cos theta is c itself and sin theta = sqrt(1 - c^2) (the same values to a few
    // ulps; |c| > 1 from rounding at the CDF's ends gives a NaN sine, as acos gives a NaN
    // angle), and the azimuth's sine and cosine come from sincospi(2 U).  The replays still
    // visit the reference's elements bit for bit; the FP64 pipe that bounds this form does
    // 10% less work.
    double ct;
    if (g != 0.0) {
      double xi = unif_closed(rng);
      if ((0.0 < xi) && (xi < 1.0)) {
        double g2 = g * g;
        double q = (1.0 - g2) / (1.0 - g * (1.0 - 2.0 * xi));
        ct = (1.0 + g2 - q * q) / (2.0 * g);
      } else {
        ct = xi > 0.5 ? 1.0 : -1.0;
      }
    } else {
      ct = 2.0 * unif_closed(rng) - 1.0;
    }
    const double st = sqrt(1.0 - ct * ct);
    double sp, cp;
    sincospi(2.0 * unif_closed(rng), &sp, &cp);
    double dxn, dyn, dzn;
    if (fabs(dir[2]) > 0.999) {
      dxn = st * cp;
      dyn = st * sp;
      dzn = dir[2] * ct / fabs(dir[2]);
    } else {
      double sq = sqrt(1.0 - dir[2] * dir[2]);
      const double isq = 1.0 / sq;
      dxn = st * (dir[0] * dir[2] * cp - dir[1] * sp) * isq + dir[0] * ct;
      dyn = st * (dir[1] * dir[2] * cp + dir[0] * sp) * isq + dir[1] * ct;
      dzn = -st * cp * sq + dir[2] * ct;
    }
    // one reciprocal for the three components (and one for the two 1 / sq above) instead of
    // a division each: the same direction to an ulp, 4.5% less FP64 work per photon
    const double inorm = 1.0 / sqrt(dxn * dxn + dyn * dyn + dzn * dzn);
    dir[0] = dxn * inorm; dir[1] = dyn * inorm; dir[2] = dzn * inorm;
    curface = -1;
  }

  // FresnelPhoton with the unoriented face normal nor (MC3D.hpp:1365-1447); true if reflected
  __device__ bool fresnel(R &rng, const double nor[3], double nipnt, int nf) {
    double costhi = -(dir[0] * nor[0] + dir[1] * nor[1] + dir[2] * nor[2]);
    double costht = 0.0;
    if (fresnel_reflects_angles(rng, nipnt, costhi, costht)) {
#pragma unroll
      for (int c = 0; c < 3; c++) dir[c] += 2.0 * costhi * nor[c];
      curface = nf;
      return true;
    }
    double m = (costhi > 0.0) ? (nipnt * costhi - costht) : (nipnt * costhi + costht);
#pragma unroll
    for (int c = 0; c < 3; c++) dir[c] = nipnt * dir[c] + m * nor[c];
    return false;
  }

  __device__ int step(const JobDev &J, R &rng, int64_t max_steps) {
    if (rng.exhausted()) { job_count(J, kJcTapeEnd); return die(J, kEvTapeEnd); }
    if (nsteps >= max_steps) {
      job_count(J, kJcCapped); job_ledger(J, kLgLost, w);
      return die(J, kEvCapped);
    }
    const Tet64 *T = tets(J) + el;
    double V[4][3];
    {
      const double2 *src = reinterpret_cast<const double2 *>(T->v);
#pragma unroll
      for (int i = 0; i < 6; i++) {
        double2 d2 = __ldg(src + i);
        reinterpret_cast<double *>(V)[2 * i] = d2.x;
        reinterpret_cast<double *>(V)[2 * i + 1] = d2.y;
      }
    }
    const int4 nb = __ldg(reinterpret_cast<const int4 *>(T->nbr));
    // WhichFace: faces (0,1,2), (0,1,3), (0,2,3), (1,2,3) in order, skipping curface
    double dist = 0.0;
    int nf = -1;
    if (curface != 0 && ray_tri(pos, dir, V[0], V[1], V[2], dist) && dist > 0.0) nf = 0;
    else if (curface != 1 && ray_tri(pos, dir, V[0], V[1], V[3], dist) && dist > 0.0) nf = 1;
    else if (curface != 2 && ray_tri(pos, dir, V[0], V[2], V[3], dist) && dist > 0.0) nf = 2;
    else if (curface != 3 && ray_tri(pos, dir, V[1], V[2], V[3], dist) && dist > 0.0) nf = 3;
    if (nf < 0) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, w);
      return die(J, kEvLost);
    }
    const int nextel = nf == 0 ? nb.x : nf == 1 ? nb.y : nf == 2 ? nb.z : nb.w;
    nsteps++;
    const double ds = fmin(prop, dist);
#pragma unroll
    for (int c = 0; c < 3; c++) pos[c] += dir[c] * ds;
    tr.put(el);
    // element fluence, MC3D.hpp:1479-1526
    const double att = exp(-mua * ds);
    if (!FD) {
      if (mua > 0.0) acc += (1.0 - att) * w;
      else acc += w * ds;
    } else {
      const double kds = J.k_scale * nidx * ds;
      double sn, cn;
      sincos(phase + kds, &sn, &cn);
      acc += w * (cph - cn * att);
      accI += w * (-sph + sn * att);
      phase += kds;
      cph = cn; sph = sn;
    }
    w *= att;
    prop -= ds;
    if (prop <= 0.0) {
      int res = kAlive;
      rng.align();
      if (mus > 0.0) { scatter(J, rng); res = kScattered; }
      prop = -log(unif_open(rng)) / mus;
      return res;
    }
    if (nextel < 0) {
      const int ib = -1 - nextel;
      const uint8_t bt = __ldg(J.bctype + ib);
      if (is_mirror(bt)) {  // MirrorPhoton(ib) with Normal(ib)
        const double *bn = J.bnorm + 4 * (int64_t)ib;
        double cdot = bn[0] * dir[0] + bn[1] * dir[1] + bn[2] * dir[2];
#pragma unroll
        for (int c = 0; c < 3; c++) dir[c] -= 2.0 * cdot * bn[c];
        curface = nf;
        return kAlive;
      }
      const double bcn = __ldg(J.bcn + ib);
      if (bcn > 0.0) {
        double nor[3];
        face_normal(V, nf, nor);
        if (fresnel(rng, nor, nidx / bcn, nf)) return kAlive;
      }
      flush(J);
      if (!FD) add_d(J, J.EBR + ib, w);
      else { add_d(J, J.EBR + ib, w * cph); add_d(J, J.EBI + ib, -(w * sph)); }
      tr.put(-1 - (int64_t)ib);
      tr.end();
      return kDied;
    }
    if (nextel >= J.Ne) {  // open face: the reference would index past its arrays here
      job_count(J, kJcLoss); job_ledger(J, kLgLost, w);
      return die(J, kEvLost);
    }
    double mua2, mus2, g2, n2;
    optics(J, nextel, mua2, mus2, g2, n2);
    if ((mus <= 0.0) && (mus2 > 0.0)) {
      prop = -log(unif_open(rng)) / mus2;
      if (w < kWeight0) {
        if (unif_closed(rng) > kChance) {
          job_count(J, kJcRoulette); job_ledger(J, kLgRouletteKill, w);
          return die(J, kEvRoulette);
        }
        job_ledger(J, kLgRouletteGain, w / kChance - w);
        w /= kChance;
      }
      if (nidx != n2) {
        double nor[3];
        face_normal(V, nf, nor);
        if (fresnel(rng, nor, nidx / n2, nf)) return kAlive;
      }
    } else {
      if (w < kWeight0) {
        if (unif_closed(rng) > kChance) {
          job_count(J, kJcRoulette); job_ledger(J, kLgRouletteKill, w);
          return die(J, kEvRoulette);
        }
        job_ledger(J, kLgRouletteGain, w / kChance - w);
        w /= kChance;
      }
      if (nidx != n2) {
        double nor[3];
        face_normal(V, nf, nor);
        if (fresnel(rng, nor, nidx / n2, nf)) return kAlive;
      }
      if (mus2 != mus) prop *= mus / mus2;  // x (mus / mus) == x: skip the division
    }
    // reverse-face lookup, MC3D.hpp:1616-1628
    const int4 nb2 = __ldg(reinterpret_cast<const int4 *>((tets(J) + nextel)->nbr));
    int f2 = nb2.x == el ? 0 : nb2.y == el ? 1 : nb2.z == el ? 2 : nb2.w == el ? 3 : -1;
    if (f2 < 0) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, w);
      return die(J, kEvLost);
    }
    flush(J);
    curface = f2;
    el = nextel;
    mua = mua2; mus = mus2; g = g2; nidx = n2;
    return kAlive;
  }

  // Normal(el, f), MC3D.hpp:408-457: the unit normal of the face through vertices a, b, c
  __device__ __forceinline__ static void normal_of(const double a[3], const double b[3], const double c[3],
                                                   double nor[3]) {
    double x1 = b[0] - a[0], y1 = b[1] - a[1], z1 = b[2] - a[2];
    double x2 = c[0] - a[0], y2 = c[1] - a[1], z2 = c[2] - a[2];
    double nx = y1 * z2 - z1 * y2, ny = z1 * x2 - x1 * z2, nz = x1 * y2 - y1 * x2;
    double norm = sqrt(nx * nx + ny * ny + nz * nz);
    nor[0] = nx / norm; nor[1] = ny / norm; nor[2] = nz / norm;
  }
  // Face f of the tetrahedron is (0,1,2), (0,1,3), (0,2,3) or (1,2,3).  The index computed
  // from f puts the step's vertex array in local memory (an L1-resident store of 96 B per
  // step); keeping it in registers to the end of the step (constant indices per case), or
  // reading the vertices again on the Fresnel paths, takes more registers, halves the
  // resident CTAs and measured 5-15 % slower on the phantom, whose FP64 pipe is the bound.
  __device__ __forceinline__ static void face_normal(const double V[4][3], int f, double nor[3]) {
    const int i0 = f == 3 ? 1 : 0;
    const int i1 = f == 0 ? 1 : f == 1 ? 1 : 2;
    const int i2 = f == 0 ? 2 : 3;
    normal_of(V[i0], V[i1], V[i2], nor);
  }
};

// =====================================================================================
// FP32 tracking form
// =====================================================================================
template <bool FD, class R>
struct Walk3D32 {
  // 4 CTAs of 256 per SM (64 registers): the walk is latency bound and 32 resident warps
  // per SM beat 24 (+7% on the 648k-tet phantom); 5 CTAs (48 registers) spill and lose
  static constexpr int kMinBlocks = 4;
  static constexpr bool kStaged = !FD;
  static constexpr bool kBuffered = false;  // a block's words are drawn again rather than carried
  static constexpr bool kPack = true;
  static constexpr bool kCap32 = true;
  static constexpr bool kDefer = false;
  using Tr = typename TraceFor<R>::type;
  float px, py, pz, dx, dy, dz;
  float w, prop, phase;
  float mua, mus, g, nidx;
  float acc, accI;
  int el;
  int32_t nsteps;
  bool outward;  // launched out through its own entry face
  Stage stage;   // shared-memory staging of ER deposits (continuous wave, single job)
  Tr tr;
  // Per-job forms (batched and served launches): the job's geometry and optics pointers,
  // optics index mask and element count, copied into registers at launch.  The one-job form
  // reads them as kernel-parameter operands; the per-job form would otherwise read them
  // from the job table on every step, the geometry pointer ahead of the record load on the
  // step's latency chain (2.7% on a two-job launch of the phantom; 56 -> 64 registers).
  const Tet32 *hg;
  const float4 *ho;
  int32_t hm, hne;

  // moves the photon's state between lanes (Packer)
  template <class F> __device__ __forceinline__ void move(const F &f) {
    if constexpr (FD) f(px, py, pz, dx, dy, dz, w, prop, mua, mus, g, nidx, acc, phase, accI, el, nsteps);
    else f(px, py, pz, dx, dy, dz, w, prop, mua, mus, g, nidx, acc, el, nsteps);
    if constexpr (!R::kOneJob) f(hg, ho, hm, hne);
  }

  __device__ __forceinline__ const Tet32 *geomp(const JobDev &J) const {
    if constexpr (R::kOneJob) return reinterpret_cast<const Tet32 *>(J.geom);
    else return hg;
  }
  __device__ __forceinline__ int32_t ne(const JobDev &J) const {
    if constexpr (R::kOneJob) return J.Ne;
    else return hne;
  }
  __device__ __forceinline__ float4 optics(const JobDev &J, int e) const {
    if constexpr (R::kOneJob) return __ldg(reinterpret_cast<const float4 *>(J.optics) + (e & J.opt_mask));
    else return __ldg(ho + (e & hm));
  }

  __device__ void launch(const JobDev &J, R &rng, int64_t q) {
    tr.begin(J, q);
    if constexpr (!R::kOneJob) {
      hg = reinterpret_cast<const Tet32 *>(J.geom);
      ho = reinterpret_cast<const float4 *>(J.optics);
      hm = J.opt_mask;
      hne = J.Ne;
    }
    float p[3], d[3];
    int cf;
    create_photon_3d_f(J, rng, p, d, el, cf);
    px = p[0]; py = p[1]; pz = p[2];
    dx = d[0]; dy = d[1]; dz = d[2];
    // The reference's WhichFace never tests the face a photon starts on, so a photon
    // launched pointing out of that face finds no exit and is lost (MC3D.hpp:1020-1056,
    // :1464-1468).  Keep that rule: the outward plane of the entry face decides.
    outward = false;
    if (cf >= 0) {
      const float4 pl = __ldg(reinterpret_cast<const float4 *>((reinterpret_cast<const Tet32 *>(J.geom) + el)->pl) + cf);
      outward = pl.x * dx + pl.y * dy + pl.z * dz > 0.0f;
    }
    w = 1.0f;
    phase = J.phase_f;
    float4 o = optics(J, el);
    mua = o.x; mus = o.y; g = o.z; nidx = o.w;
    prop = free_path_f(unif_open_f(rng), mus);
    acc = accI = 0.0f;
    nsteps = 0;
  }

  __device__ __forceinline__ void flush(const JobDev &J) {
    if (!FD) add_staged<R::kOneJob>(stage, J, el, acc);
    else add_f<R::kOneJob>(J, J.ER + el, acc);
    if (FD) add_f<R::kOneJob>(J, J.EI + el, accI);
    acc = accI = 0.0f;
  }

  __device__ __forceinline__ bool die(const JobDev &J, int64_t ev) {
    flush(J);
    tr.put(ev);
    tr.end();
    return false;
  }

  // Philox streams: a photon launched out through its own entry face is lost before its
  // first step (as the step would find it), so the step needs no test for it
  static constexpr bool kLaunchLoss = !R::kReplay;
  __device__ __forceinline__ bool lost_at_launch(const JobDev &J) {
    if (!outward) return false;
    job_count(J, kJcLoss); job_ledger(J, kLgLost, f2d_int(w));
    die(J, kEvLost);
    return true;
  }

  // What a scatter event draws: the polar cosine and sine, the azimuth's, the free path after it.
  struct Event { float ct, st, cp, sp, path; };

  // Henyey-Greenstein: cos(theta) from the inverse CDF, phi uniform (MC3D.hpp:1297-1315), and
  // the free path after the event, from the words u.  Selects, no branches.
  __device__ __forceinline__ Event draw_event(uint3 u) const {
    Event e;
    const float xi = closed_f(u.x);
    // (1 + g^2 - q^2) / (2 g) with q = (1 - g^2) / D, D = 1 - g + 2 g xi, over one
    // division: ((1 + g^2) D^2 - (1 - g^2)^2) / (2 g D^2)
    const float D = 1.0f - g + 2.0f * g * xi;
    const float a = 1.0f - g * g;
    const float D2 = D * D;
    float ct = __fdividef((1.0f + g * g) * D2 - a * a, 2.0f * g * D2);
    ct = xi > 0.0f && xi < 1.0f ? ct : xi > 0.5f ? 1.0f : -1.0f;  // theta = (1 - xi) pi at xi in {0, 1}
    ct = g != 0.0f ? ct : 2.0f * xi - 1.0f;
    e.ct = fminf(1.0f, fmaxf(-1.0f, ct));
    const float s2 = fmaxf(0.0f, 1.0f - e.ct * e.ct);
    e.st = s2 > 0.0f ? s2 * rsqrtf(s2) : 0.0f;
    // phi uniform on [-pi, pi] (the reference's [0, 2 pi] shifted; same distribution)
    __sincosf((float)kPi * (2.0f * closed_f(u.y) - 1.0f), &e.sp, &e.cp);
    e.path = free_path_f(open_f(u.z), mus);
    return e;
  }

  // the rotation of ScatterPhoton (MC3D.hpp:1316-1332)
  __device__ __forceinline__ void rotate(const Event &e) {
    const float ct = e.ct, st = e.st, cp = e.cp, sp = e.sp;
    float nx, ny, nz;
    {
      // the general rotation and the near-pole case (|dz| > 0.999) as selects, no branch
      const bool pole = fabsf(dz) > 0.999f;
      const float s2z = pole ? 1.0f : 1.0f - dz * dz;
      const float isq = rsqrtf(s2z);
      const float sq = s2z * isq;
      const float rx = st * (dx * dz * cp - dy * sp) * isq + dx * ct;
      const float ry = st * (dy * dz * cp + dx * sp) * isq + dy * ct;
      const float rz = -st * cp * sq + dz * ct;
      nx = pole ? st * cp : rx;
      ny = pole ? st * sp : ry;
      nz = pole ? (dz > 0.0f ? ct : -ct) : rz;  // cos(theta) times the sign of dz (not |cos| with that sign)
    }
    float in = rsqrtf(nx * nx + ny * ny + nz * nz);
    dx = nx * in; dy = ny * in; dz = nz * in;
  }

  // true if reflected; N is the outward unit normal of the face being crossed
  __device__ __forceinline__ bool fresnel(R &rng, float nx, float ny, float nz, float eta) {
    float dn = fmaf(dz, nz, fmaf(dx, nx, __fmul_rn(dy, ny)));  // > 0: leaving through the face
    float ci = fabsf(dn);
    float ct = 0.0f;
    if (fresnel_reflects_f(rng, eta, ci, ct)) {
      dx -= 2.0f * dn * nx; dy -= 2.0f * dn * ny; dz -= 2.0f * dn * nz;
      return true;
    }
    // refraction: d' = eta d + (ct - eta ci) s N with s the side the photon moves to
    float m = copysignf(ct, dn) - eta * dn;
    dx = fmaf(eta, dx, __fmul_rn(m, nx)); dy = fmaf(eta, dy, __fmul_rn(m, ny)); dz = fmaf(eta, dz, __fmul_rn(m, nz));
    return false;
  }

  __device__ __forceinline__ bool roulette(const JobDev &J, R &rng) {
    if (w < (float)kWeight0) {
      if (unif_closed_f(rng) > (float)kChance) {
        job_count(J, kJcRoulette); job_ledger(J, kLgRouletteKill, f2d_int(w));
        return true;
      }
      float nw = w * 10.0f;
      job_ledger(J, kLgRouletteGain, f2d_int(nw) - f2d_int(w));
      w = nw;
    }
    return false;
  }

  // One element step; false when the photon's walk has ended.  The kernel issues an
  // instruction in 74-78 % of its cycles, so its time follows the instructions of a warp's
  // step: control flow was a fifth of them.  Two branches are left on the common path, the
  // scatter and the crossing into a scattering element of the same index above the roulette
  // threshold; what either needs is drawn or tested at once, with selects, and everything
  // else branches off behind them (rare()).  Both branches run in nearly every step of a warp,
  // yet one straight run of instructions for both, with selects throughout, issues 12 % more
  // and measured slower (1e7 photons on the 648k-tet phantom: 228 ms).  Measured against the
  // form with a branch per case, both with flushed subnormals: 197.2 -> 194.4 ms there, 34.3 ->
  // 32.1 ms at 1e6 photons, 41.4 -> 40.2 ms for ten cubes in one launch; 202.2, 35.9 and
  // 42.7 ms before.
  // The products named __fmul_rn stay out of the fused multiply-adds that the compiler would
  // otherwise choose by the shape of the code around them: one photon, one rounding.
  __device__ __forceinline__ bool step(const JobDev &J, R &rng, int32_t cap, uint32_t &n_scat) {
    if constexpr (R::kReplay) {
      if (rng.exhausted()) { job_count(J, kJcTapeEnd); return die(J, kEvTapeEnd); }
      if (outward) {  // with Philox streams this is settled at launch
        job_count(J, kJcLoss); job_ledger(J, kLgLost, f2d_int(w));
        return die(J, kEvLost);
      }
    }
    const Tet32 *T = geomp(J) + el;
    const float4 *P4 = reinterpret_cast<const float4 *>(T->pl);
    const float4 p0 = __ldg(P4 + 0), p1 = __ldg(P4 + 1), p2 = __ldg(P4 + 2), p3 = __ldg(P4 + 3);
    // The neighbours: a launch of one job loads the one it crosses to when it crosses, a quarter of
    // the steps.  The gathers keep the L1 73 % busy, each 16-byte load of a warp taking 16 cycles
    // of it: 1e7 photons on the phantom 197.3 -> 187.3 ms, frequency domain at 1e6 33.9 -> 32.0,
    // the 48k-tet cube 6.74 -> 6.51.  Launches of several jobs, whose records come from the L2 more
    // often, load all four with the planes (ten cubes 41.5 ms, 42.3 the other way).
    int4 nb = make_int4(0, 0, 0, 0);
    if constexpr (!R::kOneJob) nb = __ldg(reinterpret_cast<const int4 *>(T->nbr));
    // exit: nearest face the direction points out of, as selects over all four faces (no
    // branch per face: fewer divergent regions and 6 fewer registers).  The distances
    // num / nd (nd > 0) are compared as num_f bnd < bnum nd_f, so that only the winning
    // face's quotient is computed: one reciprocal per step instead of four (bnd = 0 stands
    // for "none yet")
    float bnum = 1.0f, bnd = 0.0f;
    int nf = -1;
    {
      const float4 pl[4] = {p0, p1, p2, p3};
#pragma unroll
      for (int f = 0; f < 4; f++) {
        const float nd = pl[f].x * dx + pl[f].y * dy + pl[f].z * dz;
        const float num = pl[f].w - (pl[f].x * px + pl[f].y * py + pl[f].z * pz);
        const bool better = nd > 0.0f && num * bnd < bnum * nd;  // false where num is no number
        bnum = better ? num : bnum;
        bnd = better ? nd : bnd;
        nf = better ? f : nf;
      }
    }
    const float best = __fdividef(bnum, bnd);
    const bool found = nf >= 0;
    nsteps += found;
    const float dist = fmaxf(best, 0.0f);
    // a photon without an exit takes a step of length 0, which changes nothing of it
    const float ds = found ? fminf(prop, dist) : 0.0f;
    // a photon that leaves the element: fetch the next element's optics now, so that the
    // load runs under the deposit arithmetic
    int nextel = -1;
    float4 o2 = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (R::kOneJob) {
      if (!(prop <= dist)) nextel = __ldg(T->nbr + (nf & 3));  // also of a path that is no number
    } else {
      nextel = nf == 0 ? nb.x : nf == 1 ? nb.y : nf == 2 ? nb.z : nb.w;
    }
    if (prop > dist && (unsigned)nextel < (unsigned)ne(J)) o2 = optics(J, nextel);
    px += dx * ds; py += dy * ds; pz += dz * ds;
    if (found) tr.put(el);
    const float x = keep_mul(mua, ds);
    if (!FD) {
      const float dep = keep_mul(w, one_minus_exp_neg_keep(x));
      const bool takes = keep_positive(mua);
      acc = keep_add(acc, takes ? dep : keep_mul(w, ds));
      w = takes ? w - dep : w;
    } else {
      // w (cos phi - cos(phi + k ds) a) and w (-sin phi + sin(phi + k ds) a), a = exp(-mua ds),
      // written so that neither difference cancels: 1 - a cos(th) = (1 - a) + 2 a sin^2(th/2)
      const float th = keep_mul(keep_mul(J.k_scale_f, nidx), ds);
      const float om = one_minus_exp_neg_keep(x);
      const float a = 1.0f - om;
      const float sh = sin_small(0.5f * th);
      const float c1 = keep_fma(2.0f * a * sh, sh, om);
      const float s1 = keep_mul(a, sin_small_keep(th));
      float sp, cp;
      __sincosf(phase, &sp, &cp);
      acc = keep_fma(w, keep_fma(sp, s1, keep_mul(cp, c1)), acc);
      accI = keep_fma(w, keep_fma(cp, s1, -keep_mul(sp, c1)), accI);
      // fused in the one-job form only, as each has rounded it all along
      phase = wrap_phase(R::kOneJob ? fmaf(J.k_scale_f * nidx, ds, phase) : __fadd_rn(phase, th));
      w *= a;
    }
    prop -= ds;
    const bool going = found && nsteps < cap;  // neither lost nor at the step limit
    if (going && prop <= 0.0f && mus > 0.0f) {
      const Event ev = draw_event(rng.peek3());
      rotate(ev);
      rng.take(3);
      prop = ev.path;
      n_scat++;
      return true;
    }
    // the common crossing: interior, scattering medium, weight above the roulette threshold,
    // no index jump
    if (going && prop > 0.0f && (unsigned)nextel < (unsigned)ne(J) && mus > 0.0f && w >= (float)kWeight0 && nidx == o2.w) {
      if (o2.y != mus) prop = keep_mul(prop, keep_div(mus, o2.y));
      flush(J);
      el = nextel;
      mua = o2.x; mus = o2.y; g = o2.z;
      return true;
    }
    return rare(J, rng, nf, nextel, o2, cap, n_scat);
  }

  // The rest of a step that is neither a scatter nor a common crossing: no exit face, the end
  // of a free path without scattering, the boundary, roulette, an index jump, a vacuum element.
  // nf: the crossed face, whose plane is read again here (a common step keeps none of them).
  __device__ __forceinline__ bool rare(const JobDev &J, R &rng, int nf, int nextel, const float4 o2, int32_t cap,
                                       uint32_t &n_scat) {
    if (nf < 0) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, f2d_int(w));
      return die(J, kEvLost);
    }
    bool on = true;
    if (prop <= 0.0f) {
      if (mus > 0.0f) {  // at the step limit
        const Event ev = draw_event(rng.peek3());
        rotate(ev);
        rng.take(3);
        prop = ev.path;
        n_scat++;
      } else {
        rng.align();
        prop = free_path_f(unif_open_f(rng), mus);
      }
    } else {
      rng.reload();
      on = cross_rare(J, rng, nf, nextel, o2);
    }
    if (on && nsteps >= cap && !rng.exhausted()) {  // a tape that ends here is reported as that
      job_count(J, kJcCapped); job_ledger(J, kLgLost, f2d_int(w));
      return die(J, kEvCapped);
    }
    return on;
  }

  // The boundary, roulette, an index jump, a vacuum element.
  __device__ __forceinline__ bool cross_rare(const JobDev &J, R &rng, int nf, int nextel, const float4 o2) {
    const float4 pf = __ldg(reinterpret_cast<const float4 *>((geomp(J) + el)->pl) + nf);
    const float nx = pf.x, ny = pf.y, nz = pf.z;
    if (nextel < 0) {
      const int ib = -1 - nextel;
      const uint8_t bt = __ldg(J.bctype + ib);
      if (is_mirror(bt)) {
        const float dn = fmaf(dz, nz, fmaf(dx, nx, __fmul_rn(dy, ny)));
        dx -= 2.0f * dn * nx; dy -= 2.0f * dn * ny; dz -= 2.0f * dn * nz;
        return true;
      }
      const float bcn = d2f_int(__ldg(J.bcn + ib));
      if (bcn > 0.0f) {
        if (fresnel(rng, nx, ny, nz, nidx / bcn)) return true;
      }
      flush(J);
      if (!FD) add_f<R::kOneJob>(J, J.EBR + ib, w);
      else {
        float sp, cp;
        sincosf(phase, &sp, &cp);
        add_f<R::kOneJob>(J, J.EBR + ib, w * cp);
        add_f<R::kOneJob>(J, J.EBI + ib, -(w * sp));
      }
      tr.put(-1 - (int64_t)ib);
      tr.end();
      return false;
    }
    if (nextel >= J.Ne) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, f2d_int(w));
      return die(J, kEvLost);
    }
    if (mus <= 0.0f && o2.y > 0.0f) {
      prop = free_path_f(unif_open_f(rng), o2.y);
      if (roulette(J, rng)) return die(J, kEvRoulette);
      if (nidx != o2.w) {
        if (fresnel(rng, nx, ny, nz, nidx / o2.w)) return true;
      }
    } else {
      if (roulette(J, rng)) return die(J, kEvRoulette);
      if (nidx != o2.w) {
        if (fresnel(rng, nx, ny, nz, nidx / o2.w)) return true;
      }
      if (o2.y != mus) prop = keep_mul(prop, keep_div(mus, o2.y));
    }
    flush(J);
    el = nextel;
    mua = o2.x; mus = o2.y; g = o2.z; nidx = o2.w;
    return true;
  }
};

}  // namespace vmc
