// walk2d.cuh -- the triangular photon walk (MC2D), one element step per call.
//
// Walk2D64 follows PropagatePhoton (cpp/2d/MC2D.hpp:1307-1511) with its state in FP64:
// RayRayIntersects' choice among the edges (0,1), (1,2), (2,0) skipping the entry edge
// (WhichFace :914-955, :1710-1722), the 2D Henyey-Greenstein ScatterPhoton (:1135-1155),
// FresnelPhoton whose boundary branch transmits without refraction (:1178-1304), and the
// direction-weighted exitance DEBR/DEBI (:1410-1437).
// Walk2D32 is the FP32 tracking form with outward edge lines, as in the 3D form.
#pragma once
#include "walk3d.cuh"

namespace vmc {

// RayRayIntersects, cpp/2d/MC2D.hpp:1710-1722
__device__ __forceinline__ bool ray_seg(const double R[2], const double D[2], const double *U, const double *V,
                                        double &t) {
  double det = D[0] * (U[1] - V[1]) - D[1] * (U[0] - V[0]);
  if ((-kDblEps < det) && (det < kDblEps)) return false;
  const double ns = D[1] * (R[0] - U[0]) - D[0] * (R[1] - U[1]);
  // s = ns / det < 0 exactly when ns and det have opposite signs (the quotient of nonzero
  // coordinate differences cannot round to zero), decided before the division
  if ((ns < 0.0) != (det < 0.0) && ns != 0.0) return false;
  double s = ns / det;
  if ((s < 0.0) || (s > 1.0)) return false;
  t = ((R[1] - U[1]) * (U[0] - V[0]) - (R[0] - U[0]) * (U[1] - V[1])) / det;
  return true;
}

// The plain form, on the same lines as the tetrahedral one (walk3d.cuh): FP64 for the state,
// the exit edge picked in FP32 where that is certain, the samples on the integer pipe.
template <bool FD, class R>
struct Walk2D64 {
  static constexpr bool kBuffered = false;
  static constexpr bool kPack = true;
  static constexpr bool kCap32 = true;
  static constexpr bool kDefer = true;
  __device__ __forceinline__ bool pending() const { return pend != 0; }
  static constexpr int kMinBlocks = 2;
  static constexpr bool kStaged = false;
  static constexpr bool kLaunchLoss = false;
  Stage stage;
  using Tr = typename TraceFor<R>::type;
  double pos[2], dir[2];
  double w, prop, cph, sph;
  double mua, mus, g, nidx, imus;  // imus = 1 / mus
  uint64_t kg;                     // turn_ratio(g)
  double acc, accI;
  uint64_t turn;  // phase in 2^-64 turns
  int el, curface;
  int32_t nsteps;
  int pend;  // event to come: 1 + the face crossed, 0 none
  Tr tr;

  // moves the photon's state between lanes (Packer)
  template <class F> __device__ __forceinline__ void move(const F &f) {
    if constexpr (FD) f(pos[0], pos[1], dir[0], dir[1], w, prop, mua, mus, g, nidx, imus, kg, acc, turn, cph, sph, accI, el, curface, nsteps, pend);
    else f(pos[0], pos[1], dir[0], dir[1], w, prop, mua, mus, g, nidx, imus, kg, acc, el, curface, nsteps, pend);
  }

  __device__ __forceinline__ static const TriRec *recs(const JobDev &J) { return reinterpret_cast<const TriRec *>(J.geom); }
  __device__ __forceinline__ static const Tri64 *verts(const JobDev &J) { return reinterpret_cast<const Tri64 *>(recs(J) + J.Ne); }

  __device__ __forceinline__ void optics(const JobDev &J, int e, double &a, double &s, double &gg, double &nn) const {
    const double2 *o = reinterpret_cast<const double2 *>(J.optics) + 2 * (int64_t)(e & J.opt_mask);
    const double2 o0 = __ldg(o), o1 = __ldg(o + 1);
    a = o0.x; s = o0.y; gg = o1.x; nn = o1.y;
  }

  // (1 - g) / (1 + g); at |g| = 1 the reference's sqrt((g^2 + 1)^2 - 4 g^2) is 0 and its angle NaN
  __device__ __forceinline__ static double turn_factor(double g) {
    return fabs(g) == 1.0 ? __longlong_as_double(0x7ff8000000000000ll) : fast_div(1.0 - g, 1.0 + g);
  }

  __device__ void launch(const JobDev &J, R &rng, int64_t q) {
    tr.begin(J, q);
    create_photon_2d<false>(J, rng, pos, dir, el, curface);
    w = 1.0;
    if (FD) {
      turn = J.turn0;
      sincos_turn(turn, sph, cph);
    }
    optics(J, el, mua, mus, g, nidx);
    nidx = index_at_launch(nidx);
    imus = fast_rcp(mus);
    kg = turn_ratio(g);
    prop = neg_log_open(rng.next()) * imus;
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

  // What a scatter event draws: cosine and sine of the turn (in units of 2^-60), the free path
  // after it.
  struct Event { int64_t c, s; double path; bool held; };

  // ScatterPhoton (MC2D.hpp:1135-1155) turns the direction to atan2(dir) + 2 atan(h), h =
  // tan(pi xi) (1 - g) / (1 + g); here it is turned by that angle's cosine and sine, and no angle
  // is formed.  In fixed point, as in the tetrahedral walk: 1e6 photons on the square 8.1 -> 7.6 ms,
  // 50 000 on the uneven frequency-domain mesh 5.1 -> 4.3.
  __device__ __forceinline__ Event draw_event(uint3 u) const {
    Event e;
    e.held = turn_2d(u.x, g, kg, e.c, e.s);
    e.path = neg_log_open(u.y) * imus;
    return e;
  }

  // false: not for fixed point
  __device__ __forceinline__ bool rotate(const Event &e) {
    int64_t v[2] = {e.c, e.s};
    if ((__double_as_longlong(g) << 1) != 0) {  // else the drawn direction, whatever the old one
      if (!e.held || max(mag_of(dir[0]), mag_of(dir[1])) > 0x3ff00000u) return false;
      const Split60 c = split60(e.c), s = split60(e.s), x = split60(fixed60_of(dir[0])), y = split60(fixed60_of(dir[1]));
      v[0] = dot60(x, c, neg60(y), s);
      v[1] = dot60(y, c, x, s);
      if (!unit60(v, 2)) return false;
    }
    dir[0] = double_of_60(v[0]);
    dir[1] = double_of_60(v[1]);
    curface = -1;
    return true;
  }

  // The turn in FP64, for what fixed point does not hold: |g| near 1 or nearly 0, a direction that
  // is not a unit vector yet.  With (s0, c0) the sine and cosine of pi xi and ks = (1 - g) / (1 + g) s0 the turn's
  // cosine is (c0^2 - ks^2) / (c0^2 + ks^2) and its sine 2 ks c0 / (c0^2 + ks^2).
  struct Dir { double x, y; };
  __device__ __noinline__ static Dir turn_d(uint32_t u, double g, double dx, double dy) {
    double s0, c0;
    sincos_turn((uint64_t)u << 31, s0, c0);
    const double ks = turn_factor(g) * s0;
    const double a = c0 * c0, b = ks * ks;
    const double den = a + b;
    const double y0 = f2d_int(__frcp_rn(f32_of(den)));
    const double r = fma(-den, y0, 1.0);
    const double inv = fma(y0, fma(r, r, r), y0);
    const double k2 = ks * c0;
    const double k = unit_scale(fma(dx, dx, dy * dy));
    const double c = (a - b) * inv * k, s = (k2 + k2) * inv * k;
    return Dir{fma(dx, c, -(dy * s)), fma(dy, c, dx * s)};
  }

  // FresnelPhoton at an edge with normal (n0, n1) of any length
  __device__ __forceinline__ bool fresnel(R &rng, double n0, double n1, double nout, int nf, bool inside) {
    const float f0 = f32_of(n0), f1 = f32_of(n1);
    const Choice choice = fresnel_choice(rng, __fdividef(f32_of(nidx), f32_of(nout)), f0 * f32_of(dir[0]) + f1 * f32_of(dir[1]),
                                         f0 * f0 + f1 * f1);
    if (choice.what == Choice::kPass && !inside) return false;
    const double nn = fma(n0, n0, n1 * n1), dn = fma(dir[0], n0, dir[1] * n1);
    if (choice.what == Choice::kReflect) {
      const double k = -2.0 * div_near(dn, nn, f32_of(nn));
      dir[0] = fma(k, n0, dir[0]);
      dir[1] = fma(k, n1, dir[1]);
      curface = nf;
      return true;
    }
    const double nipnt = fast_div(nidx, nout);
    double len, inv;
    fast_sqrt(nn, len, inv);
    n0 *= inv; n1 *= inv;
    const double costhi = -dn * inv;
    double costht = 0.0;
    if (fresnel_reflects_d(rng, choice, nipnt, costhi, costht)) {
      const double k = 2.0 * costhi;
      dir[0] = fma(k, n0, dir[0]);
      dir[1] = fma(k, n1, dir[1]);
      curface = nf;
      return true;
    }
    if (!inside) return false;
    const double m = (costhi > 0.0) ? (nipnt * costhi - costht) : (nipnt * costhi + costht);
    dir[0] = fma(nipnt, dir[0], m * n0);
    dir[1] = fma(nipnt, dir[1], m * n1);
    return false;
  }

  // WhichFace, MC2D.hpp:914-955: edges (0,1), (1,2), (2,0) in order, skipping curface
  struct Exit { double dist; int nf; };
  __device__ __noinline__ static Exit which_face(const Tri64 *T, double px, double py, double dx, double dy, int curface) {
    const double *v = &T->v[0][0];
    const double pos[2] = {px, py}, dir[2] = {dx, dy};
    double dist = 0.0;
    if (curface != 0 && ray_seg(pos, dir, v, v + 2, dist) && dist > 0.0) return Exit{dist, 0};
    if (curface != 1 && ray_seg(pos, dir, v + 2, v + 4, dist) && dist > 0.0) return Exit{dist, 1};
    if (curface != 2 && ray_seg(pos, dir, v + 4, v, dist) && dist > 0.0) return Exit{dist, 2};
    return Exit{0.0, -1};
  }

  // the exit edge and the distance to it, as in the tetrahedral walk
  __device__ __forceinline__ int exit_face(const JobDev &J, double &dist, int4 &nbr) const {
    const TriRec *T = recs(J) + el;
    const double2 a0 = __ldg(reinterpret_cast<const double2 *>(T->v0));
    const double offd = __ldg(&T->off);
    const float4 q0 = __ldg(reinterpret_cast<const float4 *>(T->nf));
    const float4 q1 = __ldg(reinterpret_cast<const float4 *>(T->nf) + 1);
    nbr = __ldg(reinterpret_cast<const int4 *>(T->nbr));
    const double rx = pos[0] - a0.x, ry = pos[1] - a0.y;
    const float fx = f32_of(rx), fy = f32_of(ry), off = q1.z;
    const float dx = f32_of(dir[0]), dy = f32_of(dir[1]);
    const float n[3][2] = {{q0.x, q0.y}, {q0.z, q0.w}, {q1.x, q1.y}};
    const float rs = fabsf(fx) + fabsf(fy) + fabsf(off), ds = fabsf(dx) + fabsf(dy);
    const float en = 1e-6f * rs, ed = 8e-6f * ds, margin = 4e-6f * rs * ds;
    float num[3], nd[3], bnum = 1.0f, bnd = 0.0f;
    int nf = -1;
#pragma unroll
    for (int f = 0; f < 3; f++) {
      num[f] = (f == 1 ? off : 0.0f) - (n[f][0] * fx + n[f][1] * fy);
      nd[f] = n[f][0] * dx + n[f][1] * dy;
      const bool better = f != curface && nd[f] > ed && num[f] * bnd < bnum * nd[f];
      bnum = better ? num[f] : bnum;
      bnd = better ? nd[f] : bnd;
      nf = better ? f : nf;
    }
    bool sure = nf >= 0 && bnum > en;
#pragma unroll
    for (int f = 0; f < 3; f++)
      sure = sure && (f == nf || (num[f] * bnd - bnum * nd[f] > margin && (f == curface || num[f] > en)));
    const double *m = T->n[nf < 0 ? 0 : nf];
    const double m0 = __ldg(m), m1 = __ldg(m + 1);
    const double dn = fma(m1, dir[1], m0 * dir[0]);
    const float dnf = f32_of(dn);
    dist = div_near((nf == 1 ? offd : 0.0) - fma(m1, ry, m0 * rx), dn, dnf);
    if (sure && f32_safe(dnf)) return nf;
    const Exit e = which_face(verts(J) + el, pos[0], pos[1], dir[0], dir[1], curface);
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
    pos[0] = fma(dir[0], ds, pos[0]);
    pos[1] = fma(dir[1], ds, pos[1]);
    tr.put(el);
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
          const Dir d = turn_d(rng.peek3().x, g, dir[0], dir[1]);
          dir[0] = d.x; dir[1] = d.y;
          curface = -1;
        }
        rng.take(2);
        prop = ev.path;
        n_scat++;
      } else {
        rng.align();
        prop = neg_log_open(rng.next()) * imus;
      }
    } else {
      prop -= dist;
      const int nextel = nf == 0 ? nb.x : nf == 1 ? nb.y : nb.z;
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
    const int f2 = nb2.x == el ? 0 : nb2.y == el ? 1 : nb2.z == el ? 2 : -1;
    if (f2 < 0) return false;
    if (differ(mus2, mus)) {
      prop *= mus / mus2;  // x (mus / mus) == x
      imus = fast_rcp(mus2);
    }
    if (differ(g2, g)) kg = turn_ratio(g2);
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

  // the boundary, or the next element, behind edge nf
  __device__ __forceinline__ bool cross(const JobDev &J, R &rng, int nf, int nextel) {
    if (nextel >= J.Ne) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, w);
      return die(J, kEvLost);
    }
    const bool inside = nextel >= 0;
    const int ib = -1 - nextel;
    double mua2 = 0.0, mus2 = 0.0, g2 = 0.0, n2;
    if (inside) {
      optics(J, nextel, mua2, mus2, g2, n2);
    } else {
      if (is_mirror(__ldg(J.bctype + ib))) {
        const double *bn = J.bnorm + 4 * (int64_t)ib;
        const double cdot = bn[0] * dir[0] + bn[1] * dir[1];
        dir[0] -= 2.0 * cdot * bn[0];
        dir[1] -= 2.0 * cdot * bn[1];
        curface = nf;
        return true;
      }
      n2 = __ldg(J.bcn + ib);
    }
    const bool vacuum = inside && at_most_zero(mus) && positive(mus2);
    const bool jump = inside ? differ(nidx, n2) : positive(n2);
    const bool light = inside && below(w, kWeight0);
    if (!inside || vacuum || jump || light) {
      const double *m = (recs(J) + el)->n[nf];
      const double n0 = __ldg(m), n1 = __ldg(m + 1);  // outward
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
      if (jump && fresnel(rng, n0, n1, n2, nf, inside)) return true;
      if (!inside) {
        const double idn = fast_sqrt(fma(n0, n0, n1 * n1)) * fast_rcp(fma(dir[0], n0, dir[1] * n1));  // DEBR, MC2D.hpp:1410-1437
        flush(J);
        if (!FD) {
          add_d(J, J.EBR + ib, w);
          add_d(J, J.DEBR + ib, w * idn);
        } else {
          const double re = w * cph, im = -(w * sph);
          add_d(J, J.EBR + ib, re);
          add_d(J, J.EBI + ib, im);
          add_d(J, J.DEBR + ib, re * idn);
          add_d(J, J.DEBI + ib, im * idn);
        }
        tr.put(-1 - (int64_t)ib);
        tr.end();
        return false;
      }
    }
    const int4 nb2 = __ldg(reinterpret_cast<const int4 *>((recs(J) + nextel)->nbr));
    const int f2 = nb2.x == el ? 0 : nb2.y == el ? 1 : nb2.z == el ? 2 : -1;
    if (differ(mus2, mus)) {
      if (!vacuum) prop *= mus / mus2;  // x (mus / mus) == x
      imus = fast_rcp(mus2);
    }
    if (f2 < 0) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, w);
      return die(J, kEvLost);
    }
    if (differ(g2, g)) kg = turn_ratio(g2);
    flush(J);
    curface = f2;
    el = nextel;
    mua = mua2; mus = mus2; g = g2; nidx = n2;
    return true;
  }
};

// the reference's operation sequence, for the jobs that need it (as Walk3D64L)
template <bool FD, class R>
struct Walk2D64L {
  static constexpr bool kBuffered = true;  // words left in a block are carried from step to step
  static constexpr bool kPack = true;
  static constexpr bool kCap32 = false;
  static constexpr bool kDefer = false;
  static constexpr int kMinBlocks = 2;
  static constexpr bool kStaged = false;
  static constexpr bool kLaunchLoss = false;
  Stage stage;
  using Tr = typename TraceFor<R>::type;
  double pos[2], dir[2];
  double w, prop, phase, cph, sph;
  double mua, mus, g, nidx;
  double acc, accI;
  int el, curface;
  int64_t nsteps;
  Tr tr;

  // moves the photon's state between lanes (Packer)
  template <class F> __device__ __forceinline__ void move(const F &f) {
    if constexpr (FD) f(pos[0], pos[1], dir[0], dir[1], w, prop, mua, mus, g, nidx, acc, phase, cph, sph, accI, el, curface, nsteps);
    else f(pos[0], pos[1], dir[0], dir[1], w, prop, mua, mus, g, nidx, acc, el, curface, nsteps);
  }

  __device__ __forceinline__ static const Tri64 *tris(const JobDev &J) { return reinterpret_cast<const Tri64 *>(J.geom); }
  __device__ __forceinline__ void optics(const JobDev &J, int e, double &a, double &s, double &gg, double &nn) const {
    const double2 *o = reinterpret_cast<const double2 *>(J.optics) + 2 * (int64_t)(e & J.opt_mask);
    const double2 o0 = __ldg(o), o1 = __ldg(o + 1);
    a = o0.x; s = o0.y; gg = o1.x; nn = o1.y;
  }

  __device__ void launch(const JobDev &J, R &rng, int64_t q) {
    tr.begin(J, q);
    create_photon_2d<true>(J, rng, pos, dir, el, curface);
    w = 1.0;
    phase = J.phase0;
    if (FD) sincos(phase, &sph, &cph);
    optics(J, el, mua, mus, g, nidx);
    prop = -log(unif_open(rng)) / mus;
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

  __device__ void scatter(R &rng) {
    if (g != 0.0) {
      double xi = unif_halfup(rng);
      double g2 = g * g;
      double t = sqrt((g2 + 1.0) * (g2 + 1.0) - 4.0 * g2);
      // ScatterPhoton (MC2D.hpp:1135-1155) turns the direction to atan2(dir) + 2 atan(h);
      // here the direction is turned by the angle 2 atan(h), whose cosine and sine are
      // (1 - h^2) / (1 + h^2) and 2 h / (1 + h^2) (from 1 / h when |h| > 1), without forming
      // either angle: the same direction to a few ulps, 10% less FP64 work per photon
      const double h = tan(-xi * t * kPi / (g2 - 1.0)) * (g2 - 2 * g + 1.0) / t;
      double c, s;
      if (fabs(h) <= 1.0) {
        const double d = 1.0 / (1.0 + h * h);
        c = (1.0 - h * h) * d; s = 2.0 * h * d;
      } else {
        const double r = 1.0 / h, d = 1.0 / (1.0 + r * r);
        c = (r * r - 1.0) * d; s = 2.0 * r * d;
      }
      const double inv = 1.0 / sqrt(dir[0] * dir[0] + dir[1] * dir[1]);
      const double ux = dir[0] * inv, uy = dir[1] * inv;
      dir[0] = ux * c - uy * s;
      dir[1] = uy * c + ux * s;
    } else {
      sincospi(2.0 * unif_halfup(rng), &dir[1], &dir[0]);
    }
    curface = -1;
  }

  __device__ bool fresnel(R &rng, const double nor[2], double nipnt, int nf, bool boundary) {
    double costhi = -(dir[0] * nor[0] + dir[1] * nor[1]);
    double costht = 0.0;
    if (fresnel_reflects_angles(rng, nipnt, costhi, costht)) {
      dir[0] += 2.0 * costhi * nor[0];
      dir[1] += 2.0 * costhi * nor[1];
      curface = nf;
      return true;
    }
    if (boundary) return false;
    double m = (costhi > 0.0) ? (nipnt * costhi - costht) : (nipnt * costhi + costht);
    dir[0] = nipnt * dir[0] + m * nor[0];
    dir[1] = nipnt * dir[1] + m * nor[1];
    return false;
  }

  // Normal(el, f), MC2D.hpp:358-387: the unit normal of the edge from a to b
  __device__ __forceinline__ static void normal_of(const double a[2], const double b[2], double nor[2]) {
    double ddx = b[0] - a[0], ddy = b[1] - a[1];
    double norm = sqrt(ddx * ddx + ddy * ddy);
    nor[0] = ddy / norm; nor[1] = -ddx / norm;
  }
  // Edge f runs from vertex f to vertex f + 1 (mod 3).  Only the Fresnel and exit paths
  // need its normal, so they read the two vertices again from the element record (the same
  // doubles) instead of indexing the step's vertex array by f, which would put that array
  // in local memory for the whole step.
  __device__ static void edge_normal(const Tri64 *T, int f, double nor[2]) {
    const double *v = &T->v[0][0];
    const int i0 = f, i1 = f == 2 ? 0 : f + 1;
    const double a[2] = {__ldg(v + 2 * i0), __ldg(v + 2 * i0 + 1)};
    const double b[2] = {__ldg(v + 2 * i1), __ldg(v + 2 * i1 + 1)};
    normal_of(a, b, nor);
  }

  __device__ bool roulette(const JobDev &J, R &rng) {
    if (w < kWeight0) {
      if (unif_closed(rng) > kChance) {
        job_count(J, kJcRoulette); job_ledger(J, kLgRouletteKill, w);
        return true;
      }
      job_ledger(J, kLgRouletteGain, w / kChance - w);
      w /= kChance;
    }
    return false;
  }

  __device__ int step(const JobDev &J, R &rng, int64_t max_steps) {
    if (rng.exhausted()) { job_count(J, kJcTapeEnd); return die(J, kEvTapeEnd); }
    if (nsteps >= max_steps) {
      job_count(J, kJcCapped); job_ledger(J, kLgLost, w);
      return die(J, kEvCapped);
    }
    const Tri64 *T = tris(J) + el;
    double V[3][2];
    {
      const double2 *src = reinterpret_cast<const double2 *>(T->v);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        double2 d2 = __ldg(src + i);
        V[i][0] = d2.x; V[i][1] = d2.y;
      }
    }
    const int4 nb = __ldg(reinterpret_cast<const int4 *>(T->nbr));
    double dist = 0.0;
    int nf = -1;
    if (curface != 0 && ray_seg(pos, dir, V[0], V[1], dist) && dist > 0.0) nf = 0;
    else if (curface != 1 && ray_seg(pos, dir, V[1], V[2], dist) && dist > 0.0) nf = 1;
    else if (curface != 2 && ray_seg(pos, dir, V[2], V[0], dist) && dist > 0.0) nf = 2;
    if (nf < 0) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, w);
      return die(J, kEvLost);
    }
    const int nextel = nf == 0 ? nb.x : nf == 1 ? nb.y : nb.z;
    nsteps++;
    const double ds = fmin(prop, dist);
    pos[0] += dir[0] * ds;
    pos[1] += dir[1] * ds;
    tr.put(el);
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
      if (mus > 0.0) { scatter(rng); res = kScattered; }
      prop = -log(unif_open(rng)) / mus;
      return res;
    }
    if (nextel < 0) {
      const int ib = -1 - nextel;
      const uint8_t bt = __ldg(J.bctype + ib);
      if (is_mirror(bt)) {
        const double *bn = J.bnorm + 4 * (int64_t)ib;
        double cdot = bn[0] * dir[0] + bn[1] * dir[1];
        dir[0] -= 2.0 * cdot * bn[0];
        dir[1] -= 2.0 * cdot * bn[1];
        curface = nf;
        return kAlive;
      }
      double nor[2];
      edge_normal(T, nf, nor);
      const double bcn = __ldg(J.bcn + ib);
      if (bcn > 0.0 && fresnel(rng, nor, nidx / bcn, nf, true)) return kAlive;
      // outward edge normal for DEBR (MC2D.hpp:1410-1423)
      double tx = (V[0][0] + V[1][0] + V[2][0]) / 3.0 - pos[0];
      double ty = (V[0][1] + V[1][1] + V[2][1]) / 3.0 - pos[1];
      if (nor[0] * tx + nor[1] * ty > 0.0) { nor[0] = -nor[0]; nor[1] = -nor[1]; }
      double dn = dir[0] * nor[0] + dir[1] * nor[1];
      flush(J);
      if (!FD) {
        add_d(J, J.EBR + ib, w);
        add_d(J, J.DEBR + ib, w / dn);
      } else {
        add_d(J, J.EBR + ib, w * cph);
        add_d(J, J.EBI + ib, -(w * sph));
        add_d(J, J.DEBR + ib, w * cph / dn);
        add_d(J, J.DEBI + ib, -(w * sph / dn));
      }
      tr.put(-1 - (int64_t)ib);
      tr.end();
      return kDied;
    }
    if (nextel >= J.Ne) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, w);
      return die(J, kEvLost);
    }
    double mua2, mus2, g2, n2;
    optics(J, nextel, mua2, mus2, g2, n2);
    if ((mus <= 0.0) && (mus2 > 0.0)) {
      prop = -log(unif_open(rng)) / mus2;
      if (roulette(J, rng)) return die(J, kEvRoulette);
      if (nidx != n2) {
        double nor[2];
        edge_normal(T, nf, nor);
        if (fresnel(rng, nor, nidx / n2, nf, false)) return kAlive;
      }
    } else {
      if (roulette(J, rng)) return die(J, kEvRoulette);
      if (nidx != n2) {
        double nor[2];
        edge_normal(T, nf, nor);
        if (fresnel(rng, nor, nidx / n2, nf, false)) return kAlive;
      }
      if (mus2 != mus) prop *= mus / mus2;  // x (mus / mus) == x: skip the division
    }
    const int4 nb2 = __ldg(reinterpret_cast<const int4 *>((tris(J) + nextel)->nbr));
    int f2 = nb2.x == el ? 0 : nb2.y == el ? 1 : nb2.z == el ? 2 : -1;
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
};

template <bool FD, class R>
struct Walk2D32 {
  static constexpr bool kPack = false;  // its walks are short: packing gains nothing and costs the loop 2 %
  static constexpr bool kCap32 = false;
  static constexpr bool kDefer = true;
  __device__ __forceinline__ bool pending() const { return pend != 0; }
  static constexpr int kMinBlocks = 4;
  static constexpr bool kStaged = false;
  Stage stage;
  using Tr = typename TraceFor<R>::type;
  float px, py, dx, dy;
  float w, prop, phase;
  float mua, mus, g, nidx;
  float acc, accI;
  int el;
  int32_t nsteps;
  int pend;  // event to come: 1 + the edge crossed, 0 none
  bool outward;  // launched out through its own entry edge
  Tr tr;

  __device__ __forceinline__ float4 optics(const JobDev &J, int e) const {
    return __ldg(reinterpret_cast<const float4 *>(J.optics) + (e & J.opt_mask));
  }

  __device__ void launch(const JobDev &J, R &rng, int64_t q) {
    tr.begin(J, q);
    float p[2], d[2];
    int cf;
    create_photon_2d_f(J, rng, p, d, el, cf);
    px = p[0]; py = p[1];
    dx = d[0]; dy = d[1];
    // the entry edge is never tested by the reference's WhichFace (MC2D.hpp:927-952): a
    // photon launched out through it is lost
    outward = false;
    if (cf >= 0) {
      const float4 ln = __ldg(reinterpret_cast<const float4 *>((reinterpret_cast<const Tri32 *>(J.geom) + el)->ln) + cf);
      outward = ln.x * dx + ln.y * dy > 0.0f;
    }
    w = 1.0f;
    phase = J.phase_f;
    float4 o = optics(J, el);
    mua = o.x; mus = o.y; g = o.z; nidx = o.w;
    prop = free_path_f(unif_open_f(rng), mus);
    acc = accI = 0.0f;
    nsteps = 0;
    pend = 0;
  }

  __device__ __forceinline__ void flush(const JobDev &J) {
    add_f<R::kOneJob>(J, J.ER + el, acc);
    if (FD) add_f<R::kOneJob>(J, J.EI + el, accI);
    acc = accI = 0.0f;
  }

  __device__ __forceinline__ int die(const JobDev &J, int64_t ev) {
    flush(J);
    tr.put(ev);
    tr.end();
    return kDied;
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

  __device__ __forceinline__ void scatter(R &rng) {
    // 2D Henyey-Greenstein: the reference's angle 2 atan(tan(-xi t pi / (g^2 - 1)) (1 - g)^2 / t)
    // with t = 1 - g^2 reduces to 2 atan(tan(pi xi) (1 - g) / (1 + g))
    float xi = unif_halfup_f(rng);
    float sn, cs;
    if (g != 0.0f) {
      // th = 2 atan(z), z = k tan(pi xi), k = (1 - g) / (1 + g): with (s0, c0) the sine and
      // cosine of pi xi, cos th = (c0^2 - (k s0)^2) / (c0^2 + (k s0)^2) and
      // sin th = 2 k s0 c0 / (c0^2 + (k s0)^2) -- no arctangent, no sine of th
      float s0, c0;
      sincospif(xi, &s0, &c0);
      const float ks = __fdividef(1.0f - g, 1.0f + g) * s0;
      const float a = c0 * c0, b = ks * ks;
      const float inv = __fdividef(1.0f, a + b);
      cs = (a - b) * inv;
      sn = 2.0f * ks * c0 * inv;
      float nx = dx * cs - dy * sn, ny = dx * sn + dy * cs;
      float in = rsqrtf(nx * nx + ny * ny);
      dx = nx * in; dy = ny * in;
    } else {
      sincospif(2.0f * xi, &sn, &cs);
      dx = cs; dy = sn;
    }
  }

  __device__ __forceinline__ bool fresnel(R &rng, float nx, float ny, float eta, bool boundary) {
    float dn = fmaf(dy, ny, __fmul_rn(dx, nx));
    float ci = fabsf(dn);
    float ct = 0.0f;
    if (fresnel_reflects_f(rng, eta, ci, ct)) {
      dx -= 2.0f * dn * nx; dy -= 2.0f * dn * ny;
      return true;
    }
    if (boundary) return false;
    float m = copysignf(ct, dn) - eta * dn;
    dx = fmaf(eta, dx, __fmul_rn(m, nx)); dy = fmaf(eta, dy, __fmul_rn(m, ny));
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

  __device__ int step(const JobDev &J, R &rng, int64_t max_steps) {
    if (rng.exhausted()) { job_count(J, kJcTapeEnd); return die(J, kEvTapeEnd); }
    if (nsteps >= max_steps) {
      job_count(J, kJcCapped); job_ledger(J, kLgLost, f2d_int(w));
      return die(J, kEvCapped);
    }
    if (R::kReplay && outward) {  // with Philox streams this is settled at launch
      job_count(J, kJcLoss); job_ledger(J, kLgLost, f2d_int(w));
      return die(J, kEvLost);
    }
    const Tri32 *T = reinterpret_cast<const Tri32 *>(J.geom) + el;
    const float4 *L4 = reinterpret_cast<const float4 *>(T->ln);
    const float4 l0 = __ldg(L4 + 0), l1 = __ldg(L4 + 1), l2 = __ldg(L4 + 2);
    // selects over all three edges, no branch per edge; num / nd compared by cross
    // products, one reciprocal for the winning edge (bnd = 0: none yet)
    float bnum = 1.0f, bnd = 0.0f;
    int nf = -1;
    {
      const float4 ln[3] = {l0, l1, l2};
#pragma unroll
      for (int f = 0; f < 3; f++) {
        const float nd = ln[f].x * dx + ln[f].y * dy;
        const float num = ln[f].z - (ln[f].x * px + ln[f].y * py);
        const bool better = nd > 0.0f && num * bnd < bnum * nd;
        bnum = better ? num : bnum;
        bnd = better ? nd : bnd;
        nf = better ? f : nf;
      }
    }
    const float best = __fdividef(bnum, bnd);
    if (nf < 0) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, f2d_int(w));
      return die(J, kEvLost);
    }
    nsteps++;
    const float dist = fmaxf(best, 0.0f);
    const float ds = fminf(prop, dist);
    px += dx * ds; py += dy * ds;
    tr.put(el);
    const float x = mua * ds;
    if (!FD) {
      if (mua > 0.0f) {
        float dep = w * one_minus_exp_neg(x);
        acc += dep;
        w -= dep;
      } else {
        acc += w * ds;
      }
    } else {
      const float th = J.k_scale_f * nidx * ds;
      const float om = one_minus_exp_neg(x);
      const float a = 1.0f - om;
      const float sh = sin_small(0.5f * th);
      const float c1 = om + 2.0f * a * sh * sh;
      const float s1 = a * sin_small(th);
      float sp, cp;
      __sincosf(phase, &sp, &cp);
      // these roundings, whatever the shape of the code around them (as in the 3D walk)
      acc = fmaf(w, fmaf(sp, s1, __fmul_rn(cp, c1)), acc);
      accI = fmaf(w, fmaf(cp, s1, -__fmul_rn(sp, c1)), accI);
      phase = wrap_phase(__fadd_rn(phase, th));
      w *= a;
    }
    prop -= ds;
    if (prop <= 0.0f) {
      int res = kAlive;
      rng.align();
      if (mus > 0.0f) { scatter(rng); res = kScattered; }
      prop = free_path_f(unif_open_f(rng), mus);
      return res;
    }
    // the common crossing (scattering medium, weight above the roulette threshold, no index jump)
    const int nextel = __ldg(T->nbr + nf);
    if ((unsigned)nextel < (unsigned)J.Ne && mus > 0.0f && w >= (float)kWeight0) {
      const float4 o2 = optics(J, nextel);
      if (nidx == o2.w) {
        if (o2.y != mus) prop *= mus / o2.y;
        flush(J);
        el = nextel;
        mua = o2.x; mus = o2.y; g = o2.z;
        return kAlive;
      }
    }
    pend = 1 + nf;
    return kAlive;
  }

  // What is left of a step that ends in neither: run for several lanes of a warp together.
  __device__ __forceinline__ bool event(const JobDev &J, R &rng, int32_t, uint32_t &) {
    const int nf = pend - 1;
    pend = 0;
    const Tri32 *T = reinterpret_cast<const Tri32 *>(J.geom) + el;
    const float2 line = __ldg(reinterpret_cast<const float2 *>(T->ln[nf]));
    const float nx = line.x, ny = line.y;
    const int nextel = __ldg(T->nbr + nf);
    const int ib = -1 - nextel;  // the boundary edge when nextel < 0
    const bool inside = nextel >= 0;
    if (nextel >= J.Ne) {
      job_count(J, kJcLoss); job_ledger(J, kLgLost, f2d_int(w));
      die(J, kEvLost);
      return false;
    }
    float4 o2 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (inside) {
      o2 = optics(J, nextel);
    } else {
      if (is_mirror(__ldg(J.bctype + ib))) {
        const float dn = fmaf(dy, ny, __fmul_rn(dx, nx));
        dx -= 2.0f * dn * nx; dy -= 2.0f * dn * ny;
        return true;
      }
      o2.w = d2f_int(__ldg(J.bcn + ib));
    }
    // one copy of roulette and of the interface for elements and the boundary: each holds a
    // Philox block per draw, and the kernel waits for instructions as it is
    const bool vacuum = inside && mus <= 0.0f && o2.y > 0.0f;
    if (vacuum) prop = free_path_f(unif_open_f(rng), o2.y);
    if (inside && roulette(J, rng)) {
      die(J, kEvRoulette);
      return false;
    }
    if ((inside ? nidx != o2.w : o2.w > 0.0f) && fresnel(rng, nx, ny, nidx / o2.w, !inside)) return true;
    if (!inside) {
      const float dn = fmaf(dy, ny, __fmul_rn(dx, nx));
      flush(J);
      if (!FD) {
        add_f<R::kOneJob>(J, J.EBR + ib, w);
        add_f<R::kOneJob>(J, J.DEBR + ib, __fdividef(w, dn));
      } else {
        float sp, cp;
        sincosf(phase, &sp, &cp);
        add_f<R::kOneJob>(J, J.EBR + ib, w * cp);
        add_f<R::kOneJob>(J, J.EBI + ib, -(w * sp));
        add_f<R::kOneJob>(J, J.DEBR + ib, __fdividef(w * cp, dn));
        add_f<R::kOneJob>(J, J.DEBI + ib, -__fdividef(w * sp, dn));
      }
      tr.put(-1 - (int64_t)ib);
      tr.end();
      return false;
    }
    if (!vacuum && o2.y != mus) prop *= mus / o2.y;
    flush(J);
    el = nextel;
    mua = o2.x; mus = o2.y; g = o2.z; nidx = o2.w;
    return true;
  }
};

}  // namespace vmc
