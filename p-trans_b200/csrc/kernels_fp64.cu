/*
 * kernels_fp64.cu - FP64 transport: the reference's intersection, reflection
 * and transmission arithmetic in FP64, its 1e-7 nm nudge and its out-of-box
 * check (calcTransmit and helpers, src/RTMCphon.f90:1608-2414, 2883-3301),
 * in two forms that take the same trajectories bit for bit:
 *   - k_plain_fp64, one phonon per thread and the reference's linear scan of
 *     the box grain plus the current grain at every flight: the comparator of
 *     the persistent kernels and the replay target of the CPU oracle;
 *   - k_drain64 / k_tail64, the two phases of the persistent FP32 kernels
 *     (kernels_fp32.cu) with FP64 flights.
 *
 * Compiled with --fmad=false, so every a*b+c is rounded twice, exactly as the
 * host restatement computes it.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "fp64_math.cuh"
#include "geo_fp32.cuh"
#include "kernels.h"
#include "philox.cuh"

namespace ptg {

namespace {

constexpr double kSmall = 1.0e-5;       /* SMALL_VAL, src/RTMCphon.f90:67 */
constexpr double kBallistic = 1.0e10;   /* src/RTMCphon.f90:1686          */
/* safe-ball radius searched in a grain with a BVH, in units of the MFP */
constexpr float kBallCap64 = 32.0f;

__device__ __forceinline__ double dot3(const double* a, const double* b) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}
__device__ __forceinline__ void cross3(const double* a, const double* b, double* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}

struct Draw {
  Key2 key;
  uint32_t c1, slo, shi;
  __device__ void block(uint32_t flight, uint32_t sub, double* d0, double* d1) const {
    const uint4 p = philox10(flight, sub | c1, slo, shi, key);
    *d0 = u52d(p.x, p.y);
    *d1 = u52d(p.z, p.w);
  }
};

/* Convex-polygon sign test of src/RTMCphon.f90:2942-2955 / 2961-2983. */
__device__ bool in_polygon(const double* v, int n, const double* Rh) {
  double c1[3], ci[3], Ra[3], Rb[3];
  for (int i = 0; i < n; ++i) {
    for (int d = 0; d < 3; ++d) {
      Ra[d] = v[3 * (i + 1) + d] - v[3 * i + d];
      Rb[d] = Rh[d] - v[3 * i + d];
    }
    cross3(Ra, Rb, ci);
    if (i == 0) {
      c1[0] = ci[0]; c1[1] = ci[1]; c1[2] = ci[2];
    } else if (dot3(c1, ci) < 0.0) {
      return false;
    }
  }
  return true;
}

/* Capped cylinder (extension): unit axis and half length from the axis end
   points A = vertex 0, B = vertex 1. */
__device__ void capped_axis(const Geo64& g, int k, double* a, double* hl) {
  const double* v = g.vertex + 3 * (size_t)g.vbegin[k];
  double e[3] = {v[3] - v[0], v[4] - v[1], v[5] - v[2]};
  const double len = sqrt(dot3(e, e));
  for (int d = 0; d < 3; ++d) a[d] = e[d] / len;
  *hl = 0.5 * len;
}

/* Nearest strictly positive hit of the lateral surface (within the caps)
   and the two cap discs (within the radius). */
__device__ bool capped_distance(const Geo64& g, int k, const double* R0, const double* D,
                                double* L) {
  double a[3], hl;
  capped_axis(g, k, a, &hl);
  const double* C = g.center + 3 * k;
  double w[3] = {R0[0] - C[0], R0[1] - C[1], R0[2] - C[2]};
  const double s0 = dot3(w, a), ds = dot3(D, a);
  double wp[3], dp[3];
  for (int d = 0; d < 3; ++d) {
    wp[d] = w[d] - s0 * a[d];
    dp[d] = D[d] - ds * a[d];
  }
  const double r2 = g.radius[k] * g.radius[k];
  double best = 0.0;
  bool hit = false;
  const double A2 = dot3(dp, dp);
  if (A2 > 0.0) {
    const double B = dot3(wp, dp), Cc = dot3(wp, wp) - r2;
    const double disc = B * B - A2 * Cc;
    if (disc >= 0.0) {
      const double sq = sqrt(disc);
      const double t[2] = {(-B - sq) / A2, (-B + sq) / A2};
      for (int i = 0; i < 2; ++i) {
        if (!(t[i] > 0.0) || (hit && !(t[i] < best))) continue;
        if (fabs(s0 + t[i] * ds) <= hl) { best = t[i]; hit = true; }
      }
    }
  }
  if (ds != 0.0) {
    for (int i = 0; i < 2; ++i) {
      const double c = (i == 0) ? -hl : hl;
      const double t = (c - s0) / ds;
      if (!(t > 0.0) || (hit && !(t < best))) continue;
      double q[3];
      for (int d = 0; d < 3; ++d) q[d] = wp[d] + t * dp[d];
      if (dot3(q, q) <= r2) { best = t; hit = true; }
    }
  }
  if (!hit) return false;
  *L = best;
  return true;
}

/* Outward normal of the nearer piece: cap (+-axis) or mantle (radial). */
__device__ void capped_normal(const Geo64& g, int k, const double* R, double* N) {
  double a[3], hl;
  capped_axis(g, k, a, &hl);
  const double* C = g.center + 3 * k;
  double w[3] = {R[0] - C[0], R[1] - C[1], R[2] - C[2]};
  const double sa = dot3(w, a);
  double wp[3];
  for (int d = 0; d < 3; ++d) wp[d] = w[d] - sa * a[d];
  const double rho = sqrt(dot3(wp, wp));
  if (fabs(fabs(sa) - hl) < fabs(rho - g.radius[k])) {
    const double sg = (sa < 0.0) ? -1.0 : 1.0;
    for (int d = 0; d < 3; ++d) N[d] = sg * a[d];
  } else {
    for (int d = 0; d < 3; ++d) N[d] = wp[d] / rho;
  }
}

/* calcSurfaceDistance dispatch, src/RTMCphon.f90:2883-3088.  CULL: a polygon
   whose plane is crossed beyond lim is left before the division and the edge
   test (the product's 1e-6 is far above the rounding of either side).  EXT: as
   in the FP32 kernels, 0 without BVH and capped cylinders. */
template <bool CULL, int EXT>
__device__ bool surface_distance(const Geo64& g, int k, const double* R0, const double* D,
                                 double lim, double* L) {
  const int sh = g.shape[k];
  if (sh == 1) {
    const double* N = g.normal + 3 * k;
    const double cosangle = dot3(D, N);
    if (cosangle <= 0.0) return false;
    const double* v = g.vertex + 3 * (size_t)g.vbegin[k];
    double w[3] = {v[0] - R0[0], v[1] - R0[1], v[2] - R0[2]};
    const double num = dot3(w, N);
    if (CULL && num > lim * cosangle * 1.000001) return false;
    const double Lh = num / cosangle;
    if (Lh < 0.0) return false;
    if (CULL && Lh > lim) return false;
    double Rh[3];
    for (int d = 0; d < 3; ++d) Rh[d] = R0[d] + D[d] * Lh;
    if (!in_polygon(v, g.nvertex[k], Rh)) return false;
    *L = Lh;
    return true;
  }
  if (EXT && sh == 4) return capped_distance(g, k, R0, D, L);
  const double* C = g.center + 3 * k;
  const double r = g.radius[k];
  const double r2 = r * r;
  if (sh == 2) {
    double Rsc[3] = {C[0] - R0[0], C[1] - R0[1], C[2] - R0[2]};
    const double RD = dot3(Rsc, D);
    const double RR = dot3(Rsc, Rsc);
    if (RR > r2 - 1e-10) {
      if (RD <= 0.0) return false;
    }
    const double Dd = RD * RD + r2 - RR;
    if (Dd < 0.0) return false;
    const double sq = sqrt(Dd);
    const double L1 = RD - sq, L2 = RD + sq;
    if (L1 > 0.0) *L = L1;
    else if (L2 > 0.0) *L = L2;
    else return false;
    return true;
  }
  /* z-axis cylinder clipped to 0 <= z <= Lz */
  const double Rs0 = C[0] - R0[0], Rs1 = C[1] - R0[1];
  double t0 = D[0], t1 = D[1];
  const double nv = t0 * t0 + t1 * t1 + 0.0 * 0.0;
  const double snv = sqrt(nv);
  t0 = t0 / snv;
  t1 = t1 / snv;
  const double RD = Rs0 * t0 + Rs1 * t1;
  const double RR = Rs0 * Rs0 + Rs1 * Rs1;
  const double Dd = RD * RD + r2 - RR;
  if (Dd < 0.0) return false;
  const double sq = sqrt(Dd);
  const double L1 = RD - sq, L2 = RD + sq;
  double Lh;
  if (L1 > 0.0) Lh = L1;
  else if (L2 > 0.0) Lh = L2;
  else return false;
  Lh = Lh / sqrt(D[0] * D[0] + D[1] * D[1]);
  const double z = R0[2] + D[2] * Lh;
  if (z < 0.0 || g.box[2] < z) return false;
  *L = Lh;
  return true;
}

/* calcSurfaceNormal*, src/RTMCphon.f90:3119-3179 */
template <int EXT>
__device__ void surface_normal(const Geo64& g, int k, const double* R, double* N) {
  const int sh = g.shape[k];
  if (sh == 1) {
    N[0] = g.normal[3 * k]; N[1] = g.normal[3 * k + 1]; N[2] = g.normal[3 * k + 2];
    return;
  }
  if (EXT && sh == 4) {
    capped_normal(g, k, R, N);
    return;
  }
  const double* C = g.center + 3 * k;
  double Rcs[3];
  if (sh == 2) {
    Rcs[0] = R[0] - C[0]; Rcs[1] = R[1] - C[1]; Rcs[2] = R[2] - C[2];
  } else {
    Rcs[2] = 0.0; Rcs[0] = R[0] - C[0]; Rcs[1] = R[1] - C[1];
  }
  const double rr = dot3(Rcs, Rcs);
  const double inv = 1.0 / sqrt(rr);
  for (int d = 0; d < 3; ++d) N[d] = Rcs[d] * inv;
  if (rr > g.radius[k] * g.radius[k])
    for (int d = 0; d < 3; ++d) N[d] = -1.0 * N[d];
}

/* calcSurfaceRotation*, src/RTMCphon.f90:3181-3301 (column-major) */
template <int EXT>
__device__ void surface_rotation(const Geo64& g, int k, const double* R, double* Rm) {
  const int sh = g.shape[k];
  if (sh == 1) {
    for (int d = 0; d < 9; ++d) Rm[d] = g.tangent[9 * k + d];
    return;
  }
  const double* C = g.center + 3 * k;
  double n[3];
  if (EXT && sh == 4) {
    capped_normal(g, k, R, n);
  } else if (sh == 2) {
    double Rcs[3] = {R[0] - C[0], R[1] - C[1], R[2] - C[2]};
    const double inv = 1.0 / sqrt(dot3(Rcs, Rcs));
    for (int d = 0; d < 3; ++d) n[d] = Rcs[d] * inv;
  } else {
    double Nn[3] = {R[0] - C[0], R[1] - C[1], 0.0};
    const double inv = 1.0 / sqrt(dot3(Nn, Nn));
    for (int d = 0; d < 3; ++d) n[d] = Nn[d] * inv;
  }
  Rm[6] = n[0]; Rm[7] = n[1]; Rm[8] = n[2];
  const double pole = (sh == 3) ? fabs(n[0]) : fabs(n[2]);
  if (pole == 1.0 || (n[0] * n[0] == 0.0 && n[1] * n[1] == 0.0)) {
    Rm[3] = 0; Rm[4] = 1; Rm[5] = 0; Rm[0] = 1; Rm[1] = 0; Rm[2] = 0;
  } else {
    const double q = sqrt(n[0] * n[0] + n[1] * n[1]);
    Rm[3] = -n[1] / q; Rm[4] = n[0] / q; Rm[5] = 0.0;
    cross3(&Rm[3], &Rm[6], &Rm[0]);
  }
}

/* determinTransmit threshold, src/RTMCphon.f90:2384-2413 */
__device__ double threshold(const Geo64& g, int k, double omega, double od) {
  const int kt = g.kind_trans[k];
  const double tp = g.tparam[k];
  if (kt == 1) return tp;
  if (kt == 2 || kt == 3) {
    if (g.nmaterial == 1) return 1.0 / (tp * omega / g.max_omega + 1.0);
    const double t11 = 1.0 / (tp + 1.0);
    return t11 + od * (1 - t11);
  }
  return 0.0;
}

/* A phonon: position, direction, free path, the surface last met (grain and
   its index there; -1 after an intrinsic event) and the grain it is in. */
struct Ph64 {
  double pos[3], dir[3], fp;
  int igrain, isurf, which;
};

/* Emission; returns EndSide (1 when the direction points back out). */
__device__ int emit64(const Geo64& g, const Task64& t, const Draw& rng, Ph64& p) {
  const double Y = g.box[1], Z = g.box[2];
  double d0, d1, e0, e1;
  rng.block(0, 0, &d0, &d1);
  p.pos[0] = 0.0; p.pos[1] = d0 * Y * g.scope[0]; p.pos[2] = d1 * Z * g.scope[1];
  rng.block(0, 1, &e0, &e1);
  double sphi, cphi;
  dsincos_2pi(e0, &sphi, &cphi);
  p.dir[0] = t.cth; p.dir[1] = t.sth * cphi; p.dir[2] = t.sth * sphi;
  p.igrain = 0;
  p.isurf = 0;
  p.which = 0;
  if (g.kind_grain == 1) {
    double dmin = 1.0e10;
    for (int ig = 1; ig <= g.ngrain; ++ig) {
      if (!g.grain_incident[ig]) continue;
      const double* G = g.grain_gen + 3 * ig;
      const double a = p.pos[0] - G[0], b = p.pos[1] - G[1], c = p.pos[2] - G[2];
      const double d2 = a * a + b * b + c * c;
      if (dmin > d2) { dmin = d2; p.which = ig; }
    }
  } else {
    bool found = false;
    for (int ig = 1; ig <= g.ngrain; ++ig) {
      if (!g.grain_incident[ig]) continue;
      for (int k = g.grain_begin[ig]; k < g.grain_begin[ig + 1]; ++k) {
        if (!g.incident[k]) continue;
        if (in_polygon(g.vertex + 3 * (size_t)g.vbegin[k], g.nvertex[k], p.pos)) {
          p.which = ig;
          found = true;
          break;
        }
      }
    }
    if (!found) p.which = g.igrain_fill;
  }
  p.fp = (t.lambda == kBallistic) ? kBallistic : -t.lambda * dlog_pos(e1);
  return (p.dir[0] <= 0.0) ? 1 : 0;
}

__device__ __forceinline__ bool in_box64(const Geo64& g, const double* pos) {
  return pos[0] >= 0.0 - kSmall && pos[0] <= g.box[0] + kSmall && pos[1] >= 0.0 - kSmall &&
         pos[1] <= g.box[1] + kSmall && pos[2] >= 0.0 - kSmall && pos[2] <= g.box[2] + kSmall;
}

/* What an event of a flight draws: blocks 0 and 1, and the sine and cosine of
   its azimuth (an intrinsic event: from d1, a diffuse wall: from f0). */
struct Drawn64 {
  double d0, d1, f0, f1, sp, cp;
};

__device__ __forceinline__ void draw64(const Draw& rng, uint32_t fl, bool pp, Drawn64& w) {
  rng.block(fl, 0, &w.d0, &w.d1);
  rng.block(fl, 1, &w.f0, &w.f1);
  dsincos_2pi(pp ? w.d1 : w.f0, &w.sp, &w.cp);
}

/* Isotropic direction and free path of an intrinsic event (a used-up free
   path draws from block 1). */
__device__ __forceinline__ void pp_dir64(const Drawn64& w, double lambda, double* dir, double* fp) {
  const double ct = w.d0 * 2.0 - 1.0;
  const double st = sqrt(1.0 - ct * ct);
  dir[0] = ct; dir[1] = st * w.cp; dir[2] = st * w.sp;
  *fp = -lambda * dlog_pos(w.f0);
}

__device__ __forceinline__ void pp_draw64(const Draw& rng, double lambda, uint32_t fl, double* dir,
                                          double* fp) {
  Drawn64 w;
  draw64(rng, fl, true, w);
  pp_dir64(w, lambda, dir, fp);
}

/* A flight ends in an intrinsic event after its whole free path. */
__device__ __forceinline__ void pp_event64(const Drawn64& w, double lambda, Ph64& p) {
  for (int d = 0; d < 3; ++d) p.pos[d] = p.pos[d] + p.fp * p.dir[d];
  pp_dir64(w, lambda, p.dir, &p.fp);
  for (int d = 0; d < 3; ++d) p.pos[d] = p.pos[d] + 1.0e-7 * p.dir[d];
  p.igrain = 0;
  p.isurf = -1;
}

/* Flight fl ends after `distance` at surface p.isurf of grain p.igrain:
   bath, periodic face, reflection or transmission (src/RTMCphon.f90:1744-1792,
   2225-2413).  Returns EndSide (0 lost, 1 x-, 2 x+), -1 while it goes on.
   DRAWN: the caller has drawn w, else it is drawn here, where it is needed. */
template <bool DRAWN, int EXT>
__device__ int surface_event64(const Geo64& g, double lambda, double omega, const Draw& rng,
                               uint32_t fl, double distance, const Drawn64& w, Ph64& p) {
  double* const pos = p.pos;
  double* const dir = p.dir;
  int end_side = -1, Jreflect = 1;
  double d0, d1;
  for (int d = 0; d < 3; ++d) pos[d] = pos[d] + distance * dir[d];
  if (p.isurf < 0) {
    return 0;
  } else if (p.igrain == 0 && p.isurf == 0) {
    end_side = 1;
  } else if (p.igrain == 0 && p.isurf == 1) {
    end_side = 2;
  } else if (p.igrain == 0 && g.face_kind[p.isurf] == 1) {
    const int ax = p.isurf >> 1;
    const double L = g.box[ax];
    const double sg = (p.isurf & 1) == 0 ? L : -L;
    if (ax == 1) pos[1] = pos[1] + sg;
    else pos[2] = pos[2] + sg;
  } else {
    const int k = g.grain_begin[p.igrain] + p.isurf;
    if (DRAWN) { d0 = w.d0; d1 = w.d1; }
    else rng.block(fl, 0, &d0, &d1);
    double od = 0.0;
    if (g.nmaterial != 1 && (g.kind_trans[k] == 2 || g.kind_trans[k] == 3)) {
      double x;
      rng.block(fl, 2, &od, &x);
    }
    if (d0 <= g.spec[k]) {
      const double thr = threshold(g, k, omega, od);
      if (d1 <= thr) {
        Jreflect = 0;
      } else {
        double N[3];
        surface_normal<EXT>(g, k, pos, N);
        if (dot3(N, dir) < 0) for (int d = 0; d < 3; ++d) N[d] = -1.0 * N[d];
        const double dn = dot3(N, dir);
        for (int d = 0; d < 3; ++d) dir[d] = dir[d] - 2.0 * N[d] * dn;
        Jreflect = 1;
      }
    } else {
      double N[3], Rm[9];
      surface_normal<EXT>(g, k, pos, N);
      if (dot3(N, dir) < 0.0) for (int d = 0; d < 3; ++d) N[d] = -1.0 * N[d];
      surface_rotation<EXT>(g, k, pos, Rm);
      double f0, f1, sp, cp;
      if (DRAWN) {
        f1 = w.f1; sp = w.sp; cp = w.cp;
      } else {
        rng.block(fl, 1, &f0, &f1);
        dsincos_2pi(f0, &sp, &cp);
      }
      const double sint = sqrt(d1);
      const double cost = sqrt(1.0 - sint * sint);
      const double td[3] = {sint * cp, sint * sp, cost};
      double v[3];
      for (int i = 0; i < 3; ++i) v[i] = Rm[i] * td[0] + Rm[3 + i] * td[1] + Rm[6 + i] * td[2];
      if (dot3(dir, N) > 0.0) {
        for (int i = 0; i < 3; ++i) dir[i] = -v[i];
      } else {
        for (int i = 0; i < 3; ++i) dir[i] = v[i];
      }
      if (dot3(dir, N) > 0.0) for (int i = 0; i < 3; ++i) dir[i] = -1.0 * dir[i];
      const double thr = threshold(g, k, omega, od);
      if (f1 <= thr) {
        for (int i = 0; i < 3; ++i) dir[i] = -dir[i];
        Jreflect = 0;
      } else {
        Jreflect = 1;
      }
    }
  }
  for (int d = 0; d < 3; ++d) pos[d] = pos[d] + 1.0e-7 * dir[d];
  if (lambda == kBallistic) {
    p.fp = kBallistic;
  } else {
    p.fp = p.fp - distance;
    if (p.fp < 1.0e-10) {
      double r0, r1;
      rng.block(fl, 2, &r0, &r1);
      p.fp = -lambda * dlog_pos(r1);
    }
  }
  if (Jreflect == 0) p.which = g.gout[g.grain_begin[p.igrain] + p.isurf];
  return end_side;
}

/* One trajectory; returns EndSide (0 lost, 1 x-, 2 x+). */
__device__ int trace(const Geo64& g, const Task64& t, const Draw& rng, int64_t max_flights,
                     uint64_t* nflights, bool* capped, double* fpos) {
  Ph64 p;
  int EndSide = emit64(g, t, rng, p);
  uint64_t flight = 0;
  *capped = false;
  while (EndSide == 0) {
    if (!in_box64(g, p.pos)) break;
    if ((int64_t)flight >= max_flights) { *capped = true; break; }
    ++flight;
    double distance = 1.0e10;
    int ig_min = p.igrain, is_min = p.isurf;
    for (int pass = 0; pass < 2; ++pass) {
      const int ig = pass == 0 ? 0 : p.which;
      if (pass == 1 && p.which == 0) break;
      const int kb = g.grain_begin[ig], ke = g.grain_begin[ig + 1];
      for (int k = kb; k < ke; ++k) {
        if (!g.internal[k]) continue;
        double L;
        if (surface_distance<false, 2>(g, k, p.pos, p.dir, 0.0, &L) && distance > L) {
          distance = L;
          ig_min = ig;
          is_min = k - kb;
        }
      }
    }
    if (p.fp < distance) {
      Drawn64 w;
      draw64(rng, (uint32_t)flight, true, w);
      pp_event64(w, t.lambda, p);
    } else {
      p.igrain = ig_min;
      p.isurf = is_min;
      const int e = surface_event64<false, 2>(g, t.lambda, t.omega, rng, (uint32_t)flight, distance,
                                           Drawn64(), p);
      if (e == 0) break;
      if (e > 0) EndSide = e;
    }
  }
  *nflights = flight;
  if (fpos) { fpos[0] = p.pos[0]; fpos[1] = p.pos[1]; fpos[2] = p.pos[2]; }
  return EndSide;
}

__device__ __forceinline__ void warp_add_by_task(bool pred, long long task,
                                                 unsigned long long* arr) {
  const unsigned m = __ballot_sync(0xffffffffu, pred);
  if (pred) {
    const unsigned peers = __match_any_sync(m, (unsigned long long)task);
    const int lane = threadIdx.x & 31;
    if (lane == __ffs(peers) - 1) atomicAdd(arr + task, (unsigned long long)__popc(peers));
  }
}

__global__ void __launch_bounds__(128) k_plain_fp64(Geo64 g, Run64 r) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t task, j;
  if (r.replay_task >= 0) {
    task = r.replay_task;
    j = gid;
  } else {
    task = gid / r.np_local;
    j = gid - task * r.np_local;
  }
  const bool active = (r.replay_task >= 0) ? (gid < r.np_local) : (task < r.ntask);
  int es = -1;
  uint64_t nf = 0;
  bool capped = false;
  bool run = false;
  if (active) {
    const Task64 t = r.task[task];
    if (t.lambda > 0.0) {
      run = true;
      const int64_t p = r.rank + j * (int64_t)r.nranks;
      const uint64_t sample = (uint64_t)task * (uint64_t)r.np + (uint64_t)p;
      Draw rng;
      rng.key.k0 = r.k0;
      rng.key.k1 = r.k1;
      rng.c1 = r.c1;
      rng.slo = (uint32_t)sample;
      rng.shi = (uint32_t)(sample >> 32);
      double fp[3];
      es = trace(g, t, rng, r.max_flights, &nf, &capped, fp);
      if (r.replay_task >= 0) {
        r.end_side[j] = es;
        r.flights[j] = (unsigned)nf;
        r.final_pos[3 * j] = fp[0];
        r.final_pos[3 * j + 1] = fp[1];
        r.final_pos[3 * j + 2] = fp[2];
      }
    } else if (r.replay_task >= 0) {
      r.end_side[j] = 0;
      r.flights[j] = 0;
      r.final_pos[3 * j] = r.final_pos[3 * j + 1] = r.final_pos[3 * j + 2] = 0.0;
    }
  }
  const bool trans = run && (es == 2 || (es == 0 && r.ref_quirks));
  const bool lostp = run && es == 0;
  warp_add_by_task(trans, task, r.counts);
  warp_add_by_task(lostp, task, r.lost);
  /* warp totals of flights / lost / capped / samples */
  unsigned long long v0 = nf, v1 = lostp, v2 = capped, v3 = run;
  for (int o = 16; o > 0; o >>= 1) {
    v0 += __shfl_xor_sync(0xffffffffu, v0, o);
    v1 += __shfl_xor_sync(0xffffffffu, v1, o);
    v2 += __shfl_xor_sync(0xffffffffu, v2, o);
    v3 += __shfl_xor_sync(0xffffffffu, v3, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (v0) atomicAdd(r.stats + 0, v0);
    if (v1) atomicAdd(r.stats + 1, v1);
    if (v2) atomicAdd(r.stats + 2, v2);
    if (v3) atomicAdd(r.stats + 3, v3);
  }
}

/* ---- persistent FP64 transport ------------------------------------------- */

/* Nearest surface of the box and of grain `which` no farther than the
   flight's free path (one beyond it cannot end the flight): the same surface,
   distance and tie (box before grain, then the lower index) as the linear
   scan.  What the scan does for every surface is left out where it cannot
   matter:
     - the box faces, which the host found to be axis-aligned rectangles
       (box_is_axis_aligned), are met at (face - x) / d, which is the general
       formula's value with a normal of +-1 and zeros, and a hit well inside
       the rectangle needs no edge test;
     - a plane crossed beyond the nearest hit so far is left early;
     - a grain with a BVH is walked in FP32: the node boxes are padded by 4 eps
       and positions rounded by 2^-24 of the box, so no node that holds the
       hit is skipped.
   Returns whether there is a hit; box_only leaves the grain's surfaces out. */
template <int EXT>
__device__ bool nearest64(const Geo64& g, const Geo<false>& G, float eps, const double* pos,
                          const double* dir, double fp, int which, bool box_only, double* dist,
                          int* igrain, int* isurf) {
  double best = fp < 1.0e10 ? __longlong_as_double(__double_as_longlong(fp) + 1) : 1.0e10;
  bool hit = false;
  const double m = (double)eps;
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const double d = dir[ax];
    const double w = (d > 0.0 ? g.box[ax] : 0.0) - pos[ax];
    if (d == 0.0) continue;
    if (d > 0.0 ? (w < 0.0 || w > best * d * 1.000001) : (w > 0.0 || w < best * d * 1.000001))
      continue;
    const double L = w / d;
    if (!(best > L)) continue;
    const int b = ax == 0 ? 1 : 0, c = ax == 2 ? 1 : 2;
    const double hb = pos[b] + dir[b] * L, hc = pos[c] + dir[c] * L;
    const int k = 2 * ax + (d > 0.0 ? 1 : 0);
    bool in = hb > m && hb < g.box[b] - m && hc > m && hc < g.box[c] - m;
    if (!in) {
      const double Rh[3] = {pos[0] + dir[0] * L, pos[1] + dir[1] * L, pos[2] + dir[2] * L};
      in = in_polygon(g.vertex + 3 * (size_t)g.vbegin[k], 4, Rh);
    }
    if (in) { best = L; *igrain = 0; *isurf = k; hit = true; }
  }
  if (which > 0 && !box_only) {
    const int kb0 = g.grain_begin[which];
    const int root = EXT ? G.bvh_root(which) : -1;
    if (root < 0) {
      const int kb = G.cand_begin(which), ke = G.cand_begin(which + 1);
      for (int i = kb; i < ke; ++i) {
        const int k = G.cand(i);
        double L;
        if (surface_distance<true, EXT>(g, k, pos, dir, best, &L) && best > L) {
          best = L; *igrain = which; *isurf = k - kb0; hit = true;
        }
      }
    } else if (EXT && !behind_planes(G, which, (float)pos[0], (float)pos[1], (float)pos[2], (float)dir[0],
                              (float)dir[1], (float)dir[2], (float)fp, eps)) {
      const float px = (float)pos[0], py = (float)pos[1], pz = (float)pos[2];
      const float ix = inv_dir((float)dir[0]), iy = inv_dir((float)dir[1]),
                  iz = inv_dir((float)dir[2]);
      int stk[kBvhStack];
      float stt[kBvhStack];
      int sp = 0, node = root;
      bool mine = false;  /* the hit so far is one of this grain's */
      while (true) {
        const int cnt = __float_as_int(G.node(2 * node + 1).w);
        const int a = __float_as_int(G.node(2 * node).w);
        /* the nearest hit as an FP32 bound, rounded up by its tolerance */
        float tm = fminf((float)best * 1.00001f + eps, 3.0e38f);
        bool descended = false;
        if (cnt > 0) {
          for (int i = a; i < a + cnt; ++i) {
            const int k = G.cand(i);
            double L;
            if (surface_distance<true, EXT>(g, k, pos, dir, best, &L) &&
                (best > L || (mine && best == L && k - kb0 < *isurf))) {
              best = L; *igrain = which; *isurf = k - kb0; hit = true; mine = true;
            }
          }
          tm = fminf((float)best * 1.00001f + eps, 3.0e38f);
        } else {
          const float tl = box_entry(G.node(2 * a), G.node(2 * a + 1), px, py, pz, ix, iy, iz, tm, eps);
          const float tg = box_entry(G.node(2 * a + 2), G.node(2 * a + 3), px, py, pz, ix, iy, iz, tm,
                                     eps);
          const bool hl = tl < 3.0e38f, hg = tg < 3.0e38f;
          if (hl || hg) {
            const bool lf = hl && (!hg || tl <= tg);
            if (hl && hg && sp < kBvhStack) {
              stk[sp] = lf ? a + 1 : a;
              stt[sp] = lf ? tg : tl;
              ++sp;
            }
            node = lf ? a : a + 1;
            descended = true;
          }
        }
        if (descended) continue;
        bool found = false;
        while (sp > 0) {
          --sp;
          if (stt[sp] <= tm) {
            node = stk[sp];
            found = true;
            break;
          }
        }
        if (!found) break;
      }
    }
  }
  *dist = hit ? best : 1.0e10;
  return hit;
}

/* Safe ball and grain ball about pos from the FP32 bounds (kernels_fp32.cu),
   less the rounding of the centre, the 1e-7 nudges and the few 1e-8 of the
   box by which an FP64 root can be off: radius squared, 0 for none. */
template <int EXT>
__device__ __forceinline__ void ball64(const Geo<false>& G, const GeoF32& gp, int which,
                                       const double* pos, float lam, float* bx, float* by,
                                       float* bz, float* br2, float* gr2) {
  *bx = (float)pos[0]; *by = (float)pos[1]; *bz = (float)pos[2];
  float dg, dg2;
  int near;
  const float d = safety<EXT>(G, which, *bx, *by, *bz, gp.box[0], gp.box[1], gp.box[2], gp.eps,
                               kBallCap64 * lam, dg, dg2, near) - 1.0e-6f;
  dg -= 1.0e-6f;
  *br2 = d > 0.0f ? d * d : 0.0f;
  *gr2 = dg > 0.0f ? dg * dg : 0.0f;
}

/* Squared distance of p from the ball's centre, in FP32. */
__device__ __forceinline__ float off2(const double* p, float bx, float by, float bz) {
  const float x = (float)p[0] - bx, y = (float)p[1] - by, z = (float)p[2] - bz;
  return fmaf(x, x, fmaf(y, y, z * z));
}

__device__ __forceinline__ Draw sample_draw(const Run64& r, uint64_t sample) {
  Draw rng;
  rng.key.k0 = r.k0;
  rng.key.k1 = r.k1;
  rng.c1 = r.c1;
  rng.slo = (uint32_t)sample;
  rng.shi = (uint32_t)(sample >> 32);
  return rng;
}

__device__ __forceinline__ float4 pack2(double a, double b) {
  return make_float4(__int_as_float(__double2loint(a)), __int_as_float(__double2hiint(a)),
                     __int_as_float(__double2loint(b)), __int_as_float(__double2hiint(b)));
}
__device__ __forceinline__ void unpack2(float4 v, double* a, double* b) {
  *a = __hiloint2double(__float_as_int(v.y), __float_as_int(v.x));
  *b = __hiloint2double(__float_as_int(v.w), __float_as_int(v.z));
}

#ifdef PT_CHECK
__device__ __noinline__ void check_finite64(const Ph64& p, int task) {
  for (int d = 0; d < 3; ++d)
    if (!isfinite(p.pos[d]) || !isfinite(p.dir[d]) || isnan(p.fp)) { check_fail(2, task); return; }
}
#endif

/* ---- the two phases ---------------------------------------------------------
   The plain kernel is bound by latency: one lane per phonon, every flight a
   scan of all surfaces by divergent lanes (about 4 us a flight), to the end of
   the longest trajectory.  Porous film, 2000 modes from 5 nm, 1e5 phonons:
   plain 27.8 ms, here 3.0; wire 300 x 60 nm, MFPs from 2 nm, 1e5 phonons:
   141 -> 6.1 ms; wire 1000 x 100 nm, gray MFP 150 nm, 3e4 phonons: 5.2 -> 2.1.
   What bounds them now is latency: 7 cycles a warp instruction in the tail
   (2.6 of them fixed latencies of the FP64 chains, 1.2 instruction fetch; 22
   lanes, SMs active for a quarter of it), times the rounds of the longest
   walk. */

/* Drain phase: the work queue, one phonon per lane, idle lanes refilled from
   the warp's chunk; flights that stay in the safe ball are taken without a
   scan; once the queue is dry the live phonons go to the tail list
   (grace_passes). */
template <int EXT>
__global__ void __launch_bounds__(256, 2) k_drain64(Geo64 g, GeoF32 gp, Run64 r) {
  Geo<false> G;
  G.base = gp.blob;
  G.lay = gp.lay;
  const int lane = threadIdx.x & 31;
  int ch_task = -1, ch_next = 0, ch_left = 0;
  bool queue_done = false;
  int grace = r.grace_steps;
  bool alive = false;
  Ph64 p;
  p.pos[0] = p.pos[1] = p.pos[2] = p.dir[0] = p.dir[1] = p.dir[2] = p.fp = 0.0;
  p.igrain = p.isurf = p.which = 0;
  double lambda = 1.0;
  float bx = 0, by = 0, bz = 0, br2 = 0, gr2 = 0;
  int task = 0;
  uint32_t flight = 0;
  uint64_t sample = 0;
  unsigned long long my_flights = 0, my_samples = 0, my_capped = 0, my_lost = 0;
  while (true) {
    int end_side = -1;
    unsigned idle = __ballot_sync(FULL, !alive);
    if (!queue_done && idle && (__popc(idle) >= r.regen_threshold || idle == FULL)) {
      while (idle && !queue_done) {
        if (ch_left == 0) {
          int c = 0;
          if (lane == 0) c = atomicAdd(r.queue, 1);
          c = __shfl_sync(FULL, c, 0);
          if (c >= r.nchunk) { queue_done = true; break; }
          const int3 q = queue_chunk(r.chunks, c);
          ch_task = q.x; ch_next = q.y; ch_left = q.z;
        }
        const int take = min(__popc(idle), ch_left);
        const int rank = __popc(idle & lanemask_lt());
        if (((idle >> lane) & 1u) && rank < take) {
          const int64_t q = (int64_t)r.rank + (int64_t)(ch_next + rank) * r.nranks;
          task = ch_task;
          sample = (uint64_t)task * (uint64_t)r.np + (uint64_t)q;
          const Task64 t = r.task[task];
          lambda = t.lambda;
          const int e = emit64(g, t, sample_draw(r, sample), p);
          end_side = e > 0 ? e : -1;
          br2 = gr2 = 0.0f;
          flight = 0;
          alive = true;
          my_samples += 1;
        }
        ch_next += take;
        ch_left -= take;
        idle = __ballot_sync(FULL, !alive);
      }
    }
    if (!__any_sync(FULL, alive)) {
      if (queue_done) break;
      continue;
    }
    if (queue_done && r.coop_lanes > 0 && __popc(__ballot_sync(FULL, alive)) <= r.coop_lanes) {
      /* A round costs about as much as a pass of 32 lanes (2100 warp
         instructions).  Where the MFP is the smallest box side or more nearly
         every flight ends at a surface, so those phonons stay to the end
         (wire 1000 x 100 nm, 1e5 phonons: MFP 1000 nm 4.39 -> 2.10 ms, 150 nm
         5.39 -> 3.66; at 30 nm it would be 7.68 -> 12.2). */
      const float lam = (float)lambda;
      const bool give = alive && end_side < 0 &&
                        (lam < r.fast_lambda_max || r.fast_steps <= 0 ||
                         (grace == 0 && lam < r.round_lambda_max));
      const unsigned mw = __ballot_sync(FULL, give);
      grace -= grace > 0 ? 1 : 0;
      if (mw) {
        const int fw = __ffs(mw) - 1;
        int base = 0;
        if (lane == fw) base = atomicAdd(r.queue + 4, __popc(mw));
        base = __shfl_sync(FULL, base, fw);
        const int idx = base + __popc(mw & lanemask_lt());
        /* the list has a slot for every lane of the grid */
        if (give && idx < r.tail_cap) {
          float4* e = r.tail + (size_t)kTail64Units * (r.tail_cap - 1 - idx);
          e[0] = make_float4(bx, by, bz, br2);
          e[1] = make_float4(gr2, 0.0f, 0.0f, 0.0f);
          e[2] = pack2(p.pos[0], p.pos[1]);
          e[3] = pack2(p.pos[2], p.dir[0]);
          e[4] = pack2(p.dir[1], p.dir[2]);
          e[5] = pack2(p.fp, lambda);
          const int bucket = order_bucket((float)p.pos[0], gp.box[0], lam);
          e[6] = make_float4(__int_as_float(p.igrain), __int_as_float(p.isurf),
                             __int_as_float(bucket), __int_as_float(p.which));
          atomicAdd(r.tail_hist + bucket, 1);
          e[7] = make_float4(__int_as_float(task), __uint_as_float((uint32_t)sample),
                             __uint_as_float((uint32_t)(sample >> 32)), __uint_as_float(flight));
          alive = false;
        }
        if (!__any_sync(FULL, alive)) break;
      }
    }
    const Draw rng = sample_draw(r, sample);
    /* ---- flights inside the safe ball, one a pass: past fast_steps only
       while half of the live lanes are still in theirs ---------------- */
    bool paused = false;
    {
      const int nalive = __popc(__ballot_sync(FULL, alive));
      bool fast = alive && end_side < 0 && br2 > 0.0f;
      for (int n = 0;; ++n) {
        if (fast) {
          double q[3];
          for (int d = 0; d < 3; ++d) q[d] = p.pos[d] + p.fp * p.dir[d];
          fast = (int64_t)flight < r.max_flights && off2(q, bx, by, bz) < br2;
        }
        const unsigned gm = __ballot_sync(FULL, fast);
        if (!gm) break;
        if (n >= r.fast_steps && (n >= 4 * r.fast_steps || 2 * __popc(gm) < nalive)) {
          paused = fast;
          break;
        }
        if (fast) {
          ++flight;
          Drawn64 w;
          draw64(rng, flight, true, w);
          pp_event64(w, lambda, p);
        }
      }
    }
    if (alive && !paused && end_side < 0) {
      if (!in_box64(g, p.pos)) {
        end_side = 0;
      } else if ((int64_t)flight >= r.max_flights) {
        end_side = 0;
        my_capped += 1;
      } else {
        ++flight;
        double q[3], distance;
        for (int d = 0; d < 3; ++d) q[d] = p.pos[d] + p.fp * p.dir[d];
        const bool box_only = off2(q, bx, by, bz) < gr2 && off2(p.pos, bx, by, bz) < gr2;
        const bool hit = nearest64<EXT>(g, G, gp.eps, p.pos, p.dir, p.fp, p.which, box_only, &distance,
                                   &p.igrain, &p.isurf);
        /* both kinds of event draw alike, before the lanes part */
        const bool pp = !hit && p.fp < 1.0e10;
        Drawn64 w;
        draw64(rng, flight, pp, w);
        if (pp) {
          pp_event64(w, lambda, p);
          br2 = 0.0f;
          if (r.fast_steps > 0 && (float)lambda < r.fast_lambda_max)
            ball64<EXT>(G, gp, p.which, p.pos, (float)lambda, &bx, &by, &bz, &br2, &gr2);
        } else {
          const int which = p.which;
          end_side = surface_event64<true, EXT>(g, lambda, r.task[task].omega, rng, flight, distance, w, p);
          br2 = 0.0f;
          if (p.which != which) gr2 = 0.0f;
        }
      }
    }
#ifdef PT_CHECK
    if (alive) check_finite64(p, task);
#endif
    const bool fin = alive && end_side >= 0;
    warp_add_by_task(fin && (end_side == 2 || (end_side == 0 && r.ref_quirks)), task, r.counts);
    warp_add_by_task(fin && end_side == 0, task, r.lost);
    if (fin) {
      my_flights += flight;
      my_lost += end_side == 0 ? 1 : 0;
      alive = false;
    }
  }
  unsigned long long v0 = my_flights, v1 = my_lost, v2 = my_capped, v3 = my_samples;
  for (int o = 16; o > 0; o >>= 1) {
    v0 += __shfl_xor_sync(FULL, v0, o);
    v1 += __shfl_xor_sync(FULL, v1, o);
    v2 += __shfl_xor_sync(FULL, v2, o);
    v3 += __shfl_xor_sync(FULL, v3, o);
  }
  if (lane == 0) {
    if (v0) atomicAdd(r.stats + 0, v0);
    if (v1) atomicAdd(r.stats + 1, v1);
    if (v2) atomicAdd(r.stats + 2, v2);
    if (v3) atomicAdd(r.stats + 3, v3);
  }
}

/* flights a round tests from its first one that walks a BVH */
constexpr int kTestWindow64 = 4;
/* flights in a row that have to be drawn for a round to go without drawing:
   at 4 / 8 / 16 / 24 the 300 nm wire takes 9.60 / 9.51 / 9.43 / 9.62 ms, and
   10.2 where every round draws all of its flights */
constexpr int kReady64 = 16;
/* double2 between the rows of a warp's round */
constexpr int kRow64 = 33;

/* Tail phase: one phonon per warp, 32 flights a round, one per lane.  Every
   lane holds the phonon.  A lane draws what its flight ends with if it ends
   in an intrinsic event (the blocks depend on the counter alone); the moves
   fp d and the nudges are products of those draws, so only their sums run one
   after the other: lane c < 3 adds coordinate c's, two additions a flight,
   through shared memory.  The first flight that meets a surface, leaves the
   box or reaches the cap ends the round, and every lane takes its event. */
template <int EXT>
__global__ void __launch_bounds__(256, 2) k_tail64(Geo64 g, GeoF32 gp, Run64 r) {
  __shared__ double2 rows[8][3 * kRow64];
  double2* const row = rows[threadIdx.x >> 5];
  Geo<false> G;
  G.base = gp.blob;
  G.lay = gp.lay;
  const int lane = threadIdx.x & 31;
  const int ntail = min(r.queue[4], r.tail_cap);
  unsigned long long my_flights = 0, my_capped = 0, my_lost = 0;
  while (true) {
    int c = 0;
    if (lane == 0) c = atomicAdd(r.queue + 3, 1);
    c = __shfl_sync(FULL, c, 0);
    if (c >= ntail) break;
    const float4* e = r.tail + (size_t)kTail64Units * r.tail_order[c];
    const float4 e0 = e[0], e1 = e[1], e6 = e[6], e7 = e[7];
    float bx = e0.x, by = e0.y, bz = e0.z, br2 = e0.w, gr2 = e1.x;
    Ph64 p;
    double lambda;
    unpack2(e[2], &p.pos[0], &p.pos[1]);
    unpack2(e[3], &p.pos[2], &p.dir[0]);
    unpack2(e[4], &p.dir[1], &p.dir[2]);
    unpack2(e[5], &p.fp, &lambda);
    p.igrain = __float_as_int(e6.x);
    p.isurf = __float_as_int(e6.y);
    p.which = __float_as_int(e6.w);
    const int task = __float_as_int(e7.x);
    const Draw rng = sample_draw(r, ((uint64_t)__float_as_uint(e7.z) << 32) | __float_as_uint(e7.y));
    uint32_t flight = __float_as_uint(e7.w);
    const double omega = r.task[task].omega;
    int end_side = -1;
    bool capped = false;
    double nd[3] = {0.0, 0.0, 0.0}, nf = 0.0;
    uint32_t drawn = 0;  /* the flight that the lane's draws are for */
    while (end_side < 0) {
      /* the lane's flight is the next whose number is `lane` modulo 32, so
         what it drew serves later rounds too; the lanes whose flight has
         passed draw again once fewer than kReady64 flights in a row are ready */
      const int base = (int)((flight + 1u) & 31u);
      const int off = (lane - base) & 31;
      const uint32_t mine = flight + 1u + (uint32_t)off;
      unsigned ready = __ballot_sync(FULL, drawn == mine);
      ready = __funnelshift_r(ready, ready, base);
      int nready = ready == FULL ? 32 : __ffs(~ready) - 1;
      if (nready < kReady64) {
        if (drawn != mine) {
          pp_draw64(rng, lambda, mine, nd, &nf);
          drawn = mine;
        }
        nready = 32;
        __syncwarp();
      }
      /* flight `off` starts with what the previous one drew */
      double sfp = __shfl_sync(FULL, nf, (lane - 1) & 31), sd[3];
      if (off == 0) sfp = p.fp;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        sd[d] = __shfl_sync(FULL, nd[d], (lane - 1) & 31);
        if (off == 0) sd[d] = p.dir[d];
        row[d * kRow64 + off] = make_double2(sfp * sd[d], 1.0e-7 * nd[d]);
      }
      __syncwarp();
      if (lane < 3) {
        double2* const q = row + lane * kRow64;
        double a = lane == 0 ? p.pos[0] : (lane == 1 ? p.pos[1] : p.pos[2]);
#pragma unroll
        for (int b = 0; b < 32; b += 8) {
          double2 v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = q[b + j];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            v[j].x = a + v[j].x;
            a = v[j].x + v[j].y;
            v[j].y = a;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) q[b + j] = v[j];
        }
      }
      __syncwarp();
      /* start point, end point before the nudge, and after it */
      double sp[3], sq[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        sq[d] = row[d * kRow64 + off].x;
        sp[d] = off == 0 ? p.pos[d] : row[d * kRow64 + (off > 0 ? off - 1 : 0)].y;
      }
      const float se = off2(sq, bx, by, bz), ss = off2(sp, bx, by, bz);
      const bool in_ball = se < br2 && ss < br2;
      const bool in_gball = se < gr2 && ss < gr2;
      const bool inbox = in_box64(g, sp);
      const bool brk = !inbox || (int64_t)flight + off >= r.max_flights;
      const bool walks =
          EXT && !in_ball && !in_gball && p.which > 0 && G.bvh_root(p.which) >= 0 &&
          !behind_planes(G, p.which, (float)sp[0], (float)sp[1], (float)sp[2], (float)sd[0],
                         (float)sd[1], (float)sd[2], (float)sfp, gp.eps);
      unsigned wm = __ballot_sync(FULL, walks);
      wm = __funnelshift_r(wm, wm, base);
      const int jw = wm ? min(nready, __ffs(wm) - 1 + kTestWindow64) : nready;
      double distance = 1.0e10;
      int ig = off == 0 ? p.igrain : 0, is = off == 0 ? p.isurf : -1;
      bool stop = brk;
      if (!brk && !in_ball && off < jw) {
        const bool hit = nearest64<EXT>(g, G, gp.eps, sp, sd, sfp, p.which, in_gball, &distance, &ig, &is);
        stop = hit || !(sfp < 1.0e10);
      }
      unsigned sm = __ballot_sync(FULL, stop && off < jw);
      sm = __funnelshift_r(sm, sm, base);
      const int j = sm ? __ffs(sm) - 1 : jw;
      const int jl = (base + j) & 31;      /* the lane of flight j ... */
      const int jp = (base + j - 1) & 31;  /* ... and of the one before */
      flight += (uint32_t)j;
      if (j < 32) {
        /* the state at the start of flight j */
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          p.pos[d] = __shfl_sync(FULL, sp[d], jl);
          p.dir[d] = __shfl_sync(FULL, sd[d], jl);
        }
        p.fp = __shfl_sync(FULL, sfp, jl);
      } else {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          p.pos[d] = row[d * kRow64 + 31].y;
          p.dir[d] = __shfl_sync(FULL, nd[d], jp);
        }
        p.fp = __shfl_sync(FULL, nf, jp);
      }
      __syncwarp();  /* the next round rewrites the rows */
      if (j > 0) { p.igrain = 0; p.isurf = -1; }
      if (sm) {
        if (__shfl_sync(FULL, (int)brk, jl)) {
          capped = __shfl_sync(FULL, (int)inbox, jl) != 0;
          end_side = 0;
          break;
        }
        const double L = __shfl_sync(FULL, distance, jl);
        p.igrain = __shfl_sync(FULL, ig, jl);
        p.isurf = __shfl_sync(FULL, is, jl);
        const int which = p.which;
        ++flight;
        end_side = surface_event64<false, EXT>(g, lambda, omega, rng, flight, L, Drawn64(), p);
        br2 = 0.0f;
        if (p.which != which) gr2 = 0.0f;
      } else if (r.fast_steps > 0 && !__shfl_sync(FULL, (int)in_gball, jp)) {
        /* a new ball where the walk left the grain ball */
        ball64<EXT>(G, gp, p.which, p.pos, (float)lambda, &bx, &by, &bz, &br2, &gr2);
      }
    }
#ifdef PT_CHECK
    if (lane == 0) check_finite64(p, task);
#endif
    my_flights += flight;
    my_capped += capped ? 1 : 0;
    my_lost += end_side == 0 ? 1 : 0;
    if (lane == 0) {
      if (end_side == 2 || (end_side == 0 && r.ref_quirks)) atomicAdd(r.counts + task, 1ull);
      if (end_side == 0) atomicAdd(r.lost + task, 1ull);
    }
  }
  if (lane == 0) {
    if (my_flights) atomicAdd(r.stats + 0, my_flights);
    if (my_lost) atomicAdd(r.stats + 1, my_lost);
    if (my_capped) atomicAdd(r.stats + 2, my_capped);
  }
}

}  // namespace

cudaError_t launch_plain_fp64(const Geo64& g, const Run64& r, cudaStream_t st, int* grid_out,
                              int* block_out) {
  const int block = 128;
  const int64_t nthreads = (r.replay_task >= 0) ? r.np_local : r.ntask * r.np_local;
  if (nthreads <= 0) return cudaSuccess;
  const int64_t grid = (nthreads + block - 1) / block;
  if (grid > 2147483647LL) return cudaErrorInvalidConfiguration;
  k_plain_fp64<<<(unsigned)grid, block, 0, st>>>(g, r);
  if (grid_out) *grid_out = (int)grid;
  if (block_out) *block_out = block;
  return cudaGetLastError();
}

/* Kernels without BVH and capped cylinders, or with both: a round's or pass's
   instructions are fetched again and again, and the shorter code stalls less
   for them (gray wire, 3e4 phonons: 2.25 -> 2.09 ms; porous film 3.19 -> 2.89,
   wire 300 x 60 nm 9.43 -> 8.97). */
cudaError_t drain64_occupancy(int block, int* bps, int ext) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, ext ? k_drain64<2> : k_drain64<0>, block, 0);
}

cudaError_t tail64_occupancy(int block, int* bps, int ext) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, ext ? k_tail64<2> : k_tail64<0>, block, 0);
}

cudaError_t launch_drain64(const Geo64& g, const GeoF32& gp, const Run64& r, int grid, int block,
                           cudaStream_t st) {
  if (block > 256 || block % 32) return cudaErrorInvalidConfiguration;
  if (gp.has_ext) k_drain64<2><<<grid, block, 0, st>>>(g, gp, r);
  else k_drain64<0><<<grid, block, 0, st>>>(g, gp, r);
  return cudaGetLastError();
}

cudaError_t launch_tail64(const Geo64& g, const GeoF32& gp, const Run64& r, int grid, int block,
                          cudaStream_t st) {
  if (block > 256 || block % 32) return cudaErrorInvalidConfiguration;
  if (gp.has_ext) k_tail64<2><<<grid, block, 0, st>>>(g, gp, r);
  else k_tail64<0><<<grid, block, 0, st>>>(g, gp, r);
  return cudaGetLastError();
}

#ifdef PT_CHECK
cudaError_t check_report_fp64(long long* count, int* code, int* index, bool reset) {
  return check_read(count, code, index, reset);
}
#endif

}  // namespace ptg
