// Ray tracing for the mixed-precision forward model.
//
// Same algorithm, step rule, refraction scheme and clipping as raytrace
// (jurassic.c:4201-4438, restated in FP64 in jgb_fp64.cu), with numerics
// chosen for GB300, whose FP64 pipe is ~64x narrower than FP32:
//  * the position x stays FP64 (three adds per step), but the altitude is
//    carried as z (FP64) plus exact FP32 increments
//      dz = (2 r (xhat . d) + |d|^2) / (r + sqrt(r^2 + 2 r (xhat . d) + |d|^2))
//    (no cancellation, relative error ~1e-7 of the step), so no FP64 square
//    roots, divisions or cart2geo per step;
//  * atmosphere interpolation (log-linear p, linear T, q, k; intpol_atm,
//    jurassic.c:3685-3706) runs in FP32 with per-level constants;
//  * the refractivity finite difference of the reference,
//    (N(xh + h e_k) - N(xh)) / h with N = 7.753e-5 p / T and h = 20 m,
//    is evaluated without cancellation:
//      N(z + dl) - N(z) = c p / (T T') (T expm1(s_p dl) - s_T dl)
//    inside one level (split at a level boundary), where N itself would only
//    carry ~7 significant digits in FP32;
//  * longitude and latitude are computed only at the points that use them
//    (first, last and the neighbours of the lowest point, for the tangent
//    point and the solar geometry);
//  * trapezoid lengths, column densities and Curtis-Godson sums in FP32
//    (compensated sums), written by the walk itself when the next point is
//    placed; the point data go to FP32 planes (z stays FP64);
//  * finite-difference perturbations in large EGA batches take their base
//    ray's geometry or walk on from the base's walk (TraceResume).
// The count and fill passes share the walk, so they agree on the point count.
#include "jgb_common.cuh"
#include "jgb_internal.h"

namespace jgb {
namespace {

constexpr float kRefracC = 7.753e-05f;

struct AtmM {
  int np;
  long long stride;
  const double *z, *p, *t, *q, *k;
  double clz, cldz, sfz, sfp, sft;
};

__device__ inline AtmM atm_m(const BatchDev& b, const CtlDev& c, int o) {
  AtmM a;
  const int l0 = b.lev_off[o];
  a.np = b.lev_off[o + 1] - l0;
  a.stride = b.nlev;
  a.z = b.z + l0;
  a.p = b.p + l0;
  a.t = b.t + l0;
  a.q = b.q + l0;
  a.k = b.k + l0;
  const double* s = b.scal + (long long)o * b.nscal;
  a.clz = s[0];
  a.cldz = s[1];
  a.sfz = s[2 + c.ncl];
  a.sfp = s[3 + c.ncl];
  a.sft = s[4 + c.ncl];
  return a;
}

// One level interval [z_i, z_i+1] of the profile in FP32 form.  Points are
// placed in it by their FP32 offset dl = z - z_i, so checking whether a
// point (or a refraction sub-point) is still in the interval needs no load.
struct Lev {
  int i;
  double z0;        // z_i
  float dz;         // z_i+1 - z_i
  float p0, p1, t0, t1;
  float sp;         // log(p1/p0)/dz (log-linear p) or (p1-p0)/dz (linear fallback)
  float st;         // (t1-t0)/dz
  bool plog;
  bool first, last; // lowest / highest interval (extrapolation below / above)
};

// x / y > 0, the division only where it might underflow or has special
// operands: positive numbers between 1e-154 and 1e154 need none.
static __device__ __noinline__ bool ratio_positive_rare(double x, double y) { return x / y > 0; }
__device__ __forceinline__ bool ratio_positive(double x, double y) {
  const unsigned hx = (unsigned)__double2hiint(x), hy = (unsigned)__double2hiint(y);
  if (hx - (512u << 20) < (1023u << 20) && hy - (512u << 20) < (1023u << 20)) return true;
  return ratio_positive_rare(x, y);
}

__device__ inline void lev_load(const AtmM& a, int i, Lev& L) {
  L.i = i;
  L.first = i == 0;
  L.last = i == a.np - 2;
  L.z0 = a.z[i];
  L.dz = d2f_bits(a.z[i + 1] - a.z[i]);
  L.p0 = d2f_bits(a.p[i]);
  L.p1 = d2f_bits(a.p[i + 1]);
  L.t0 = d2f_bits(a.t[i]);
  L.t1 = d2f_bits(a.t[i + 1]);
  L.plog = ratio_positive(a.p[i + 1], a.p[i]);
  L.sp = L.plog ? logf(L.p1 / L.p0) / L.dz : (L.p1 - L.p0) / L.dz;
  L.st = (L.t1 - L.t0) / L.dz;
}

// Is offset dl inside the interval (locate_irr semantics: the lowest
// interval also takes points below the grid, the highest those above)?
// Only for an ascending grid; otherwise the caller brackets.
__device__ inline bool lev_holds(const Lev& L, float dl) {
  return L.i >= 0 && L.dz > 0.f && (dl >= 0.f || L.first) && (dl < L.dz || L.last);
}

// Interval of z with the cached interval as hint, then its neighbour towards
// z (a ray or a refraction sub-point mostly crosses one level at a time:
// one round of independent loads instead of a bisection's chain); returns
// dl = z - z_i.  An interval that holds z is the one the bisection finds,
// so the hints change no result.
__device__ inline float lev_find(const AtmM& a, double z, Lev& L) {
  if (L.i >= 0) {
    const float dl = d2f_bits(z - L.z0);
    if (lev_holds(L, dl)) return dl;
    const int j = dl < 0.f ? L.i - 1 : L.i + 1;
    if (j >= 0 && j <= a.np - 2) {
      Lev M;
      lev_load(a, j, M);
      const float dm = d2f_bits(z - M.z0);
      if (lev_holds(M, dm)) {
        L = M;
        return dm;
      }
    }
  }
  lev_load(a, bracket_irr(a.z, a.np, z), L);
  return d2f_bits(z - L.z0);
}

__device__ inline void lev_pt(const Lev& L, float dl, float* p, float* t) {
  *p = L.plog ? L.p0 * __expf(L.sp * dl) : L.p0 + L.sp * dl;
  *t = L.t0 + L.st * dl;
}

// exp(x) - 1 for the small exponents of the refraction finite differences:
// the Taylor series to x^4 where |x| < 1/64 (truncation below x^4/120
// relative, far under FP32 rounding), else expm1f.
__device__ inline float expm1_small(float x) {
  if (fabsf(x) < 0.015625f)
    return x * (1.f + x * (0.5f + x * (0.16666667f + x * 0.041666668f)));
  return expm1f(x);
}

// N(z + dl) - N(z) inside one level, from p, T at z (no cancellation).
__device__ inline float dN_in(const Lev& L, float p, float t, float dl) {
  const float t2 = t + L.st * dl;
  if (L.plog) return kRefracC * p / (t * t2) * (t * expm1_small(L.sp * dl) - L.st * dl);
  return kRefracC * dl * (L.sp * t - p * L.st) / (t * t2);
}

// Altitude increment of a displacement d from a point at radius r with
// radial unit vector xh.
__device__ inline float dz_of(const float* xh, float r, const float* d) {
  const float u = xh[0] * d[0] + xh[1] * d[1] + xh[2] * d[2];
  const float dd = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
  const float num = 2.f * r * u + dd;
  return num / (r + sqrtf(r * r + num));
}

// Lon/lat bookkeeping of the fill pass (positions of the first and last
// point and of the neighbours of the lowest one).
struct GeoKeep {
  double x_first[3], x_m1[3], x_p1[3], x_last[3];
  double zmin_seen;
  double ds_clip;     // the clipped last segment (point n - 2) in FP64
  float ds_m, ds_p1;  // raw segment lengths of the lowest point and the next
  int imin;
  bool want_p1;
};

// The walk's state at LOS point n, for walking on from there: position,
// direction and altitude at the point, the previous point's position and
// altitude, and the previous point's level interval (the search hint).
struct WalkFrom {
  int n;
  double x[3], e[3], z;
  double x_last[3], z_last;
  int lev_last;
  float raw_last;  // raw segment length of the previous point
};

// Mixing ratio or extinction at offset dl in a level interval, from the
// level value v0 and the slope (v1 - v0) / dz, rounded after the product
// and after the sum (shared by the walk and the copies of a base's
// geometry, so both give the same bits).
__device__ __forceinline__ float qk_at(float v0, float slope, float dl) {
  return __fadd_rn(v0, __fmul_rn(slope, dl));
}

// Column density of a segment, 10 / k_B q p / T ds (p in hPa, ds in km).
__device__ __forceinline__ float col_density(float q, float p, float t, float ds) {
  return (float)(10.0 / kKB) * q * p / t * ds;
}

// Threads per block of the trace kernels (the fill pass keeps per-thread
// level caches in shared memory with this stride).
constexpr int kTraceThreads = 64;

// The emitter and window values of level i and their slopes (v1 - v0) / dz
// over interval i, into the per-thread cache qc (stride kTraceThreads):
// qc[k] = v0, qc[nqk + k] = slope, nqk = ng + nw.
__device__ __forceinline__ void level_values(const CtlDev& c, const AtmM& a, int i, float dz,
                                             float* qc) {
  const int nqk = c.ng + c.nw;
  for (int k = 0; k < nqk; k++) {
    const double* src = k < c.ng ? a.q + k * a.stride : a.k + (k - c.ng) * a.stride;
    const float v0 = d2f_bits(src[i]), v1 = d2f_bits(src[i + 1]);
    qc[k * kTraceThreads] = v0;
    qc[(nqk + k) * kTraceThreads] = (v1 - v0) / dz;
  }
}

// Per-thread shared memory of the fill pass, stride kTraceThreads: the
// current level's emitter and window values and slopes (qc[k], qc[nqk + k],
// nqk = ng + nw) and the mixing ratios of the point waiting for its trapezoid
// length (pq[ig]).
__host__ __device__ inline int trace_smem_floats(const CtlDev& c) {
  return 2 * (c.ng + c.nw) + c.ng;
}

// a < b on the integer pipe, false for NaN
__device__ __forceinline__ bool less(double a, double b) {
  return is_number(a) && is_number(b) && lt(a, b);
}

// The altitudes that end ray r: 1, or 0 for a ray above the atmosphere, -1 on
// error.
__device__ int ray_bounds_m(const CtlDev& c, const AtmM& a, const double* g, long long nray, int r,
                            double* zlo, double* zhi, unsigned* err) {
  const double obsz = g[1 * nray + r], vpz = g[4 * nray + r];
  double zmin = a.z[0], zmax = a.z[0];
  for (int i = 0; i < a.np; i++) {
    zmin = less(a.z[i], zmin) ? a.z[i] : zmin;
    zmax = less(zmax, a.z[i]) ? a.z[i] : zmax;
  }
  if (c.nsf > 0) {
    zmin = a.sfz > zmin ? a.sfz : zmin;
    if (a.sfp > 0) {
      const int i = bracket_irr(a.p, a.np, a.sfp);
      const double zs = lin(log(a.p[i]), a.z[i], log(a.p[i + 1]), a.z[i + 1], log(a.sfp));
      zmin = zs > zmin ? zs : zmin;
    }
  }
  if (obsz < zmin) {
    atomicOr(err, kErrObserverBelowSurface);
    return -1;
  }
  *zlo = zmin;
  *zhi = zmax;
  return vpz > zmax ? 0 : 1;
}

// Position, direction and altitude of ray r's first point.
__device__ void ray_first_m(const double* g, long long nray, int r, double zmax, double* x,
                            double* ex0, double* zout) {
  const double obsz = g[1 * nray + r], obslon = g[2 * nray + r], obslat = g[3 * nray + r];
  const double vpz = g[4 * nray + r], vplon = g[5 * nray + r], vplat = g[6 * nray + r];
  double z;
  double xobs[3], xvp[3];
  to_cart(obsz, obslon, obslat, xobs);
  to_cart(vpz, vplon, vplat, xvp);
  for (int i = 0; i < 3; i++) ex0[i] = xvp[i] - xobs[i];
  const double norm = sqrt(ex0[0] * ex0[0] + ex0[1] * ex0[1] + ex0[2] * ex0[2]);
  for (int i = 0; i < 3; i++) {
    ex0[i] /= norm;
    x[i] = xobs[i];
  }
  z = obsz;
  if (obsz > zmax) {  // entry into the atmosphere: bisection on the line of sight (FP64, once)
    double dmax = norm, dmin = 0;
    for (int guard = 0; fabs(dmin - dmax) > 0.001 && guard < 200; guard++) {
      const double d = (dmax + dmin) / 2;
      for (int i = 0; i < 3; i++) x[i] = xobs[i] + d * ex0[i];
      z = sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]) - kRE;
      if (z <= zmax && z > zmax - 0.001) break;
      if (z < zmax - 0.0005) dmax = d; else dmin = d;
    }
  }
  z = sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]) - kRE;
  *zout = z;
}

// STORE places every point with its final values: its trapezoid length
// 0.5 (ds_(i-1) + ds_i) and column densities 10 / k_B q p / T ds are written
// when the next point is placed (the clip of the last segment changes the
// previous point's raw length), so the walk keeps the raw lengths of the last
// two points.  It serves resumed perturbations, which are EGA only (no
// Curtis-Godson sums).  With wf it walks on from the state wf (a base's walk).
template <bool STORE>
__device__ int walk_m(const CtlDev& c, const AtmM& a, const double* g, long long nray, int r,
                      const LosDev& L, long long base, int cap, double* sft_out, GeoKeep* gk,
                      float* qc, unsigned* err, const WalkFrom* wf = nullptr) {
  const float h = 0.02f;
  const double zrefrac = 60;
  *sft_out = -999;
  double zmin, zmax;
  const int ok = ray_bounds_m(c, a, g, nray, r, &zmin, &zmax, err);
  if (ok <= 0) return ok;

  // the direction stays FP64: renormalising an FP32 unit vector every step
  // would random-walk it by ~1e-7 rad per step (metres over a limb path)
  double x[3], ex0[3], z;
  double last_z = 0, x_last[3] = {0, 0, 0};
  Lev lv;
  lv.i = -1;
  int n = 0, stop = 0, qc_level = -1;
  if (STORE && wf) {  // on from a base's walk
    for (int i = 0; i < 3; i++) {
      x[i] = wf->x[i];
      ex0[i] = wf->e[i];
      x_last[i] = wf->x_last[i];
    }
    z = wf->z;
    last_z = wf->z_last;
    n = wf->n;
    lev_load(a, wf->lev_last, lv);
  } else {
    ray_first_m(g, nray, r, zmax, x, ex0, &z);
  }
  const int nqk = c.ng + c.nw;
  const float rayds = (float)c.rayds, raydz = (float)c.raydz;
  // the direction in FP32 (carried from the previous step's conversion)
  float ef[3] = {(float)ex0[0], (float)ex0[1], (float)ex0[2]};
  // the point waiting for its final values (STORE): raw lengths of it and
  // of the point before, its p and T; its mixing ratios in pq
  float* pq = STORE ? qc + 2 * nqk * kTraceThreads : nullptr;
  float raw_before = 0.f, raw_pend = 0.f, pend_p = 0.f, pend_t = 0.f;
  const int n0 = n;
  if (STORE && wf) raw_pend = wf->raw_last;
  auto finalize = [&](int k) {
    const long long sk = base + k;
    const float dsT = k == 0 ? 0.5f * raw_pend : 0.5f * (raw_before + raw_pend);
    L.f.ds[sk] = dsT;
    for (int ig = 0; ig < c.ng; ig++) {
      const float uu = col_density(pq[ig * kTraceThreads], pend_p, pend_t, dsT);
      L.f.u[ig * L.cap + sk] = uu;
    }
  };
  for (;;) {
    // radial unit vector and radius at x
    const double rr = z + kRE;
    const float rf = d2f_bits(rr), rinv = 1.f / rf;
    float xh[3] = {d2f_bits(x[0]) * rinv, d2f_bits(x[1]) * rinv, d2f_bits(x[2]) * rinv};
    // step length from this point (jurassic.c:4278-4287)
    float step = rayds;
    if (raydz > 0) {
      const float cosa = fabsf(ef[0] * xh[0] + ef[1] * xh[1] + ef[2] * xh[2]);
      if (cosa != 0) step = rayds < raydz / cosa ? rayds : raydz / cosa;
    }
    // ground or top of the atmosphere: clip the last segment (4292-4306;
    // the previous point's step becomes this point's step times frac)
    const bool low = less(z, zmin);
    if ((low || less(zmax, z)) && n > 0) {
      if (!STORE) {
        if (n >= cap) {
          atomicOr(err, cap < c.nlos_max ? kErrSlabOverflow : kErrLosOverflow);
          return -1;
        }
        return n + 1;
      }
      stop = low ? 2 : 1;
      const double frac = ((low ? zmin : zmax) - last_z) / (z - last_z);
      for (int i = 0; i < 3; i++) x[i] = x_last[i] + frac * (x[i] - x_last[i]);
      z = last_z + frac * (z - last_z);
      const double dsc = (double)step * frac;
      raw_pend = (float)dsc;
      gk->ds_clip = dsc;
      step = 0.f;
    }
    if (n >= cap) {
      atomicOr(err, cap < c.nlos_max ? kErrSlabOverflow : kErrLosOverflow);
      return -1;
    }
    const float dl = lev_find(a, z, lv);
    float p, t;
    lev_pt(lv, dl, &p, &t);
    if (STORE) {
      if (n > n0) finalize(n - 1);
      const long long s = base + n;
      L.z[s] = z;
      L.f.p[s] = p;
      L.f.t[s] = t;
      raw_before = raw_pend;
      raw_pend = step;
      pend_p = p;
      pend_t = t;
      const int i = lv.i;
      if (i != qc_level) {  // a new level: its values and slopes q0 + (q1 - q0) / dz * dl
        qc_level = i;
        level_values(c, a, i, lv.dz, qc);
      }
      for (int ig = 0; ig < c.ng; ig++) {
        const float v = qk_at(qc[ig * kTraceThreads], qc[(nqk + ig) * kTraceThreads], dl);
        pq[ig * kTraceThreads] = v;
        if (ig == c.ig_h2o) L.f.qh2o[s] = v;
      }
      for (int iw = 0; iw < c.nw; iw++)
        L.f.kw[iw * L.cap + s] = qk_at(qc[(c.ng + iw) * kTraceThreads],
                                       qc[(nqk + c.ng + iw) * kTraceThreads], dl);
      if (c.ncl > 0 && a.cldz > 0) {
        const float v = (float)((z - a.clz) / a.cldz);
        L.f.aux[s] = expf(-0.5f * v * v);
      } else {
        L.f.aux[s] = 0.f;
      }
      // geometry kept for lon/lat of the points that need them
      if (n == 0)
        for (int i2 = 0; i2 < 3; i2++) gk->x_first[i2] = x[i2];
      if (gk->want_p1) {
        for (int i2 = 0; i2 < 3; i2++) gk->x_p1[i2] = x[i2];
        gk->ds_p1 = step;
        gk->want_p1 = false;
      }
      if (n == 0 || less(z, gk->zmin_seen)) {
        gk->zmin_seen = z;
        gk->imin = n;
        gk->ds_m = step;
        for (int i2 = 0; i2 < 3; i2++) gk->x_m1[i2] = x_last[i2];   // the previous point
        gk->want_p1 = true;
      }
    }
    last_z = z;
    for (int i2 = 0; i2 < 3; i2++) x_last[i2] = x[i2];
    n++;
    if (stop) {
      if (c.nsf > 0 && a.sft > 0) t = (float)a.sft;
      *sft_out = (stop == 2 ? (c.nsf > 0 && a.sft > 0 ? a.sft : (double)t) : -999);
      if (STORE) {
        for (int i2 = 0; i2 < 3; i2++) gk->x_last[i2] = x[i2];
        finalize(n - 1);
      }
      break;
    }
    // refraction (jurassic.c:4388-4415): ex1 = (n ex0 + ds grad N) / |...|
    // = (ex0 + inc) / |ex0 + inc| with inc = ds grad N / n, the increment in
    // FP32 and the renormalisation as a series in delta = |ex0 + inc|^2 - 1
    const bool bend = c.refrac && is_number(z) && !lt(zrefrac, z);
    double ex1[3] = {ex0[0], ex0[1], ex0[2]};
    if (bend) {
      const float nref = 1.f + kRefracC * p / t;
      // midpoint xh = x + ds/2 ex0 and its radial unit vector
      const float d[3] = {0.5f * step * ef[0], 0.5f * step * ef[1], 0.5f * step * ef[2]};
      const float dzh = dz_of(xh, rf, d);
      const float rh = rf + dzh, rhinv = 1.f / rh;
      const float xhh[3] = {(xh[0] * rf + d[0]) * rhinv, (xh[1] * rf + d[1]) * rhinv,
                            (xh[2] * rf + d[2]) * rhinv};
      // midpoint offset in the point's interval (FP64 only when it leaves it)
      Lev lh = lv;
      float dlh = dl + dzh;
      if (!lev_holds(lh, dlh)) dlh = lev_find(a, z + f2d_bits(dzh), lh);
      float ph, th;
      lev_pt(lh, dlh, &ph, &th);
      float inc[3];
      for (int k = 0; k < 3; k++) {
        float dk[3] = {0.f, 0.f, 0.f};
        dk[k] = h;
        const float dlk = dz_of(xhh, rh, dk);
        float dN;
        if (lev_holds(lh, dlh + dlk)) {
          dN = dN_in(lh, ph, th, dlk);
        } else {
          // split at the level boundary between the midpoint and zk
          const double zh = lh.z0 + f2d_bits(dlh), zk = zh + f2d_bits(dlk);
          Lev lk = lh;
          const float dlk0 = lev_find(a, zk, lk);
          if (lk.i == lh.i) {
            dN = dN_in(lh, ph, th, dlk);
          } else {
            const bool up = lk.i > lh.i;
            const double zb = up ? a.z[lh.i + 1] : a.z[lh.i];
            const float d1 = d2f_bits(zb - zh);
            const float dn1 = dN_in(lh, ph, th, d1);
            float pb, tb;
            const float dlb = d2f_bits(zb - lk.z0);
            lev_pt(lk, dlb, &pb, &tb);
            dN = dn1 + dN_in(lk, pb, tb, dlk0 - dlb);
          }
        }
        inc[k] = step * (dN / h) / nref;
      }
      const float delta = 2.f * (ef[0] * inc[0] + ef[1] * inc[1] + ef[2] * inc[2]) +
                          (inc[0] * inc[0] + inc[1] * inc[1] + inc[2] * inc[2]);
      for (int k = 0; k < 3; k++) ex1[k] = ex0[k] + f2d_bits(inc[k]);
      if (fabsf(delta) < 1e-3f) {
        const float corr = delta * (-0.5f + delta * (0.375f - 0.3125f * delta));
        for (int k = 0; k < 3; k++) ex1[k] += ex1[k] * f2d_bits(corr);
      } else {
        const double nn = sqrt(ex1[0] * ex1[0] + ex1[1] * ex1[1] + ex1[2] * ex1[2]);
        for (int k = 0; k < 3; k++) ex1[k] /= nn;
      }
    }
    float D[3], efn[3];
    for (int k = 0; k < 3; k++) {
      efn[k] = d2f_bits(ex1[k]);
      D[k] = 0.5f * step * (ef[k] + efn[k]);
    }
    const float dzs = dz_of(xh, rf, D);
    for (int k = 0; k < 3; k++) {
      x[k] += f2d_bits(D[k]);
      ex0[k] = ex1[k];
      ef[k] = efn[k];
    }
    z += f2d_bits(dzs);
  }
  return n;
}

__global__ void k_trace_count_m(CtlDev c, BatchDev b, LosDev L, unsigned* err) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= b.nray) return;
  if (b.obs_skip && b.obs_skip[b.ray_obs[r]]) {
    L.count[r] = 0;
    return;
  }
  const AtmM a = atm_m(b, c, b.ray_obs[r]);
  double sft;
  const int n = walk_m<false>(c, a, b.geo, b.nray, r, L, 0, c.nlos_max, &sft, nullptr, nullptr,
                              err);
  L.count[r] = n < 0 ? 0 : n;
}

// Upper bound of the LOS points of every ray, for tracing a large batch in
// one pass.  The step rule ds = min(RAYDS, RAYDZ/|cos a|) (jurassic.c:
// 4278-4287) makes every step either RAYDS long or move the point by RAYDZ
// along the local vertical, less the curvature term ds^2/(2 r) <=
// RAYDS^2/(2 RE).  A path of length S through a total altitude change V so
// takes at most S/RAYDS + V/(RAYDZ - RAYDS^2/(2 RE)) steps, plus the first
// and the clipped last point.  S and V come from the straight line of sight
// (entry at the top of the atmosphere, exit at the top or at the lowest
// level), with 10 % and, with refraction, 4 km of altitude as margins for
// the bending; the bound is scaled by jgb_set_los_bound_scale.  A ray that
// still outgrows its bound raises
// kErrSlabOverflow in the fill pass and the batch is traced again with
// exact counts, so the bound only decides the memory and the speed.
__global__ void k_los_bound_m(CtlDev c, BatchDev b, double scale, int* cap) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= b.nray) return;
  if (b.obs_skip && b.obs_skip[b.ray_obs[r]]) {
    cap[r] = 0;
    return;
  }
  const AtmM a = atm_m(b, c, b.ray_obs[r]);
  double zmin = a.z[0], zmax = a.z[0];
  for (int i = 1; i < a.np; i++) {
    zmin = fmin(zmin, a.z[i]);
    zmax = fmax(zmax, a.z[i]);
  }
  const long long nr = b.nray;
  const double* g = b.geo;
  const double obsz = g[1 * nr + r], vpz = g[4 * nr + r];
  if (vpz > zmax || obsz < zmin) {  // no LOS, or an error raised by the fill pass
    cap[r] = 2;
    return;
  }
  double xo[3], xv[3], d[3];
  to_cart(obsz, g[2 * nr + r], g[3 * nr + r], xo);
  to_cart(vpz, g[5 * nr + r], g[6 * nr + r], xv);
  const double dn = sqrt((xv[0] - xo[0]) * (xv[0] - xo[0]) + (xv[1] - xo[1]) * (xv[1] - xo[1]) +
                         (xv[2] - xo[2]) * (xv[2] - xo[2]));
  for (int i = 0; i < 3; i++) d[i] = dn > 0 ? (xv[i] - xo[i]) / dn : 0.0;
  // |xo + s d|^2 = r02 + 2 bb s + s^2
  const double bb = xo[0] * d[0] + xo[1] * d[1] + xo[2] * d[2];
  const double r02 = xo[0] * xo[0] + xo[1] * xo[1] + xo[2] * xo[2];
  const double rt = kRE + zmax, rb = kRE + zmin;
  const double disc_t = fmax(bb * bb - (r02 - rt * rt), 0.0);
  const double s_in = r02 > rt * rt ? fmax(-bb - sqrt(disc_t), 0.0) : 0.0;
  const double r_in = sqrt(fmax(r02 + 2 * bb * s_in + s_in * s_in, 0.0));
  const double s_t = -bb, rmin = sqrt(fmax(r02 - bb * bb, 0.0));
  double s_out, V;
  if (rmin < rb && s_t > s_in) {  // down to the lowest level
    s_out = -bb - sqrt(fmax(bb * bb - (r02 - rb * rb), 0.0));
    V = r_in - rb;
  } else {
    s_out = -bb + sqrt(disc_t);
    V = (s_t > s_in && s_t < s_out) ? (r_in - rmin) + (rt - rmin) : fabs(rt - r_in);
  }
  const double S = fmax(s_out - s_in, 0.0);
  double est = c.rayds > 0 ? S / c.rayds : 0.0;
  if (c.raydz > 0) {
    const double per = fmax(c.raydz - c.rayds * c.rayds / (2 * kRE), 0.5 * c.raydz);
    est += (V + (c.refrac ? 4.0 : 0.0)) / per;
  }
  const double bound = ceil(scale * 1.1 * est) + 16;
  cap[r] = bound >= (double)c.nlos_max ? c.nlos_max : (int)bound;
}

// Resumed perturbation of mode 2 (TraceResume): ray r takes base ray rb's
// LOS geometry, p, T, cloud weights, segment lengths, tangent point and
// ends, and evaluates its own mixing ratios and extinctions on the base's
// level intervals, as its own walk would.
__device__ void copy_base_geometry(const CtlDev& c, const BatchDev& b, const LosDev& L,
                                   const AtmM& a, int r, int rb, int cap, const TraceResume& R,
                                   float* qc, unsigned* err) {
  const long long base = L.off[r], ob = L.off[rb];
  const int n = L.count[rb];
  if (n > cap) {
    atomicOr(err, cap < c.nlos_max ? kErrSlabOverflow : kErrLosOverflow);
    return;
  }
  const long long nr = b.nray;
  for (int k = 0; k < 3; k++) b.tp[k * nr + r] = b.tp[k * nr + rb];
  for (int k = 0; k < 6; k++) L.ends[6LL * r + k] = L.ends[6LL * rb + k];
  L.sft[r] = L.sft[rb];
  L.count[r] = n;
  const int nqk = c.ng + c.nw;
  int qc_level = -1;
  double z0 = 0;
  for (int ip = 0; ip < n; ip++) {
    const long long q = ob + ip, s = base + ip;
    const double z = L.z[q];
    const float pf = L.f.p[q], tf = L.f.t[q], dsf = L.f.ds[q];
    L.z[s] = z;
    L.f.p[s] = pf;
    L.f.t[s] = tf;
    L.f.ds[s] = dsf;
    L.f.aux[s] = L.f.aux[q];
    const int i = R.lev[q];
    if (i != qc_level) {  // the walk's level values and slopes
      qc_level = i;
      z0 = a.z[i];
      level_values(c, a, i, (float)(a.z[i + 1] - a.z[i]), qc);
    }
    const float dl = (float)(z - z0);
    for (int ig = 0; ig < c.ng; ig++) {
      const float v = qk_at(qc[ig * kTraceThreads], qc[(nqk + ig) * kTraceThreads], dl);
      if (ig == c.ig_h2o) L.f.qh2o[s] = v;
      L.f.u[ig * L.cap + s] = col_density(v, pf, tf, dsf);
    }
    for (int iw = 0; iw < c.nw; iw++)
      L.f.kw[iw * L.cap + s] = qk_at(qc[(c.ng + iw) * kTraceThreads],
                                     qc[(nqk + c.ng + iw) * kTraceThreads], dl);
  }
}

// What a ray leaves beside its points: count, surface temperature, tangent
// point and ends.
__device__ void ray_finish_m(const BatchDev& b, const LosDev& L, int r, int n, double sft,
                             const GeoKeep& gk) {
  const long long base = L.off[r];
  L.sft[r] = sft;
  if (n > 0) L.count[r] = n;
  const long long nr = b.nray;
  double* tp = b.tp;
  // tangent point defaults to the view point (jurassic.c:4218-4220)
  tp[0 * nr + r] = b.geo[4 * nr + r];
  tp[1 * nr + r] = b.geo[5 * nr + r];
  tp[2 * nr + r] = b.geo[6 * nr + r];
  if (n <= 0) {
    L.count[r] = 0;
    return;
  }
  const double* z = L.z + base;
  double dummy, lon0, lat0, lonl, latl;
  to_geo(gk.x_first, &dummy, &lon0, &lat0);
  to_geo(gk.x_last, &dummy, &lonl, &latl);
  // tangent point (tangent_point, jurassic.c:5223-5263) from the raw lengths
  const int imin = gk.imin;
  if (imin <= 0 || imin >= n - 1) {
    tp[0 * nr + r] = z[n - 1];
    tp[1 * nr + r] = lonl;
    tp[2 * nr + r] = latl;
  } else {
    const double y0 = z[imin - 1], y1 = z[imin], y2 = z[imin + 1];
    // raw segment lengths (the clipped last one, of point n - 2, in FP64)
    const double d1 = imin == n - 2 ? gk.ds_clip : (double)gk.ds_m;
    const double d2 = imin + 1 == n - 2 ? gk.ds_clip : (double)gk.ds_p1;
    const double x1 = sqrt(d1 * d1 - (y1 - y0) * (y1 - y0));
    const double x2 = x1 + sqrt(d2 * d2 - (y2 - y1) * (y2 - y1));
    const double aa = 1 / (x1 - x2) * (-(y0 - y1) / x1 + (y0 - y2) / x2);
    const double bb = -(y0 - y1) / x1 - aa * x1;
    const double cc = y0;
    const double xt = -bb / (2 * aa);
    tp[0 * nr + r] = aa * xt * xt + bb * xt + cc;
    double v[3], tlon, tlat;
    for (int i = 0; i < 3; i++) v[i] = lin(0.0, gk.x_m1[i], x2, gk.x_p1[i], xt);
    to_geo(v, &dummy, &tlon, &tlat);
    tp[1 * nr + r] = tlon;
    tp[2 * nr + r] = tlat;
  }
  double* e = L.ends + 6LL * r;
  e[0] = z[0];
  e[1] = lon0;
  e[2] = lat0;
  e[3] = z[n - 1];
  e[4] = lonl;
  e[5] = latl;
}

// order (optional): thread t traces ray order[t], else ray r0 + t, so that a
// warp's rays have similar LOS capacities and finish together; each ray's
// outputs go to its own slots, so the order does not change any result.
// The perturbations of resumed tracing (R.plan; EGA only: the Curtis-Godson
// sums run from the first point).
__global__ void k_trace_fill_m(CtlDev c, BatchDev b, LosDev L, const int* order, int r0, int nr_l,
                               TraceResume R, unsigned* err) {
  const int th = blockIdx.x * blockDim.x + threadIdx.x;
  if (th >= nr_l) return;
  const int r = order ? order[th] : r0 + th;
  if (b.obs_skip && b.obs_skip[b.ray_obs[r]]) {
    L.count[r] = 0;
    return;
  }
  const AtmM a = atm_m(b, c, b.ray_obs[r]);
  const long long base = L.off[r];
  const int cap = L.count[r];
  extern __shared__ float qcache[];  // trace_smem_floats(c) per thread
  const int4 pl = R.plan[r];
  if (pl.z == 2) {
    copy_base_geometry(c, b, L, a, r, pl.x, cap, R, qcache + threadIdx.x, err);
    return;
  }
  double sft;
  GeoKeep gk;
  gk.want_p1 = false;
  gk.imin = 0;
  gk.zmin_seen = 0;
  gk.ds_clip = 0;
  gk.ds_m = gk.ds_p1 = 0.f;
  for (int i = 0; i < 3; i++) gk.x_m1[i] = gk.x_p1[i] = gk.x_first[i] = gk.x_last[i] = 0;
  // mode 1: points [0, m) are the base's (final values); the walk goes on
  // from the base's state at m, its lon/lat bookkeeping restated from the
  // base's points before m
  int m = 0;
  long long ob = 0;
  WalkFrom wf;
  if (pl.z == 1) {
    m = pl.y;
    ob = L.off[pl.x];
    if (m > cap) {
      atomicOr(err, cap < c.nlos_max ? kErrSlabOverflow : kErrLosOverflow);
      return;
    }
    const long long bp = R.bpts;
    for (int ip = 0; ip < m; ip++) {
      const long long q = ob + ip, s = base + ip;
      L.z[s] = L.z[q];
      L.f.p[s] = L.f.p[q];
      L.f.t[s] = L.f.t[q];
      L.f.ds[s] = L.f.ds[q];
      L.f.aux[s] = L.f.aux[q];
      if (c.ig_h2o >= 0) L.f.qh2o[s] = L.f.qh2o[q];
      for (int ig = 0; ig < c.ng; ig++) L.f.u[ig * L.cap + s] = L.f.u[ig * L.cap + q];
      for (int iw = 0; iw < c.nw; iw++) L.f.kw[iw * L.cap + s] = L.f.kw[iw * L.cap + q];
    }
    wf.n = m;
    for (int i = 0; i < 3; i++) {
      wf.x[i] = R.xs[i * bp + ob + m];
      wf.e[i] = R.es[i * bp + ob + m];
      wf.x_last[i] = R.xs[i * bp + ob + m - 1];
      gk.x_first[i] = R.xs[i * bp + ob];
    }
    wf.z = L.z[ob + m];
    wf.z_last = L.z[ob + m - 1];
    wf.lev_last = R.lev[ob + m - 1];
    wf.raw_last = R.dsr[ob + m - 1];
    // the first lowest point so far and its neighbours
    int imin = 0;
    double zmin = L.z[ob];
    for (int ip = 1; ip < m; ip++)
      if (L.z[ob + ip] < zmin) {
        zmin = L.z[ob + ip];
        imin = ip;
      }
    gk.imin = imin;
    gk.zmin_seen = zmin;
    gk.want_p1 = imin == m - 1;
    gk.ds_m = R.dsr[ob + imin];
    if (imin + 1 < m) gk.ds_p1 = R.dsr[ob + imin + 1];
    for (int i = 0; i < 3; i++) {
      gk.x_m1[i] = imin > 0 ? R.xs[i * bp + ob + imin - 1] : 0.0;
      gk.x_p1[i] = imin + 1 < m ? R.xs[i * bp + ob + imin + 1] : 0.0;
    }
  }
  const int n = walk_m<true>(c, a, b.geo, b.nray, r, L, base, cap, &sft, &gk,
                                   qcache + threadIdx.x, err, m > 0 ? &wf : nullptr);
  ray_finish_m(b, L, r, n, sft, gk);
}

// The fill pass of a batch takes two kernels.  A ray's walk is a chain of
// dependent steps, bound by latency, so k_walk_m does nothing but the chain and
// leaves z, p, T, the trapezoid lengths and the level interval of every point;
// k_points_m adds the mixing ratios, column densities and extinctions, which
// no step needs, for all points at once.
//
// k_walk_m: four lanes per ray, lanes 0-2 the components of the FP64 position
// and direction and the three refraction sub-points.  Conversions and compares
// run on the integer pipe (an FP64 instruction, these among them, holds a warp
// for 64 cycles; 7 are left per step).  Every value is formed as in walk_m, in
// the same order, so both give the same LOS.  All lanes stay in the loop until
// the warp's eight rays are done.
// Walks of one nadir ray of 901 points, 1500 of 801 and 20000 limb rays (CGA),
// both kernels: 1.49, 1.47 and 1.60 ms.  With the emitters in the same kernel,
// dealt over the four lanes, 1.87, 2.12 and 2.27; with one lane per ray 2.40,
// 2.70 and 2.28.  A step takes 3000 cycles of a warp at one ray; with many rays
// the loads of their level values add to it (a build of 96 registers, for more
// warps, was slower: 3.1 ms with the emitters inside against 2.3).
constexpr int kWalk4 = 4;

__device__ __forceinline__ float from4(float v, int k) {
  return __shfl_sync(0xffffffffu, v, k, kWalk4);
}
__device__ __forceinline__ double from4(double v, int k) {
  return __shfl_sync(0xffffffffu, v, k, kWalk4);
}

template <int ROLE>
__global__ void __launch_bounds__(kTraceThreads)
    k_walk_m(CtlDev c, BatchDev b, LosDev L, const int* order, int r0, int nr_l,
                    TraceResume R, unsigned* err) {
  __shared__ GeoKeep keep[kTraceThreads / kWalk4];
  const int s = threadIdx.x & (kWalk4 - 1);
  const int th = (int)(blockIdx.x * blockDim.x + threadIdx.x) / kWalk4;
  GeoKeep& gk = keep[threadIdx.x / kWalk4];
  int r = th < nr_l ? (order ? order[th] : r0 + th) : -1;
  const bool skipped = r >= 0 && b.obs_skip && b.obs_skip[b.ray_obs[r]];
  if (skipped) {
    if (s == 0) L.count[r] = 0;
    r = -1;
  }
  const AtmM a = atm_m(b, c, r >= 0 ? b.ray_obs[r] : 0);
  const long long base = r >= 0 ? L.off[r] : 0;
  const int cap = r >= 0 ? L.count[r] : 0;
  const int k = s < 3 ? s : 0;  // component of this lane
  const float h = 0.02f;
  const double zrefrac = 60;
  const float rayds = (float)c.rayds, raydz = (float)c.raydz;
  double zmin = 0, zmax = 0, x = 0, e = 0, z = 0, sft = -999;
  float xf[3] = {1.f, 0.f, 0.f}, ef[3] = {1.f, 0.f, 0.f};
  int n = 0, stop = 0;
  const int st = r >= 0 ? ray_bounds_m(c, a, b.geo, b.nray, r, &zmin, &zmax, err) : 0;
  bool alive = st > 0;
  if (st < 0) n = -1;
  if (alive) {
    double x0[3], e0[3];
    ray_first_m(b.geo, b.nray, r, zmax, x0, e0, &z);
    for (int i = 0; i < 3; i++) {
      xf[i] = (float)x0[i];
      ef[i] = (float)e0[i];
      if (i == k) {
        x = x0[i];
        e = e0[i];
      }
    }
  }
  if (s == 0) {  // each field has one writer; read after the walk
    gk.imin = 0;
    gk.ds_clip = 0;
    gk.ds_m = gk.ds_p1 = 0.f;
  }
  if (s < 3) gk.x_m1[s] = gk.x_p1[s] = gk.x_first[s] = gk.x_last[s] = 0;
  bool want_p1 = false;
  double zmin_seen = 0, last_z = 0, x_last = 0;
  Lev lv;
  lv.i = -1;
  // lanes 1-3 write p, T and the offset in the level interval of a point
  float* const dst = (s == 1 ? L.f.p : s == 2 ? L.f.t : L.f.aux) + base;
  float raw_before = 0.f, raw_pend = 0.f;
  while (__any_sync(0xffffffffu, alive)) {
    const float rf = d2f_bits(z + kRE), rinv = 1.f / rf;
    float xh[3];
    for (int i = 0; i < 3; i++) xh[i] = xf[i] * rinv;
    float step = rayds;
    if (raydz > 0) {
      const float cosa = fabsf(ef[0] * xh[0] + ef[1] * xh[1] + ef[2] * xh[2]);
      if (cosa != 0) step = rayds < raydz / cosa ? rayds : raydz / cosa;
    }
    const bool low = less(z, zmin), high = less(zmax, z);
    if (alive && (low || high) && n > 0) {  // clip (see walk_m)
      stop = low ? 2 : 1;
      const double frac = ((low ? zmin : zmax) - last_z) / (z - last_z);
      x = x_last + frac * (x - x_last);
      z = last_z + frac * (z - last_z);
      const double dsc = (double)step * frac;
      raw_pend = (float)dsc;
      if (s == 0) gk.ds_clip = dsc;
      if (ROLE == 1 && s == 3) R.dsr[base + n - 1] = raw_pend;
      step = 0.f;
    }
    if (alive && n >= cap) {
      if (s == 0) atomicOr(err, cap < c.nlos_max ? kErrSlabOverflow : kErrLosOverflow);
      alive = false;
      n = -1;
    }
    float dl = 0.f, p = 0.f, t = 1.f;
    if (alive) {
      dl = lev_find(a, z, lv);
      lev_pt(lv, dl, &p, &t);
      if (n > 0 && s == 0)
        L.f.ds[base + n - 1] = n == 1 ? 0.5f * raw_pend : 0.5f * (raw_before + raw_pend);
      const long long q = base + n;
      raw_before = raw_pend;
      raw_pend = step;
      if (s == 0) L.z[q] = z;
      else dst[n] = s == 1 ? p : s == 2 ? t : dl;
      if (s == 3) L.f.qh2o[q] = __int_as_float(lv.i);
      if (ROLE == 1) {
        if (s < 3) {
          R.xs[s * R.bpts + q] = x;
          R.es[s * R.bpts + q] = e;
        } else {
          R.lev[q] = lv.i;
          R.dsr[q] = step;
        }
      }
      if (n == 0 && s < 3) gk.x_first[s] = x;
      const bool newmin = n == 0 || less(z, zmin_seen);
      if (want_p1) {
        if (s < 3) gk.x_p1[s] = x;
        if (s == 0) gk.ds_p1 = step;
      }
      if (newmin) {
        zmin_seen = z;
        if (s < 3) gk.x_m1[s] = x_last;  // the previous point
        if (s == 0) {
          gk.imin = n;
          gk.ds_m = step;
        }
      }
      want_p1 = newmin;
      last_z = z;
      x_last = x;
      n++;
      if (stop) {
        sft = stop == 2 ? (c.nsf > 0 && a.sft > 0 ? a.sft : (double)t) : -999;
        if (s == 0)
          L.f.ds[base + n - 1] = n == 1 ? 0.5f * raw_pend : 0.5f * (raw_before + raw_pend);
        if (s < 3) gk.x_last[s] = x;
        alive = false;
      }
    }
    // refraction (see walk_m), a sub-point per lane
    const bool bend = alive && c.refrac && is_number(z) && !lt(zrefrac, z);
    const float nref = 1.f + kRefracC * p / t;
    float inc_k = 0.f;
    if (bend) {
      const float d[3] = {0.5f * step * ef[0], 0.5f * step * ef[1], 0.5f * step * ef[2]};
      const float dzh = dz_of(xh, rf, d);
      const float rh = rf + dzh, rhinv = 1.f / rh;
      const float xhh[3] = {(xh[0] * rf + d[0]) * rhinv, (xh[1] * rf + d[1]) * rhinv,
                            (xh[2] * rf + d[2]) * rhinv};
      Lev lh = lv;
      float dlh = dl + dzh;
      if (!lev_holds(lh, dlh)) dlh = lev_find(a, z + f2d_bits(dzh), lh);
      float ph, thp;
      lev_pt(lh, dlh, &ph, &thp);
      const float dk[3] = {k == 0 ? h : 0.f, k == 1 ? h : 0.f, k == 2 ? h : 0.f};
      const float dlk = dz_of(xhh, rh, dk);
      float dN;
      if (lev_holds(lh, dlh + dlk)) {
        dN = dN_in(lh, ph, thp, dlk);
      } else {
        // split at the level boundary between the midpoint and zk
        const double zh = lh.z0 + f2d_bits(dlh), zk = zh + f2d_bits(dlk);
        Lev lk = lh;
        const float dlk0 = lev_find(a, zk, lk);
        if (lk.i == lh.i) {
          dN = dN_in(lh, ph, thp, dlk);
        } else {
          const bool up = lk.i > lh.i;
          const double zb = up ? a.z[lh.i + 1] : a.z[lh.i];
          const float d1 = d2f_bits(zb - zh);
          const float dn1 = dN_in(lh, ph, thp, d1);
          float pb, tb;
          const float dlb = d2f_bits(zb - lk.z0);
          lev_pt(lk, dlb, &pb, &tb);
          dN = dn1 + dN_in(lk, pb, tb, dlk0 - dlb);
        }
      }
      inc_k = step * (dN / h) / nref;
    }
    float inc[3];
    for (int i = 0; i < 3; i++) inc[i] = from4(inc_k, i);
    double e1 = e;
    if (bend) e1 = e + f2d_bits(inc_k);
    const float delta = 2.f * (ef[0] * inc[0] + ef[1] * inc[1] + ef[2] * inc[2]) +
                        (inc[0] * inc[0] + inc[1] * inc[1] + inc[2] * inc[2]);
    const bool large = bend && !(fabsf(delta) < 1e-3f);
    if (bend && !large) {
      const float corr = delta * (-0.5f + delta * (0.375f - 0.3125f * delta));
      e1 += e1 * f2d_bits(corr);
    }
    if (__any_sync(0xffffffffu, large)) {
      const double e0 = from4(e1, 0), e1c = from4(e1, 1), e2 = from4(e1, 2);
      if (large) e1 /= sqrt(e0 * e0 + e1c * e1c + e2 * e2);
    }
    const float en = d2f_bits(e1);
    float D[3], efn[3];
    for (int i = 0; i < 3; i++) {
      efn[i] = from4(en, i);
      D[i] = 0.5f * step * (ef[i] + efn[i]);
    }
    const float dzs = dz_of(xh, rf, D);
    const float Dk = k == 0 ? D[0] : k == 1 ? D[1] : D[2];
    if (alive) {
      x += f2d_bits(Dk);
      e = e1;
      z += f2d_bits(dzs);
    }
    const float xn = d2f_bits(x);
    for (int i = 0; i < 3; i++) {
      xf[i] = from4(xn, i);
      ef[i] = efn[i];
    }
  }
  __syncwarp();
  if (r >= 0 && s == 0) ray_finish_m(b, L, r, n, sft, gk);
}

// k_points_m: a block per ray, a thread per point, over the points that
// k_walk_m left (the level interval in qh2o, the offset in it in aux).  The
// Curtis-Godson sums run along the ray: a thread per emitter walks the block's
// points in shared memory, kSumGas emitters at a time.
constexpr int kPointThreads = 128, kSumGas = 8;

template <bool CGA>
__global__ void __launch_bounds__(kPointThreads) k_points_m(CtlDev c, BatchDev b, LosDev L, int r0) {
  __shared__ float su[CGA ? kSumGas : 1][kPointThreads], sp[CGA ? kSumGas : 1][kPointThreads],
      st[CGA ? kSumGas : 1][kPointThreads], pt[2][CGA ? kPointThreads : 1];
  const int r = r0 + (int)blockIdx.x, tid = threadIdx.x;
  const int n = L.count[r];
  if (n <= 0) return;
  const long long base = L.off[r];
  const AtmM a = atm_m(b, c, b.ray_obs[r]);
  const bool cloud = c.ncl > 0 && a.cldz > 0;
  float u_c, p_c, t_c, u_s, p_s, t_s;
  const int groups = CGA ? (c.ng + kSumGas - 1) / kSumGas : 1;
  // the groups after the first find the level interval already overwritten, so
  // the last group writes the point's own values
  for (int gr = 0; gr < max(groups, 1); gr++) {
    const int g0 = gr * kSumGas, g1 = CGA ? min(g0 + kSumGas, c.ng) : c.ng;
    const bool last = gr >= groups - 1;
    u_c = p_c = t_c = u_s = p_s = t_s = 0.f;
    for (int ip0 = 0; ip0 < n; ip0 += kPointThreads) {
      const int ip = ip0 + tid;
      const long long q = base + ip;
      if (ip < n) {
        const int i = __float_as_int(L.f.qh2o[q]);
        const float dl = L.f.aux[q], p = L.f.p[q], t = L.f.t[q], ds = L.f.ds[q];
        const float dz = d2f_bits(a.z[i + 1] - a.z[i]);
        auto at = [&](const double* src) {
          const float v0 = d2f_bits(src[i]), v1 = d2f_bits(src[i + 1]);
          return qk_at(v0, (v1 - v0) / dz, dl);
        };
        if (CGA) {
          pt[0][tid] = p;
          pt[1][tid] = t;
        }
        for (int g = g0; g < g1; g++) {
          const float u = col_density(at(a.q + g * a.stride), p, t, ds);
          L.f.u[g * L.cap + q] = u;
          if (CGA) su[g - g0][tid] = u;
        }
        if (last) {
          for (int iw = 0; iw < c.nw; iw++) L.f.kw[iw * L.cap + q] = at(a.k + iw * a.stride);
          if (c.ig_h2o >= 0) L.f.qh2o[q] = at(a.q + c.ig_h2o * a.stride);
          float aux = 0.f;
          if (cloud) {
            const float v = (float)((L.z[q] - a.clz) / a.cldz);
            aux = expf(-0.5f * v * v);
          }
          L.f.aux[q] = aux;
        }
      }
      if (CGA) {
        __syncthreads();
        if (tid < g1 - g0) {  // compensated running sums
          const int m = min(n - ip0, kPointThreads);
          for (int k = 0; k < m; k++) {
            const float uu = su[tid][k];
            float y = uu - u_c, s2 = u_s + y;
            u_c = (s2 - u_s) - y;
            u_s = s2;
            y = uu * pt[0][k] - p_c;
            s2 = p_s + y;
            p_c = (s2 - p_s) - y;
            p_s = s2;
            y = uu * pt[1][k] - t_c;
            s2 = t_s + y;
            t_c = (s2 - t_s) - y;
            t_s = s2;
            su[tid][k] = u_s;
            sp[tid][k] = p_s;
            st[tid][k] = t_s;
          }
        }
        __syncthreads();
        if (ip < n)
          for (int g = g0; g < g1; g++) {
            const float uu = su[g - g0][tid];
            L.f.cgu[g * L.cap + q] = uu;
            L.f.cgp[g * L.cap + q] = sp[g - g0][tid] / uu;
            L.f.cgt[g * L.cap + q] = st[g - g0][tid] / uu;
          }
        __syncthreads();
      }
    }
  }
}

}  // namespace

void launch_trace_count_mixed(const CtlDev& c, const BatchDev& b, const LosDev& L, unsigned* err,
                              cudaStream_t s) {
  const int bs = kTraceThreads;
  k_trace_count_m<<<(b.nray + bs - 1) / bs, bs, 0, s>>>(c, b, L, err);
}

void launch_los_bound_mixed(const CtlDev& c, const BatchDev& b, double scale, int* cap,
                            cudaStream_t s) {
  const int bs = 128;
  k_los_bound_m<<<(b.nray + bs - 1) / bs, bs, 0, s>>>(c, b, scale, cap);
}

namespace {
template <int ROLE>
void launch_walk(const CtlDev& c, const BatchDev& b, const LosDev& L, const int* order, int r0, int nr,
                 const TraceResume& R, unsigned* err, cudaStream_t s) {
  if (nr <= 0) return;
  const int rays = kTraceThreads / kWalk4;
  k_walk_m<ROLE><<<(nr + rays - 1) / rays, kTraceThreads, 0, s>>>(c, b, L, order, r0, nr, R, err);
  if (L.cga) k_points_m<true><<<nr, kPointThreads, 0, s>>>(c, b, L, r0);
  else k_points_m<false><<<nr, kPointThreads, 0, s>>>(c, b, L, r0);
}
}  // namespace

// order: a permutation of the batch's rays
void launch_trace_fill_mixed(const CtlDev& c, const BatchDev& b, const LosDev& L, const int* order,
                             unsigned* err, cudaStream_t s) {
  launch_walk<0>(c, b, L, order, 0, b.nray, TraceResume{}, err, s);
}

int trace_fill_resident(int sms) {
  // blocks per SM are set by the registers (the shared memory of a few
  // emitters does not bind); computed once, thread-safely
  static const int per_sm = [] {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_trace_fill_m, kTraceThreads, 0) !=
            cudaSuccess ||
        nb < 1)
      nb = 1;
    return nb * kTraceThreads;
  }();
  return per_sm * sms;
}

void launch_trace_fill_resumed(const CtlDev& c, const BatchDev& b, const LosDev& L,
                               const int* order, int r0, int nr, const TraceResume& R, int role,
                               unsigned* err, cudaStream_t s) {
  const int bs = kTraceThreads;
  if (nr <= 0) return;
  if (role == 1)
    launch_walk<1>(c, b, L, order, r0, nr, R, err, s);
  else
    k_trace_fill_m<<<(nr + bs - 1) / bs, bs, sizeof(float) * trace_smem_floats(c) * kTraceThreads,
                     s>>>(c, b, L, order, r0, nr, R, err);
}

}  // namespace jgb
