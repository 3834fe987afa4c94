// FP64 kernels: ray tracing and the plain FP64 forward model.
//
// This translation unit is compiled with -fmad=false so that every FP64
// expression is rounded like the reference's (no fused multiply-add), which
// keeps the FP64 path within rounding of the reference results.
//
//   k_trace_fill; k_walk8, k_points64
//                 raytrace (jurassic.c:4201-4438) + tangent_point
//                 (jurassic.c:5223-5263), one or eight lanes per ray, in one
//                 pass into per-ray capacities; k_trace_count counts the
//                 points where a capacity was too small.
//   k_path_fp64   formod_pencil (jurassic.c:3196-3338) with intpol_tbl_ega /
//                 intpol_tbl_cga (3710-3891), formod_continua (3075-3117),
//                 formod_srcfunc (3483-3496), surface/reflection/solar terms,
//                 BT conversion and the observation mask of formod
//                 (3026-3071); one thread per (ray, channel), without any
//                 workspace (the allocation-free entry point; the others
//                 take jgb_path64.cu).
//   k_srcfunc     init_srcfunc (jurassic.c:3631-3681) on the device.
//   k_hydro_means, k_hydro_chain  hydrostatic (jurassic.c:3520-3582), a lane per
//                 layer, then a thread per profile.
#include "../../include/jurassic_gb300.h"
#include "jgb_common.cuh"
#include "jgb_internal.h"

namespace jgb {

// ---------------------------------------------------------------------------
// atmosphere access

struct AtmView {
  int np, ng, nw;
  bool asc;           // altitude grid strictly ascending
  long long stride;   // level stride of q/k planes (total levels of the batch)
  const double *z, *p, *t, *q, *k;   // q[ig*stride + i], k[iw*stride + i]
  // slopes of the interpolations on interval i (k_level_slopes; nullptr:
  // formed when a ray enters the interval), in the strides of p, t, q, k
  const double *sp, *st, *sq, *sk;
  double clz, cldz, sfz, sfp, sft;
};

__device__ inline AtmView atm_view(const CtlDev& c, const BatchDev& b, const double* slopes,
                                   int o) {
  AtmView a;
  const int l0 = b.lev_off[o];
  a.np = b.lev_off[o + 1] - l0;
  a.ng = c.ng;
  a.nw = c.nw;
  a.stride = b.nlev;
  a.z = b.z + l0;
  a.p = b.p + l0;
  a.t = b.t + l0;
  a.q = b.q + l0;
  a.k = b.k + l0;
  a.sp = slopes ? slopes + l0 : nullptr;
  a.st = a.sp + a.stride;
  a.sq = a.st + a.stride;
  a.sk = a.sq + a.stride * c.ng;
  const double* s = b.scal + (long long)o * b.nscal;
  a.clz = s[0];
  a.cldz = s[1];
  a.sfz = s[2 + c.ncl];
  a.sfp = s[3 + c.ncl];
  a.sft = s[4 + c.ncl];
  a.asc = true;
  for (int i = 0; i + 1 < a.np; i++)
    if (!(a.z[i] < a.z[i + 1])) a.asc = false;
  return a;
}

// Slope of LOGY on an interval, log(y1 / y0) / (x1 - x0), NaN where LOGY falls
// back to LIN.
__device__ inline double log_slope(double x0, double y0, double x1, double y1) {
  const double q = y1 / y0;
  return q > 0 ? log(q) / (x1 - x0) : __longlong_as_double(0x7ff8000000000000LL);
}

// The slopes of every level interval, one warp per observation: sp, st, sq[],
// sk[] planes of nlev.
__global__ void k_level_slopes(CtlDev c, BatchDev b, double* out) {
  const int o = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  if (o >= b.nobs || (b.obs_skip && b.obs_skip[o])) return;
  const int l1 = b.lev_off[o + 1];
  const long long nl = b.nlev;
  for (int l = b.lev_off[o] + (threadIdx.x & 31); l + 1 < l1; l += 32) {
    const double dz = b.z[l + 1] - b.z[l];
    out[l] = log_slope(b.z[l], b.p[l], b.z[l + 1], b.p[l + 1]);
    out[nl + l] = (b.t[l + 1] - b.t[l]) / dz;
    for (int k = 0; k < c.ng; k++)
      out[(2 + k) * nl + l] = (b.q[k * nl + l + 1] - b.q[k * nl + l]) / dz;
    for (int k = 0; k < c.nw; k++)
      out[(2 + c.ng + k) * nl + l] = (b.k[k * nl + l + 1] - b.k[k * nl + l]) / dz;
  }
}

// One level interval with its slopes.
struct Lev64 {
  int i;
  double z0, z1, p0, sp, t0, st;
};

__device__ inline void lev64_load(const AtmView& a, int i, Lev64& v) {
  v.i = i;
  v.z0 = a.z[i];
  v.z1 = a.z[i + 1];
  v.p0 = a.p[i];
  v.t0 = a.t[i];
  if (a.sp) {
    v.sp = a.sp[i];
    v.st = a.st[i];
  } else {
    v.sp = log_slope(v.z0, v.p0, v.z1, a.p[i + 1]);
    v.st = (a.t[i + 1] - v.t0) / (v.z1 - v.z0);
  }
}

// On a strictly ascending grid the bisection of locate_irr returns the unique
// i with z[i] <= x < z[i+1] (0 below, n-2 above the grid), so an interval
// that holds z is the bisection's result: the current one is tried first,
// then its neighbour towards z.
__device__ inline bool lev64_holds(const AtmView& a, const Lev64& v, double z) {
  return (v.i == 0 || !lt(z, v.z0)) && (v.i == a.np - 2 || lt(z, v.z1));
}

__device__ inline void lev64_find(const AtmView& a, double z, Lev64& v) {
  if (a.asc && v.i >= 0) {
    if (lev64_holds(a, v, z)) return;
    const int j = lt(z, v.z0) ? v.i - 1 : v.i + 1;
    if (j >= 0 && j <= a.np - 2) {
      lev64_load(a, j, v);
      if (lev64_holds(a, v, z)) return;
    }
  }
  lev64_load(a, bracket_irr(a.z, a.np, z), v);
}

// LOGY where its ratio is not positive: LIN
__device__ __noinline__ double p_linear(const AtmView& a, int i, double z) {
  return lin(a.z[i], a.p[i], a.z[i + 1], a.p[i + 1], z);
}

// intpol_atm (jurassic.c:3685-3706): p (log-linear) and T only.
__device__ __forceinline__ void lev64_pt(const AtmView& a, const Lev64& v, double z, double* p,
                                         double* t) {
  const double dz = z - v.z0;
  *p = v.sp == v.sp ? v.p0 * exp(v.sp * dz) : p_linear(a, v.i, z);
  *t = v.t0 + v.st * dz;
}

constexpr double kRefrac = 7.753e-05;  // N = kRefrac p / T

// Rounded quotient of a by w from the reciprocal r of w: quotient, exact
// remainder, one correction (Markstein, IBM J. Res. Dev. 34, 1990).
__device__ __forceinline__ double div_by(double a, double w, double r) {
  const double q = a * r;
  return fma(fma(-q, w, a), r, q);
}

__device__ __forceinline__ double norm2(const double* x) {
  return x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
}

__device__ __forceinline__ void div3(double* x, double w) {
  const double r = 1 / w;
  for (int k = 0; k < 3; k++) x[k] = div_by(x[k], w, r);
}

// What the walk keeps for the tangent point and the ends.
struct Keep64 {
  double x0[3], xm[3], xp[3], xl[3];     // first, around the lowest point, last
  double z0, zl, zm1, zmin, zp1;         // their altitudes (zm1: before the lowest)
  double ds_m, ds_p1, ds_clip;           // raw lengths at the lowest point and the next
  int imin;
  bool want_p1;
};

constexpr int kTrace64Threads = 32;

// Doubles of shared memory per thread of the fill pass: mixing ratios of the
// point waiting for its segment length, and in CGA the running sums.
__host__ __device__ inline int trace64_smem(const CtlDev& c) {
  return c.ng + (c.formod == 0 ? 3 * c.ng : 0);
}

// Position and direction at the ray's first point, and the altitudes that end
// it: 1, or 0 for a ray above the atmosphere, -1 on error.
__device__ int ray_start(const CtlDev& c, const AtmView& a, const double* g, long long nray, int r,
                         double* x, double* ex0, double* zlo, double* zhi, unsigned* err) {
  double xobs[3], xvp[3], z;
  const double obsz = g[1 * nray + r], obslon = g[2 * nray + r], obslat = g[3 * nray + r];
  const double vpz = g[4 * nray + r], vplon = g[5 * nray + r], vplat = g[6 * nray + r];
  double zmin = a.z[0], zmax = a.z[0];
  for (int i = 0; i < a.np; i++) {
    zmin = a.z[i] < zmin ? a.z[i] : zmin;
    zmax = a.z[i] > zmax ? a.z[i] : zmax;
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
  if (vpz > zmax) return 0;
  *zlo = zmin;
  *zhi = zmax;

  to_cart(obsz, obslon, obslat, xobs);
  to_cart(vpz, vplon, vplat, xvp);
  for (int i = 0; i < 3; i++) ex0[i] = xvp[i] - xobs[i];
  double norm = sqrt(norm2(ex0));
  for (int i = 0; i < 3; i++) ex0[i] /= norm;
  for (int i = 0; i < 3; i++) x[i] = xobs[i];

  if (obsz > zmax) {
    double dmax = norm, dmin = 0;
    for (int guard = 0; fabs(dmin - dmax) > 0.001 && guard < 200; guard++) {
      const double d = (dmax + dmin) / 2;
      for (int i = 0; i < 3; i++) x[i] = xobs[i] + d * ex0[i];
      z = sqrt(norm2(x)) - kRE;
      if (z <= zmax && z > zmax - 0.001) break;
      if (z < zmax - 0.0005) dmax = d; else dmin = d;
    }
  }
  return 1;
}

// One ray walk (raytrace, jurassic.c:4201-4438).  STORE=false only counts
// points; STORE=true writes the LOS planes, every point with its final
// trapezoid length, column densities and Curtis-Godson means once the next
// point is placed (the clip changes the last raw length).  Positions,
// directions and altitudes round as in the reference, which matters because
// an altitude |x| - RE carries 1e-12 km of rounding that finite differences
// of two walks must share.  Returns the number of points, or -1 on error.
template <bool STORE>
__device__ int walk(const CtlDev& c, const AtmView& a, const double* g, long long nray, int r,
                    const LosDev& L, long long base, int cap, double* sft_out, Keep64* kp,
                    double* sm, unsigned* err) {
  const double h = 0.02, zrefrac = 60;
  double ex0[3], ex1[3], x[3], xh[3];
  double z, p, t;
  int stop = 0, n = 0;
  double last_z = 0, last_x[3] = {0, 0, 0};
  *sft_out = -999;

  double zmin, zmax;
  const int st = ray_start(c, a, g, nray, r, x, ex0, &zmin, &zmax, err);
  if (st <= 0) return st;

  Lev64 lv;
  lv.i = -1;
  // raw lengths of the point before the pending one and of that one, and its
  // p, T and 1 / (kB T)
  double raw_before = 0, raw_pend = 0, pend_p = 0, pend_t = 0, pend_r = 0;
  constexpr int S = kTrace64Threads;
  double* const pq = sm;
  double* const cg = STORE ? sm + c.ng * S : nullptr;
  auto finalize = [&](int k) {
    const long long s = base + k;
    const double dsT = k == 0 ? raw_pend * 0.5 : 0.5 * (raw_before + raw_pend);
    L.ds[s] = dsT;
    const double kt = kKB * pend_t;
    for (int ig = 0; ig < a.ng; ig++) {
      const double u = div_by(10 * pq[ig * S] * pend_p, kt, pend_r) * dsT;
      L.u[ig * L.cap + s] = u;
      if (L.cga) {
        double* q = cg + 3 * ig * S;
        const double su = k ? q[0] + u : u;
        const double sp = k ? q[S] + u * pend_p : u * pend_p;
        const double st = k ? q[2 * S] + u * pend_t : u * pend_t;
        q[0] = su;
        q[S] = sp;
        q[2 * S] = st;
        const double ru = 1 / su;
        L.cgu[ig * L.cap + s] = su;
        L.cgp[ig * L.cap + s] = div_by(sp, su, ru);
        L.cgt[ig * L.cap + s] = div_by(st, su, ru);
      }
    }
  };

  for (;;) {
    double ds = c.rayds;
    const double norm = sqrt(norm2(x));
    if (c.raydz > 0) {
      const double rn = 1 / norm;
      for (int i = 0; i < 3; i++) xh[i] = div_by(x[i], norm, rn);
      const double cosa = fabs(ex0[0] * xh[0] + ex0[1] * xh[1] + ex0[2] * xh[2]);
      if (__double_as_longlong(cosa) != 0) {
        const double v = c.raydz / cosa;
        ds = lt(c.rayds, v) ? c.rayds : v;
      }
    }
    z = norm - kRE;
    // a position that is not a number is inside: the walk ends with an overflow
    const bool num = is_number(z);
    const bool low = num && lt(z, zmin), high = num && lt(zmax, z);
    if ((low || high) && n > 0) {
      if (!STORE) {  // the clipped last point ends the count
        if (n >= cap) {
          atomicOr(err, cap < c.nlos_max ? kErrSlabOverflow : kErrLosOverflow);
          return -1;
        }
        return n + 1;
      }
      stop = low ? 2 : 1;
      const double frac = ((low ? zmin : zmax) - last_z) / (z - last_z);
      double lz, llon, llat;
      to_geo(last_x, &lz, &llon, &llat);  // the reference keeps the last point in geographic form
      to_cart(lz, llon, llat, xh);
      for (int i = 0; i < 3; i++) x[i] = xh[i] + frac * (x[i] - xh[i]);
      z = sqrt(norm2(x)) - kRE;
      raw_pend = ds * frac;
      if (STORE) kp->ds_clip = raw_pend;
      ds = 0;
    }
    if (n >= cap) {
      atomicOr(err, cap < c.nlos_max ? kErrSlabOverflow : kErrLosOverflow);
      return -1;
    }
    lev64_find(a, z, lv);
    lev64_pt(a, lv, z, &p, &t);
    if (STORE) {
      if (n > 0) finalize(n - 1);
      const long long s = base + n;
      const int i = lv.i;
      const double dz = z - lv.z0;
      L.p[s] = p;
      L.t[s] = t;
      raw_before = raw_pend;
      raw_pend = ds;
      pend_p = p;
      pend_t = t;
      pend_r = 1 / (kKB * t);
      for (int ig = 0; ig < a.ng; ig++) {
        const double q0 = a.q[ig * a.stride + i];
        const double sq = a.sp ? a.sq[ig * a.stride + i]
                               : (a.q[ig * a.stride + i + 1] - q0) / (lv.z1 - lv.z0);
        const double v = q0 + sq * dz;
        pq[ig * S] = v;
        if (ig == c.ig_h2o) L.qh2o[s] = v;
      }
      for (int iw = 0; iw < a.nw; iw++) {
        const double k0 = a.k[iw * a.stride + i];
        const double sk = a.sp ? a.sk[iw * a.stride + i]
                               : (a.k[iw * a.stride + i + 1] - k0) / (lv.z1 - lv.z0);
        L.kw[iw * L.cap + s] = k0 + sk * dz;
      }
      L.aux[s] = (c.ncl > 0 && a.cldz > 0) ? exp(-0.5 * ((z - a.clz) / a.cldz) * ((z - a.clz) / a.cldz)) : 0.0;
      if (n == 0) {
        kp->z0 = z;
        for (int k = 0; k < 3; k++) kp->x0[k] = x[k];
      }
      if (kp->want_p1) {
        kp->want_p1 = false;
        kp->zp1 = z;
        kp->ds_p1 = ds;
        for (int k = 0; k < 3; k++) kp->xp[k] = x[k];
      }
      if (n == 0 || lt(z, kp->zmin)) {
        kp->zmin = z;
        kp->imin = n;
        kp->ds_m = ds;
        kp->zm1 = last_z;
        for (int k = 0; k < 3; k++) kp->xm[k] = last_x[k];
        kp->want_p1 = true;
      }
    }
    last_z = z;
    for (int k = 0; k < 3; k++) last_x[k] = x[k];
    n++;
    if (stop) {
      if (c.nsf > 0 && a.sft > 0) t = a.sft;
      *sft_out = (stop == 2 ? t : -999);
      if (STORE) {
        finalize(n - 1);
        kp->zl = z;
        for (int k = 0; k < 3; k++) kp->xl[k] = x[k];
      }
      break;
    }
    const double hds = 0.5 * ds;
    if (c.refrac && !lt(zrefrac, z)) {
      const double nref = 1 + kRefrac * p / t;
      for (int k = 0; k < 3; k++) xh[k] = x[k] + hds * ex0[k];
      const double zm = sqrt(norm2(xh)) - kRE;
      Lev64 lm = lv;
      lev64_find(a, zm, lm);
      lev64_pt(a, lm, zm, &p, &t);
      const double nm = kRefrac * p / t;
      for (int k = 0; k < 3; k++) {
        xh[k] += h;
        const double zk = sqrt(norm2(xh)) - kRE;
        lev64_find(a, zk, lm);
        lev64_pt(a, lm, zk, &p, &t);
        ex1[k] = ex0[k] * nref + ds * ((kRefrac * p / t - nm) / h);
        xh[k] -= h;
      }
    } else {
      for (int k = 0; k < 3; k++) ex1[k] = ex0[k];
    }
    div3(ex1, sqrt(norm2(ex1)));
    for (int k = 0; k < 3; k++) {
      x[k] += hds * (ex0[k] + ex1[k]);
      ex0[k] = ex1[k];
    }
  }
  return n;
}

// What a ray leaves beside its points: count, surface temperature, tangent
// point (tangent_point, jurassic.c:5223-5263, from the raw lengths) and ends.
__device__ void ray_finish(const BatchDev& b, const LosDev& L, int r, int n, double sft,
                           const Keep64& kp) {
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
  double dummy, lon0, lat0, lonl, latl;
  to_geo(kp.x0, &dummy, &lon0, &lat0);
  to_geo(kp.xl, &dummy, &lonl, &latl);
  // tangent point (tangent_point, jurassic.c:5223-5263) from the raw lengths
  const int imin = kp.imin;
  if (imin <= 0 || imin >= n - 1) {
    tp[0 * nr + r] = kp.zl;
    tp[1 * nr + r] = lonl;
    tp[2 * nr + r] = latl;
  } else {
    const double y0 = kp.zm1, y1 = kp.zmin, y2 = kp.zp1;
    const double d1 = imin == n - 2 ? kp.ds_clip : kp.ds_m;
    const double d2 = imin + 1 == n - 2 ? kp.ds_clip : kp.ds_p1;
    const double x1 = sqrt(d1 * d1 - (y1 - y0) * (y1 - y0));
    const double x2 = x1 + sqrt(d2 * d2 - (y2 - y1) * (y2 - y1));
    const double aa = 1 / (x1 - x2) * (-(y0 - y1) / x1 + (y0 - y2) / x2);
    const double bb = -(y0 - y1) / x1 - aa * x1;
    const double cc = y0;
    const double xt = -bb / (2 * aa);
    tp[0 * nr + r] = aa * xt * xt + bb * xt + cc;
    double v0[3], v2[3], v[3], lon, lat, tlon, tlat;
    to_geo(kp.xm, &dummy, &lon, &lat);
    to_cart(y0, lon, lat, v0);
    to_geo(kp.xp, &dummy, &lon, &lat);
    to_cart(y2, lon, lat, v2);
    for (int i = 0; i < 3; i++) v[i] = lin(0.0, v0[i], x2, v2[i], xt);
    to_geo(v, &dummy, &tlon, &tlat);
    tp[1 * nr + r] = tlon;
    tp[2 * nr + r] = tlat;
  }
  double* e = L.ends + 6LL * r;
  e[0] = kp.z0;
  e[1] = lon0;
  e[2] = lat0;
  e[3] = kp.zl;
  e[4] = lonl;
  e[5] = latl;
}

__global__ void k_trace_count(CtlDev c, BatchDev b, LosDev L, const double* slopes,
                              unsigned* err) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= b.nray) return;
  if (b.obs_skip && b.obs_skip[b.ray_obs[r]]) {
    L.count[r] = 0;
    return;
  }
  const AtmView a = atm_view(c, b, slopes, b.ray_obs[r]);
  double sft;
  const int n = walk<false>(c, a, b.geo, b.nray, r, L, 0, c.nlos_max, &sft, nullptr, nullptr, err);
  L.count[r] = n < 0 ? 0 : n;
}

// order (optional): thread t traces ray order[t], so that a warp's rays have
// similar capacities and finish together.
__global__ void __launch_bounds__(kTrace64Threads)
    k_trace_fill(CtlDev c, BatchDev b, LosDev L, const int* order, const double* slopes,
                 unsigned* err) {
  extern __shared__ double sm_trace[];
  const int th = blockIdx.x * blockDim.x + threadIdx.x;
  if (th >= b.nray) return;
  const int r = order ? order[th] : th;
  if (b.obs_skip && b.obs_skip[b.ray_obs[r]]) return;
  const AtmView a = atm_view(c, b, slopes, b.ray_obs[r]);
  const long long base = L.off[r];
  const int cap = L.count[r];
  double sft;
  Keep64 kp{};
  const int n = walk<true>(c, a, b.geo, b.nray, r, L, base, cap, &sft, &kp, sm_trace + threadIdx.x,
                           err);
  ray_finish(b, L, r, n, sft, kp);
}

// A batch of few rays leaves the FP64 pipes idle while each ray waits for its
// own chain (an instruction takes 64 cycles whether 1 or 32 lanes are active,
// and three warps share an SM without slowing each other), so eight lanes walk
// one ray (k_walk8): lanes 0-2 the components of the vectors and the refraction
// sub-points, lane 3 the midpoint, the others the LOS point, whose five altitude
// and atmosphere evaluations then run as one.  The lanes exchange squares and
// products, formed once per component.  What no step needs (mixing ratios,
// column densities, extinctions, Curtis-Godson sums) follows in k_points64.
// Every value is formed as in walk(), in the same order, so both give the same
// LOS.  Measured (trace stage, from the walk with one lane per ray in two
// passes, slopes, compares and lon/lat at every point: 1247 FP64 instructions
// per step; with the emitters dealt over the lanes and vectors in every lane:
// 130; here about 100):
// 10 limb rays 67.8, 9.7 and 7.3 ms; 273 limb rays 21.2, 2.9 and 2.2; 1000 nadir
// rays 49.1, 6.6 and 5.1.
// All lanes stay in the loop until the warp's four rays are done.
constexpr int kWalk8Rays = 4;  // rays of a warp

__device__ __forceinline__ double from_lane(double v, int k) {
  return __shfl_sync(0xffffffffu, v, k, 8);
}
// the sum over the components of a value that lanes 0-2 hold, as x + y + z
__device__ __forceinline__ double sum3(double v) {
  const double x = from_lane(v, 0), y = from_lane(v, 1), z = from_lane(v, 2);
  return x + y + z;
}

__global__ void __launch_bounds__(32)
    k_walk8(CtlDev c, BatchDev b, LosDev L, const int* order, const double* slopes,
            unsigned* err) {
  __shared__ Keep64 keep[kWalk8Rays];
  const int s = threadIdx.x & 7, th = (int)blockIdx.x * kWalk8Rays + (threadIdx.x >> 3);
  Keep64& kp = keep[threadIdx.x >> 3];
  int r = th < b.nray ? (order ? order[th] : th) : -1;
  if (r >= 0 && b.obs_skip && b.obs_skip[b.ray_obs[r]]) r = -1;
  const AtmView a = atm_view(c, b, slopes, r >= 0 ? b.ray_obs[r] : 0);
  const long long base = r >= 0 ? L.off[r] : 0;
  const int cap = r >= 0 ? L.count[r] : 0;
  const int k = s < 3 ? s : 0;  // component of this lane
  double x = k == 0 ? kRE : 0, e = k == 0 ? 1 : 0, zmin = 0, zmax = 0;
  int st = 0;
  if (r >= 0) {
    double x0[3] = {kRE, 0, 0}, e0[3] = {1, 0, 0};
    st = ray_start(c, a, b.geo, b.nray, r, x0, e0, &zmin, &zmax, err);
    for (int i = 0; i < 3; i++)
      if (i == k) {
        x = x0[i];
        e = e0[i];
      }
  }
  bool alive = st > 0;
  const double h = 0.02, rh = 1 / h, zrefrac = 60;
  const bool sub = s < 3, main_pt = s >= 4;
  double last_z = 0, last_x = 0, sft = -999, zmin_seen = 0;
  double raw_before = 0, raw_pend = 0;
  int n = 0, stop = 0;
  bool want_p1 = false;
  Lev64 lv;
  lv.i = -1;
  __syncwarp();
  while (__any_sync(0xffffffffu, alive)) {
    double ds = c.rayds;
    const double norm = sqrt(sum3(x * x));
    if (c.raydz > 0) {
      const double cosa = fabs(sum3(e * (x / norm)));
      if (__double_as_longlong(cosa) != 0) {
        const double v = c.raydz / cosa;
        ds = lt(c.rayds, v) ? c.rayds : v;
      }
    }
    double z = norm - kRE;
    // a position that is not a number is inside: the walk ends with an overflow
    const bool num = is_number(z);
    const bool low = num && lt(z, zmin), high = num && lt(zmax, z);
    const bool clip = alive && (low || high) && n > 0;
    if (__any_sync(0xffffffffu, clip)) {
      double xs[3], xl[3];
      for (int i = 0; i < 3; i++) {
        xs[i] = from_lane(x, i);
        xl[i] = from_lane(last_x, i);
      }
      if (clip) {
        stop = low ? 2 : 1;
        const double frac = ((low ? zmin : zmax) - last_z) / (z - last_z);
        double lz, llon, llat, xc[3];
        to_geo(xl, &lz, &llon, &llat);
        to_cart(lz, llon, llat, xc);
        for (int i = 0; i < 3; i++) {
          xs[i] = xc[i] + frac * (xs[i] - xc[i]);
          if (i == k) x = xs[i];
        }
        z = sqrt(norm2(xs)) - kRE;
        raw_pend = ds * frac;
        if (s == 0) kp.ds_clip = raw_pend;
        ds = 0;
      }
    }
    if (alive && n >= cap) {
      if (s == 0) atomicOr(err, cap < c.nlos_max ? kErrSlabOverflow : kErrLosOverflow);
      alive = false;
      n = -1;
    }
    // this lane's evaluation point: midpoint m, sub-point (the reference adds h
    // to a component and takes it off again before the next) or LOS point
    const double hds = 0.5 * ds;
    double zl;
    {
      const double m = x + hds * e, mh = m + h, mr = mh - h;
      const double qm = m * m, qh = mh * mh, qr = mr * mr;
      const double m0 = from_lane(qm, 0), m1 = from_lane(qm, 1), m2 = from_lane(qm, 2);
      const double h0 = from_lane(qh, 0), h1 = from_lane(qh, 1), h2 = from_lane(qh, 2);
      const double r0 = from_lane(qr, 0), r1 = from_lane(qr, 1);
      const double y0 = !sub ? m0 : s == 0 ? h0 : r0;
      const double y1 = !sub || s < 1 ? m1 : s == 1 ? h1 : r1;
      const double y2 = !sub || s < 2 ? m2 : h2;
      zl = main_pt ? z : sqrt(y0 + y1 + y2) - kRE;
    }
    double pl, tl;
    if (alive) lev64_find(a, zl, lv);
    else if (lv.i < 0) lev64_load(a, 0, lv);
    lev64_pt(a, lv, zl, &pl, &tl);
    const double nl = kRefrac * pl / tl;
    const double nmain = from_lane(nl, 4), nmid = from_lane(nl, 3), t = from_lane(tl, 4);
    if (alive) {
      const long long q = base + n;
      if (n > 0 && s == 0)
        L.ds[q - 1] = n == 1 ? raw_pend * 0.5 : 0.5 * (raw_before + raw_pend);
      raw_before = raw_pend;
      raw_pend = ds;
      // for k_points64: the altitude and its level interval in aux and qh2o
      if (s == 4) L.p[q] = pl;
      if (s == 5) L.t[q] = tl;
      if (s == 6) L.aux[q] = zl;
      if (s == 7) L.qh2o[q] = __longlong_as_double(lv.i);
      const bool newmin = n == 0 || lt(z, zmin_seen);
      if (s < 3) {
        if (n == 0) kp.x0[s] = x;
        if (want_p1) kp.xp[s] = x;
        if (newmin) kp.xm[s] = last_x;
      }
      if (s == 0) {
        if (n == 0) kp.z0 = z;
        if (want_p1) {
          kp.zp1 = z;
          kp.ds_p1 = ds;
        }
        if (newmin) {
          kp.zmin = z;
          kp.imin = n;
          kp.ds_m = ds;
          kp.zm1 = last_z;
        }
      }
      if (newmin) zmin_seen = z;
      want_p1 = newmin;
      last_z = z;
      last_x = x;
      n++;
      if (stop) {
        sft = stop == 2 ? (c.nsf > 0 && a.sft > 0 ? a.sft : t) : -999;
        if (s == 0) {
          L.ds[q] = n == 1 ? raw_pend * 0.5 : 0.5 * (raw_before + raw_pend);
          kp.zl = z;
        }
        if (s < 3) kp.xl[s] = x;
        alive = false;
      }
    }
    const bool bend = c.refrac && !lt(zrefrac, z);
    const double ec = bend ? e * (1 + nmain) + ds * div_by(nl - nmid, h, rh) : e;
    const double en = ec / sqrt(sum3(ec * ec));
    if (alive) {
      x += hds * (e + en);
      e = en;
    }
  }
  __syncwarp();
  if (r >= 0 && s == 0) ray_finish(b, L, r, st < 0 ? -1 : n, sft, kp);
}

// A block per ray, a thread per point: what k_walk8 left out.  The sums of a
// ray's column densities run along it, a thread per emitter over the block's
// points in shared memory, kSumGas emitters at a time.
constexpr int kPointThreads = 128, kSumGas = 8;

template <bool CGA>
__global__ void __launch_bounds__(kPointThreads)
    k_points64(CtlDev c, BatchDev b, LosDev L, const double* slopes) {
  __shared__ double su[CGA ? kSumGas : 1][kPointThreads], sp[CGA ? kSumGas : 1][kPointThreads],
      st[CGA ? kSumGas : 1][kPointThreads];
  const int r = blockIdx.x, tid = threadIdx.x;
  const int n = L.count[r];
  if (n <= 0) return;
  const long long base = L.off[r];
  const AtmView a = atm_view(c, b, slopes, b.ray_obs[r]);
  const bool cloud = c.ncl > 0 && a.cldz > 0;
  const int groups = CGA ? max((c.ng + kSumGas - 1) / kSumGas, 1) : 1;
  for (int gr = 0; gr < groups; gr++) {
    const int g0 = gr * kSumGas, g1 = CGA ? min(g0 + kSumGas, c.ng) : c.ng;
    double u_s = 0, p_s = 0, t_s = 0;
    for (int ip0 = 0; ip0 < n; ip0 += kPointThreads) {
      const int ip = ip0 + tid;
      const long long q = base + ip;
      if (ip < n) {
        const int i = (int)__double_as_longlong(L.qh2o[q]);
        const double z = L.aux[q], dz = z - a.z[i], p = L.p[q], t = L.t[q], ds = L.ds[q];
        const double kt = kKB * t, rt = 1 / kt;
        for (int g = g0; g < g1; g++) {
          const double v = a.q[g * a.stride + i] + a.sq[g * a.stride + i] * dz;
          const double u = div_by(10 * v * p, kt, rt) * ds;
          L.u[g * L.cap + q] = u;
          if (CGA) {
            su[g - g0][tid] = u;
            sp[g - g0][tid] = u * p;
            st[g - g0][tid] = u * t;
          }
        }
        if (gr == groups - 1) {  // the point's altitude and interval end here
          for (int iw = 0; iw < a.nw; iw++)
            L.kw[iw * L.cap + q] = a.k[iw * a.stride + i] + a.sk[iw * a.stride + i] * dz;
          if (c.ig_h2o >= 0)
            L.qh2o[q] = a.q[c.ig_h2o * a.stride + i] + a.sq[c.ig_h2o * a.stride + i] * dz;
          L.aux[q] = cloud ? exp(-0.5 * ((z - a.clz) / a.cldz) * ((z - a.clz) / a.cldz)) : 0.0;
        }
      }
      if (CGA) {
        __syncthreads();
        if (tid < g1 - g0)
          for (int j = 0; j < min(n - ip0, kPointThreads); j++) {
            const bool first = ip0 + j == 0;
            su[tid][j] = u_s = first ? su[tid][j] : u_s + su[tid][j];
            sp[tid][j] = p_s = first ? sp[tid][j] : p_s + sp[tid][j];
            st[tid][j] = t_s = first ? st[tid][j] : t_s + st[tid][j];
          }
        __syncthreads();
        if (ip < n)
          for (int g = g0; g < g1; g++) {
            const double uu = su[g - g0][tid], ru = 1 / uu;
            L.cgu[g * L.cap + q] = uu;
            L.cgp[g * L.cap + q] = div_by(sp[g - g0][tid], uu, ru);
            L.cgt[g * L.cap + q] = div_by(st[g - g0][tid], uu, ru);
          }
        __syncthreads();
      }
    }
  }
}

// ---------------------------------------------------------------------------
// tables

struct Row {
  const float* u;
  const float* e;
  int n;
};

__device__ inline Row row_at(const TblDev& T, long long dg, int ip, int it) {
  const long long r = (dg * T.tp + ip) * T.tt + it;
  Row w;
  w.u = T.u + r * T.tu;
  w.e = T.eps + r * T.tu;
  w.n = T.nu[r];
  return w;
}

// intpol_tbl_eps (jurassic.c:3895-3929)
__device__ inline double row_eps(const Row& r, double u) {
  if (u < (double)r.u[0]) return lin_f(0.0f, 0.0f, r.u[0], r.e[0], u);
  if (u > (double)r.u[r.n - 1]) {
    const double a = log((double)(1 - r.e[r.n - 1])) / (double)r.u[r.n - 1];
    return 1 - exp(a * u);
  }
  const int i = bracket_row(r.u, r.n, u);
  return lin_f(r.u[i], r.e[i], r.u[i + 1], r.e[i + 1], u);
}

// intpol_tbl_u (jurassic.c:3933-3967)
__device__ inline double row_u(const Row& r, double e) {
  if (e < (double)r.e[0]) return lin_f(0.0f, 0.0f, r.e[0], r.u[0], e);
  if (e > (double)r.e[r.n - 1]) {
    const double a = log((double)(1 - r.e[r.n - 1])) / (double)r.u[r.n - 1];
    return log(1 - e) / a;
  }
  const int i = bracket_row(r.e, r.n, e);
  return lin_f(r.e[i], r.u[i], r.e[i + 1], r.u[i + 1], e);
}

// Segment emissivity of one (channel, emitter) at one LOS point; updates
// the extended-path transmittance (intpol_tbl_ega / intpol_tbl_cga).
__device__ inline double gas_eps(const TblDev& T, long long dg, bool cga, double pq, double tq,
                                 double du, double ucg, double* tau_path) {
  const int np = T.np[dg];
  if (np < 30) return 0;
  if (*tau_path < 1e-9) return 1;
  const double* pg = T.p + dg * T.tp;
  const int* ntg = T.nt + dg * T.tp;
  const int ipr = bracket_irr(pg, np, pq);
  const double* t0g = T.t + (dg * T.tp + ipr) * T.tt;
  const double* t1g = t0g + T.tt;
  const int it0 = bracket_reg(t0g, ntg[ipr], tq);
  const int it1 = bracket_reg(t1g, ntg[ipr + 1], tq);
  if (ntg[ipr] < 2 || ntg[ipr + 1] < 2) return 0;
  const Row r00 = row_at(T, dg, ipr, it0), r01 = row_at(T, dg, ipr, it0 + 1);
  const Row r10 = row_at(T, dg, ipr + 1, it1), r11 = row_at(T, dg, ipr + 1, it1 + 1);
  if (r00.n < 2 || r01.n < 2 || r10.n < 2 || r11.n < 2) return 0;
  double e00, e01, e10, e11;
  if (cga) {
    e00 = row_eps(r00, ucg);
    e01 = row_eps(r01, ucg);
    e10 = row_eps(r10, ucg);
    e11 = row_eps(r11, ucg);
  } else {
    const double prev = 1 - *tau_path;
    e00 = row_eps(r00, row_u(r00, prev) + du);
    e01 = row_eps(r01, row_u(r01, prev) + du);
    e10 = row_eps(r10, row_u(r10, prev) + du);
    e11 = row_eps(r11, row_u(r11, prev) + du);
  }
  e00 = lin(t0g[it0], e00, t0g[it0 + 1], e01, tq);
  e11 = lin(t1g[it1], e10, t1g[it1 + 1], e11, tq);
  e00 = cga ? logx(pg[ipr], e00, pg[ipr + 1], e11, pq) : lin(pg[ipr], e00, pg[ipr + 1], e11, pq);
  e00 = e00 < 1 ? e00 : 1;
  e00 = e00 > 0 ? e00 : 0;
  return 1 - (1 - e00) / *tau_path;
}

// formod_srcfunc (jurassic.c:3483-3496) for one channel
__device__ inline double src_at(const TblDev& T, int nd, int id, double t) {
  const int it = bracket_reg(T.st, kNS, t);
  return lin(T.st[it], T.sr[(long long)it * nd + id], T.st[it + 1], T.sr[(long long)(it + 1) * nd + id], t);
}

// continua (ctmco2/ctmh2o/ctmn2/ctmo2 with the wavenumber-only factors
// precomputed per channel on the host, see ctm_coefficients in jgb_api.cu)
__device__ inline double continuum_beta(const CtlDev& c, const double* cc, double kext, double p,
                                        double t, double ds, double uco2, double uh2o,
                                        double qh2o, double nu) {
  double beta = kext;
  if (c.ctm_co2 && c.ig_co2 >= 0 && cc[0] != 0) {
    const double d230 = t - 230, d260 = t - 260, d296 = t - 296;
    const double ctw = d260 * 5.050505e-4 * d296 * cc[3] - d230 * 9.259259e-4 * d296 * cc[2] +
                       d230 * 4.208754e-4 * d260 * cc[1];
    beta += uco2 / kNA / 1000 * p / kP0 * ctw / ds;
  }
  if (c.ctm_h2o && c.ig_h2o >= 0 && cc[4] != 0) {
    const double self = cc[5] * pow(cc[6], (296 - t) / (296 - 260));
    const double a1 = nu * uh2o * tanh(.7193876 / t * nu);
    const double a2 = 296 / t;
    const double a3 = p / kP0 * (qh2o * self + (1 - qh2o) * cc[7]) * 1e-20;
    beta += a1 * a2 * a3 / ds;
  }
  if (c.ctm_n2 && cc[8] != 0) {
    const double qn = 0.79, t0 = 273.0, tr = 296.0;
    const double x = p / kP0 * t0 / t;
    beta += 0.1 * (x * x) * exp(cc[10] * (1 / tr - 1 / t)) * qn * cc[9] *
            (qn + (1 - qn) * (1.294 - 0.4545 * t / tr));
  }
  if (c.ctm_o2 && cc[11] != 0) {
    const double qo = 0.21, t0 = 273, tr = 296;
    const double x = p / kP0 * t0 / t;
    beta += 0.1 * (x * x) * exp(cc[13] * (1 / tr - 1 / t)) * qo * cc[12];
  }
  return beta;
}

// Per-(observation, channel) constants derived from the atmosphere record.
__device__ inline void obs_channel_consts(const CtlDev& c, const ChanDev& ch, const double* s,
                                          int id, double* cloud, bool* has_cloud,
                                          double* sfeps) {
  const double nu = ch.nu[id];
  *has_cloud = c.ncl > 0 && s[1] > 0;
  *cloud = 0;
  if (*has_cloud) {
    const int icl = bracket_irr(ch.clnu, c.ncl, nu);
    *cloud = lin(ch.clnu[icl], s[2 + icl], ch.clnu[icl + 1], s[2 + icl + 1], nu);
  }
  *sfeps = 1.0;
  if (c.nsf > 0) {
    const double* se = s + 5 + c.ncl;
    const int isf = bracket_irr(ch.sfnu, c.nsf, nu);
    *sfeps = lin(ch.sfnu[isf], se[isf], ch.sfnu[isf + 1], se[isf + 1], nu);
  }
}

__global__ void k_path_fp64(CtlDev c, TblDev T, ChanDev ch, BatchDev b, LosDev L,
                            double* refl_scratch) {
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nray = b.nray;
  if (gid >= nray * c.nd) return;
  const int id = (int)(gid / nray);
  const int r = (int)(gid % nray);
  const int o = b.ray_obs[r];
  if (b.obs_skip && b.obs_skip[o]) return;
  const int n = b.skip_masked && b.mask[gid] ? 0 : L.count[r];  // gid = id * nray + r
  const long long base = L.off[r];
  const double nu = ch.nu[id];
  const double* cc = ch.ctm + (long long)id * kCtmStride;
  const double* s = b.scal + (long long)o * b.nscal;
  double cloud, sfeps;
  bool has_cloud;
  obs_channel_consts(c, ch, s, id, &cloud, &has_cloud, &sfeps);
  const int w = c.nw > 0 ? ch.window[id] : 0;
  double tau_path[kMaxG];
  for (int ig = 0; ig < c.ng; ig++) tau_path[ig] = 1;
  double rad = 0, tau = 1;
  const bool cga = c.formod == 0;
  const bool refl = c.sftype >= 2 && sfeps < 1 && L.sft[r] > 0 && c.sftype >= 1;
  double* sc = refl ? refl_scratch + 2 * base * c.nd : nullptr;

  for (int ip = 0; ip < n; ip++) {
    const long long q = base + ip;
    const double p = L.p[q], t = L.t[q], ds = L.ds[q];
    double tau_gas = 1;
    for (int ig = 0; ig < c.ng; ig++) {
      const long long dg = (long long)id * c.ng + ig;
      const double du = cga ? 0.0 : L.u[ig * L.cap + q];
      const double pq = cga ? L.cgp[ig * L.cap + q] : p;
      const double tq = cga ? L.cgt[ig * L.cap + q] : t;
      const double ucg = cga ? L.cgu[ig * L.cap + q] : 0.0;
      const double eps = gas_eps(T, dg, cga, pq, tq, du, ucg, &tau_path[ig]);
      tau_path[ig] *= (1 - eps);
      tau_gas *= (1 - eps);
    }
    double kext = c.nw > 0 ? L.kw[w * L.cap + q] : 0.0;
    if (has_cloud) kext += L.aux[q] * cloud;
    const double uco2 = c.ig_co2 >= 0 ? L.u[c.ig_co2 * L.cap + q] : 0.0;
    const double uh2o = c.ig_h2o >= 0 ? L.u[c.ig_h2o * L.cap + q] : 0.0;
    const double qh2o = c.ig_h2o >= 0 ? L.qh2o[q] : 0.0;
    const double beta = continuum_beta(c, cc, kext, p, t, ds, uco2, uh2o, qh2o, nu);
    const double src = src_at(T, c.nd, id, t);
    double eps = 0;
    if (tau_gas > 0) {
      eps = 1 - tau_gas * exp(-beta * ds);
      rad += src * eps * tau;
      tau *= (1 - eps);
    }
    if (sc) {
      sc[2 * ((long long)ip * c.nd + id)] = src;
      sc[2 * ((long long)ip * c.nd + id) + 1] = eps;
    }
  }

  // surface emission, reflection and solar term (jurassic.c:3264-3328)
  const double sft = L.sft[r];
  if (c.sftype >= 1 && sft > 0) {
    rad += sfeps * src_at(T, c.nd, id, sft) * tau;
    if (refl) {
      double tau_refl = 1;
      for (int ip = n - 1; ip >= 0; ip--) {
        const double src = sc[2 * ((long long)ip * c.nd + id)];
        const double e = sc[2 * ((long long)ip * c.nd + id) + 1];
        rad += src * e * tau_refl * tau * (1 - sfeps);
        tau_refl *= (1 - e);
      }
      if (c.sftype >= 3) {
        const double* e6 = L.ends + 6LL * r;
        const double sza2 = c.sfsza < 0 ? solar_zenith(b.geo[r], e6[4], e6[5]) : c.sfsza;
        if (sza2 < 89.999) {
          double x0[3], x1[3];
          to_cart(e6[3], e6[4], e6[5], x0);
          to_cart(e6[0], e6[1], e6[2], x1);
          for (int i = 0; i < 3; i++) x1[i] -= x0[i];
          const double cosa = (x0[0] * x1[0] + x0[1] * x1[1] + x0[2] * x1[2]) /
                              sqrt(x0[0] * x0[0] + x0[1] * x0[1] + x0[2] * x0[2]) /
                              sqrt(x1[0] * x1[0] + x1[1] * x1[1] + x1[2] * x1[2]);
          const double rcos = cosa / cos(sza2 * (kPI / 180.0));
          rad += 6.764e-5 / (2. * kPI) * planck(kTSUN, nu) * tau_refl * (1 - sfeps) * tau * rcos;
        }
      }
    }
  }
  const long long oi = (long long)id * nray + r;
  if (c.fov) {  // pencil beam only: FOV convolution, BT and mask follow in k_fov
    b.rad[oi] = rad;
    b.tau[oi] = tau;
    return;
  }
  if (c.write_bbt) rad = kC2 * nu / log1p(kC1 * (nu * nu * nu) / rad);
  b.rad[oi] = b.mask[oi] ? __longlong_as_double(0x7ff8000000000000LL) : rad;
  b.tau[oi] = tau;
}

// init_srcfunc (jurassic.c:3631-3681): one thread per (temperature, channel)
__global__ void k_srcfunc(int nd, int id0, int nch, const int* fn_off, const double* fnu,
                          const double* f, const double* st, double* sr) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= kNS * nch) return;
  const int it = gid % kNS;
  const int j = gid / kNS;
  const int id = id0 + j;
  const double* x = fnu + fn_off[j];
  const double* y = f + fn_off[j];
  const int n = fn_off[j + 1] - fn_off[j];
  double dnu = 1.0;
  for (int i = 1; i < n; i++) dnu = (x[i] - x[i - 1]) < dnu ? (x[i] - x[i - 1]) : dnu;
  const double temp = st[it];
  double fsum = 0, acc = 0;
  for (double v = x[0]; v <= x[n - 1]; v += dnu) {
    const int i = bracket_irr(x, n, v);
    const double w = lin(x[i], y[i], x[i + 1], y[i + 1], v);
    fsum += w;
    acc += w * planck(temp, v);
  }
  sr[(long long)it * nd + id] = acc / fsum;
}

// hydrostatic (jurassic.c:3520-3582) in two kernels.  The mean of g M / (R T)
// over a layer depends on nothing but the layer: a warp per profile, a lane per
// layer, leaves mean * 1000 * dz in the place of the pressure that it leads to.
// The pressures follow each other along the profile, a thread per profile.
// Every value is formed as in a loop over the profile, one thread of which took
// 2.04 ms for 1500 profiles of 77 levels: 20 means of 17 FP64 instructions per
// layer, one after the other; 0.42 ms here.
__device__ int hydro_ref(const double* z, int np, double hydz) {
  double best = 1e99;
  int iref = 0;
  for (int ip = 0; ip < np; ip++)
    if (fabs(z[ip] - hydz) < best) {
      best = fabs(z[ip] - hydz);
      iref = ip;
    }
  return iref;
}

__global__ void k_hydro_means(CtlDev c, BatchDev b, double* p_out) {
  const int lane = threadIdx.x & 31;
  const int o = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (o >= b.nobs || c.hydz < 0) return;
  if (b.obs_skip && b.obs_skip[o]) return;
  const int l0 = b.lev_off[o], np = b.lev_off[o + 1] - l0;
  const double* z = b.z + l0;
  const double* t = b.t + l0;
  const double* qw = c.ig_h2o >= 0 ? b.q + (long long)c.ig_h2o * b.nlev + l0 : nullptr;
  const double mmair = 28.96456e-3, mmh2o = 18.0153e-3;
  const int npts = 20;
  const int iref = hydro_ref(z, np, c.hydz);
  for (int ip = lane; ip < np; ip += 32) {
    if (ip == iref) continue;
    const int i0 = ip > iref ? ip - 1 : ip + 1;
    double mean = 0, e = 0;
    for (int i = 0; i < npts; i++) {
      if (qw) e = lin(0.0, qw[i0], npts - 1.0, qw[ip], (double)i);
      mean += (e * mmh2o + (1 - e) * mmair) * kG0 / kRI /
              lin(0.0, t[i0], npts - 1.0, t[ip], (double)i) / npts;
    }
    p_out[l0 + ip] = mean * 1000 * (z[ip] - z[i0]);
  }
}

__global__ void k_hydro_chain(CtlDev c, BatchDev b, double* p_out) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= b.nobs || c.hydz < 0) return;
  if (b.obs_skip && b.obs_skip[o]) return;
  const int l0 = b.lev_off[o], np = b.lev_off[o + 1] - l0;
  double* p = p_out + l0;
  const int iref = hydro_ref(b.z + l0, np, c.hydz);
  for (int ip = iref + 1; ip < np; ip++) p[ip] = exp(log(p[ip - 1]) - p[ip]);
  for (int ip = iref - 1; ip >= 0; ip--) p[ip] = exp(log(p[ip + 1]) - p[ip]);
}

// ---------------------------------------------------------------------------
// launch wrappers

// Eight lanes per ray up to here: a step is about 100 FP64 instructions of a
// warp (4 rays) against 330 (32 rays), 64 cycles each until about three warps
// share an SM, 19 of the SM's then, so the two forms meet between 6000 and
// 7000 rays on 152 SMs.  Eight lanes and one, ms: nadir 500 rays 4.06 and 9.57, 5000
// 8.25 and 9.91, 6144 9.65 and 9.99, 7000 10.53 and 10.01, 12000 20.7 and 10.2; limb
// 6144 3.90 and 5.13, 8192 4.87 and 5.22, 12000 6.18 and 5.40.
constexpr int kWalk8MaxRays = 6144;

size_t level_slope_bytes(const CtlDev& c, long long nlev) {
  return sizeof(double) * (size_t)nlev * (2 + c.ng + c.nw);
}

void launch_level_slopes(const CtlDev& c, const BatchDev& b, double* slopes, cudaStream_t s) {
  const long long nth = (long long)b.nobs * 32;
  k_level_slopes<<<(unsigned)((nth + 127) / 128), 128, 0, s>>>(c, b, slopes);
}

void launch_trace_count(const CtlDev& c, const BatchDev& b, const LosDev& L, const double* slopes,
                        unsigned* err, cudaStream_t s) {
  const int bs = kTrace64Threads;
  k_trace_count<<<(b.nray + bs - 1) / bs, bs, 0, s>>>(c, b, L, slopes, err);
}

void launch_trace_fill(const CtlDev& c, const BatchDev& b, const LosDev& L, const int* order,
                       const double* slopes, unsigned* err, cudaStream_t s) {
  if (slopes && b.nray <= kWalk8MaxRays) {
    k_walk8<<<(b.nray + kWalk8Rays - 1) / kWalk8Rays, 32, 0, s>>>(c, b, L, order, slopes, err);
    if (L.cga) k_points64<true><<<b.nray, kPointThreads, 0, s>>>(c, b, L, slopes);
    else k_points64<false><<<b.nray, kPointThreads, 0, s>>>(c, b, L, slopes);
    return;
  }
  const int bs = kTrace64Threads;
  k_trace_fill<<<(b.nray + bs - 1) / bs, bs, sizeof(double) * trace64_smem(c) * bs, s>>>(
      c, b, L, order, slopes, err);
}

void launch_path_fp64(const CtlDev& c, const TblDev& T, const ChanDev& ch, const BatchDev& b,
                      const LosDev& L, double* refl_scratch, cudaStream_t s) {
  const long long nth = (long long)b.nray * c.nd;
  const int bs = 128;
  k_path_fp64<<<(unsigned)((nth + bs - 1) / bs), bs, 0, s>>>(c, T, ch, b, L, refl_scratch);
}

void launch_srcfunc(int nd, int id0, int nch, const int* fn_off, const double* fnu,
                    const double* f, const double* st, double* sr, cudaStream_t s) {
  const int nth = kNS * nch, bs = 128;
  k_srcfunc<<<(nth + bs - 1) / bs, bs, 0, s>>>(nd, id0, nch, fn_off, fnu, f, st, sr);
}

// formod_fov (jurassic.c:3121-3192), then BRIGHT and the mask of formod
// (3057-3067): one thread per (ray, channel) reads the pencil beams of the
// rays within +-5 of its own in the same observation with the same time.
__global__ void k_fov(CtlDev c, BatchDev b, const double* prad, const double* ptau, int nfov,
                      const double* fdz, const double* fw, const double* nu, unsigned* err) {
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nray = b.nray;
  if (gid >= nray * c.nd) return;
  const int id = (int)(gid / nray);
  const int r = (int)(gid % nray);
  const int o = b.ray_obs[r];
  if (b.obs_skip && b.obs_skip[o]) return;
  const double* time = b.geo;
  const double* vpz = b.geo + 4 * nray;
  double zz[11];
  int ray[11], nz = 0;
  const int lo = r - 5 > 0 ? r - 5 : 0;
  const int hi = r + 6 < nray ? r + 6 : (int)nray;
  for (int r2 = lo; r2 < hi; r2++)
    if (b.ray_obs[r2] == o && time[r2] == time[r]) {
      zz[nz] = vpz[r2];
      ray[nz++] = r2;
    }
  if (nz < 2) {
    atomicOr(err, kErrFov);
    return;
  }
  const double* pr = prad + (long long)id * nray;
  const double* pt = ptau + (long long)id * nray;
  double rs = 0, ts = 0, wsum = 0;
  for (int i = 0; i < nfov; i++) {
    const double zf = vpz[r] + fdz[i];
    const int k = bracket_irr(zz, nz, zf);
    rs += fw[i] * lin(zz[k], pr[ray[k]], zz[k + 1], pr[ray[k + 1]], zf);
    ts += fw[i] * lin(zz[k], pt[ray[k]], zz[k + 1], pt[ray[k + 1]], zf);
    wsum += fw[i];
  }
  rs /= wsum;
  ts /= wsum;
  if (c.write_bbt) {
    const double v = nu[id];
    rs = kC2 * v / log1p(kC1 * (v * v * v) / rs);
  }
  const long long oi = (long long)id * nray + r;
  b.rad[oi] = b.mask[oi] ? __longlong_as_double(0x7ff8000000000000LL) : rs;
  b.tau[oi] = ts;
}

void launch_fov(const CtlDev& c, const BatchDev& b, const double* prad, const double* ptau,
                int nfov, const double* fdz, const double* fw, const double* nu, unsigned* err,
                cudaStream_t s) {
  const long long nth = (long long)b.nray * c.nd;
  const int bs = 128;
  k_fov<<<(unsigned)((nth + bs - 1) / bs), bs, 0, s>>>(c, b, prad, ptau, nfov, fdz, fw, nu, err);
}

void launch_hydrostatic(const CtlDev& c, const BatchDev& b, double* p_out, cudaStream_t s) {
  k_hydro_means<<<(b.nobs + 3) / 4, 128, 0, s>>>(c, b, p_out);
  k_hydro_chain<<<(b.nobs + 31) / 32, 32, 0, s>>>(c, b, p_out);
}

// Loads the FP64 forward-model kernels onto the current device (CUDA loads
// modules lazily, at a kernel's first launch or attribute query), so that a
// later first launch allocates no device memory for their code.
int preload_fp64_kernels() {
  cudaFuncAttributes a;
  const void* fns[] = {(const void*)k_trace_count, (const void*)k_trace_fill, (const void*)k_path_fp64, (const void*)k_hydro_means, (const void*)k_hydro_chain};
  for (const void* f : fns)
    if (cudaFuncGetAttributes(&a, f) != cudaSuccess) return JGB_ERR_CUDA;
  return JGB_OK;
}

}  // namespace jgb
