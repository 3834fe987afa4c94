// FP64 path: formod_pencil (jurassic.c:3196-3338) with intpol_tbl_ega /
// intpol_tbl_cga (3710-3891), formod_continua (3075-3117) and
// formod_srcfunc (3483-3496) in double precision, as four kernels over
// tiles of 32 length-sorted rays:
//
//   k_prep64   one thread per (LOS point, ray): everything that does not
//              depend on the channel (p-T cell and interpolation weights of
//              every emitter, continuum factors, source-table index),
//              written lane-major so that the channels read it coalesced;
//   k_gas64    the only chain along the path: one warp per (tile, channel,
//              emitter) walks the points with that emitter's path
//              emissivity and writes its path transmittances.  Small batches
//              give each ray four lanes, one per corner of the p-T cell;
//   k_seg64    one warp per (point, channel): continua, source function and
//              the segment's emissivity, all points at once;
//   k_scan64   one thread per (ray, channel): radiance and transmittance
//              sums, surface, reflection, sun, BT and mask.
//
// Why this split: an FP64 instruction of a warp holds its scheduler for 64
// cycles on GB300 and the whole SM for 19 (measured with chains of DFMA, 1
// to 8 warps per SM, however many lanes are active; a compare or a conversion
// costs about the same, a division 5 of them, exp 16, log 31), so the path is
// bound by the number of FP64 instructions, and a small batch by how many of
// them follow one another.  One thread per (ray, channel) for the whole of
// formod_pencil issued 292 of them per (point, channel, emitter); here it is
// 63 in the gas chain and, per (point, channel), 100 in the parallel part:
//  * table searches compare floats: the entries are floats, and g <= x holds
//    for a double x exactly where g <= x rounded down to float, so one
//    rounding on the integer pipe replaces ~50 FP64 compares per point;
//    searches start from the last point's bracket;
//  * p-T cells and continuum factors once per point instead of per channel;
//  * divisions by grid steps take the step's reciprocal (div_by: the same
//    quotient in three instructions);
//  * lanes whose searches end differently interpolate together.
// Every interpolation and path product rounds as in formod_pencil (a finite
// difference of two of these radiances sees no other rounding); only the
// continuum's factors are grouped differently.
// Measured, path stage of a call: nadir 1000 observations x 100 channels x 5
// emitters (1e6 points) 372 -> 91 ms (k_gas64 27 and k_seg64 6.7 ms per 352
// observations, the FP64 pipe 80-100 % busy by its 19 cycles); 10 limb rays x
// 3 channels x 2 emitters (904 points) 69.6 -> 3.4 ms; 273 limb rays x 11
// channels x 4 emitters, CGA, 30.2 -> 3.2 ms.
//
// Compiled with -fmad=false; products and sums are fused only where fma() is
// written, so that every variant rounds alike (a ray's result does not
// depend on its batch).
#include "../../include/jurassic_gb300.h"
#include "jgb_common.cuh"
#include "jgb_internal.h"
#include "jgb_path64.cuh"

namespace jgb {
namespace {

// ---------------------------------------------------------------------------
// per-point fields: doubles fd[(point * nfd + field) * 32 + lane] and words
// fu[(point * nfu + field) * 32 + lane]

// emitter: u (EGA: column of the segment, CGA: of the path), then d, w, r of the
// pressure and of the two temperature interpolations
constexpr int kGas64 = 10;

struct Fields64 {
  int ds, rds, ws, aux, kw0, co2, h2o, n2, g0;  // doubles; emitter g at g0 + kGas64 g
  int nfd, nfu;                            // words: 0 source index, 1 + g rows
};

__host__ __device__ inline Fields64 fields64(const CtlDev& c) {
  Fields64 f;
  int k = 0;
  f.ds = k++;
  f.rds = k++;
  f.ws = k++;
  f.aux = k;
  if (c.ncl > 0) k++;
  f.kw0 = k;
  k += c.nw;
  f.co2 = k;
  if (c.ctm_co2 && c.ig_co2 >= 0) k += 4;
  f.h2o = k;
  if (c.ctm_h2o && c.ig_h2o >= 0) k += 4;
  f.n2 = k;
  if (c.ctm_n2 || c.ctm_o2) k += 3;
  f.g0 = k;
  f.nfd = k + kGas64 * c.ng;
  f.nfu = 1 + c.ng;
  return f;
}

constexpr unsigned kNoCell = 0xffffffffu;  // no temperature rows at that pressure
constexpr unsigned kLogP = 0x8000u;        // pressure weight in log form (in the rows word)

// One interpolation y0 + (y1 - y0) / w * d (LIN) with the reciprocal r of w.
struct Lin64 {
  double d, w, r;
};

// The p-T cell of (p, t) in table dg: rows ra = ipr * tt + it0 and rc =
// (ipr + 1) * tt + it1 (ra < 0: no rows), the interpolations in pressure and
// at both pressures in temperature (intpol_tbl_ega, intpol_tbl_cga).
struct Cell64 {
  int ra, rc;
  bool logp;
  Lin64 p, a, b;
};

template <bool CGA>
__device__ inline Cell64 cell64(const TblDev& T, long long dg, int np, double pq, double tq) {
  Cell64 k{};
  k.ra = -1;
  const double* pg = T.p + dg * T.tp;
  const int* ntg = T.nt + dg * T.tp;
  const int ipr = bracket_irr(pg, np, pq);
  const int nt0 = ntg[ipr], nt1 = ntg[ipr + 1];
  if (nt0 < 2 || nt1 < 2) return k;
  const double* t0g = T.t + (dg * T.tp + ipr) * T.tt;
  const double* t1g = t0g + T.tt;
  const int it0 = bracket_reg(t0g, nt0, tq), it1 = bracket_reg(t1g, nt1, tq);
  k.ra = ipr * T.tt + it0;
  k.rc = (ipr + 1) * T.tt + it1;
  k.a.d = tq - t0g[it0];
  k.a.w = t0g[it0 + 1] - t0g[it0];
  k.a.r = 1 / k.a.w;
  k.b.d = tq - t1g[it1];
  k.b.w = t1g[it1 + 1] - t1g[it1];
  k.b.r = 1 / k.b.w;
  const double pa = pg[ipr], pb = pg[ipr + 1];
  k.logp = CGA && pq / pa > 0 && pb / pa > 0;
  k.p.d = k.logp ? log(pq / pa) : pq - pa;
  k.p.w = k.logp ? log(pb / pa) : pb - pa;
  k.p.r = 1 / k.p.w;
  return k;
}

// a / w from the reciprocal r of w: the quotient, its exact remainder and one
// correction (Markstein, IBM J. Res. Dev. 34, 1990) give the correctly rounded
// quotient of a division, in three instructions.
__device__ __forceinline__ double div_by(double a, double w, double r) {
  const double q = a * r;
  return fma(fma(-q, w, a), r, q);
}

__device__ __forceinline__ double lin64(double y0, double y1, const Lin64& l) {
  return y0 + div_by(y1 - y0, l.w, l.r) * l.d;
}

template <bool CGA>
__global__ void __launch_bounds__(128) k_prep64(CtlDev c, TblDev T, LosDev L, Path64 P) {
  const int tile = P.tile0 + (int)blockIdx.y;
  const int lane = threadIdx.x & 31;
  const int ip = (int)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int r = P.perm[tile * 32 + lane];
  const long long lp = P.toff[tile] - P.pt0 + ip;
  if (P.toff[tile] + ip >= P.toff[tile + 1] || r < 0 || ip >= L.count[r]) return;
  const Fields64 F = fields64(c);
  double* fd = P.fd + lp * F.nfd * 32 + lane;
  unsigned* fu = P.fu + lp * F.nfu * 32 + lane;
  const long long q = L.off[r] + ip;
  const double p = L.p[q], t = L.t[q], ds = L.ds[q];
  fd[F.ds * 32] = ds;
  // source-function table: index and offset
  const int it = bracket_reg(T.st, kNS, t);
  fu[0] = (unsigned)it;
  fd[F.ws * 32] = t - T.st[it];
  if (c.ncl > 0) fd[F.aux * 32] = L.aux[q];
  for (int w = 0; w < c.nw; w++) fd[(F.kw0 + w) * 32] = L.kw[w * L.cap + q];
  // continua: everything but the channel's coefficients (ctmco2, ctmh2o,
  // ctmn2, ctmo2), as factors of beta
  const double rds = 1 / ds;
  fd[F.rds * 32] = rds;
  if (c.ctm_co2 && c.ig_co2 >= 0) {
    const double d230 = t - 230, d260 = t - 260, d296 = t - 296;
    fd[(F.co2 + 0) * 32] = L.u[c.ig_co2 * L.cap + q] / kNA / 1000 * p / kP0;
    fd[(F.co2 + 1) * 32] = d260 * 5.050505e-4 * d296;
    fd[(F.co2 + 2) * 32] = d230 * 9.259259e-4 * d296;
    fd[(F.co2 + 3) * 32] = d230 * 4.208754e-4 * d260;
  }
  if (c.ctm_h2o && c.ig_h2o >= 0) {
    const double qh = L.qh2o[q];
    const double f = L.u[c.ig_h2o * L.cap + q] * (296 / t) * (p / kP0) * 1e-20 * rds;
    fd[(F.h2o + 0) * 32] = .7193876 / t;
    fd[(F.h2o + 1) * 32] = (296 - t) / (296 - 260);
    fd[(F.h2o + 2) * 32] = f * qh;
    fd[(F.h2o + 3) * 32] = f * (1 - qh);
  }
  if (c.ctm_n2 || c.ctm_o2) {
    const double x = p / kP0 * 273.0 / t, x2 = 0.1 * (x * x);
    fd[(F.n2 + 0) * 32] = 1 / 296.0 - 1 / t;
    fd[(F.n2 + 1) * 32] = x2;
    fd[(F.n2 + 2) * 32] = x2 * 0.79 * (0.79 + (1 - 0.79) * (1.294 - 0.4545 * t / 296.0));
  }
  for (int g = 0; g < c.ng; g++) {
    double* f = fd + (F.g0 + kGas64 * g) * 32;
    const double pq = CGA ? L.cgp[g * L.cap + q] : p;
    const double tq = CGA ? L.cgt[g * L.cap + q] : t;
    f[0] = CGA ? L.cgu[g * L.cap + q] : L.u[g * L.cap + q];
    if (!((P.shared >> g) & 1u)) {  // grids differ between channels: the cell is found there
      f[32] = pq;
      f[64] = tq;
      continue;
    }
    const long long dg = (long long)P.gref[g] * c.ng + g;
    const int np = T.np[dg];
    unsigned rows = kNoCell;
    if (np >= 30) {
      const Cell64 k = cell64<CGA>(T, dg, np, pq, tq);
      if (k.ra >= 0) rows = (unsigned)k.ra | ((unsigned)k.rc << 16) | (k.logp ? kLogP : 0u);
      const Lin64* l[3] = {&k.p, &k.a, &k.b};
      for (int i = 0; i < 3; i++) {
        f[(1 + 3 * i) * 32] = l[i]->d;
        f[(2 + 3 * i) * 32] = l[i]->w;
        f[(3 + 3 * i) * 32] = l[i]->r;
      }
    }
    fu[(1 + g) * 32] = rows;
  }
}

// ---------------------------------------------------------------------------
// exact float helpers on the integer pipe

// The rare forms are calls: written inline they become predicated
// conversions and compares that every pass through the FP64 pipe pays for
// (105 instead of 56 FP64 instructions per step of k_gas64).
__device__ __noinline__ float round_down_slow(double x) { return __double2float_rd(x); }
__device__ __noinline__ bool above_slow(double x, float g) { return x > (double)g; }

// x rounded down to float (toward zero for x >= 0): for a float g, g <= x,
// g > x, x < g hold exactly where they hold for the rounded value.  Normal
// positive values by truncating the mantissa, others by the conversion.
__device__ __forceinline__ float round_down_f(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  if (hi - (897u << 20) < (254u << 20))
    return __uint_as_float(((hi - (896u << 20)) << 3) | (lo >> 29));
  if ((hi | lo) == 0u) return 0.f;
  return round_down_slow(x);
}

// x > g for a float g, given d = round_down_f(x)
__device__ __forceinline__ bool above_f(double x, float d, float g) {
  if (d == g) return above_slow(x, g);
  return d > g;
}

// e clamped to [0, 1] without FP64 compares.  What is not a number gives 0, as in
// k_path_fp64 and the mixed path: an emitter without a column has no Curtis-Godson
// pressure (0 / 0), and adds nothing.
__device__ __forceinline__ double clamp01(double e) {
  const unsigned hi = (unsigned)__double2hiint(e);
  if (hi < 0x3ff00000u) return e;
  const bool number = hi < 0x7ff00000u || (hi == 0x7ff00000u && __double2loint(e) == 0);
  return number ? 1.0 : 0.0;  // negative numbers are above 0x7ff00000 as well
}

// a < b for doubles that are not negative (and not NaN), on the integer pipe
__device__ __forceinline__ bool less_pos(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}

// ---------------------------------------------------------------------------
// table rows

template <int C>
__device__ __forceinline__ float part(const float2 v) {
  return C == 0 ? v.x : v.y;
}

// Largest i in [lo, hi - 1] with component C of g[i] <= x as the bisection of
// locate_tbl (jurassic.c:4152-4170) finds it from [lo, hi].
template <int C>
__device__ __forceinline__ int bisect64(const float2* g, int lo, int hi, float x) {
  const float* gc = reinterpret_cast<const float*>(g) + C;
  while (hi > lo + 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(gc + 2 * mid) > x) hi = mid; else lo = mid;
  }
  return lo;
}

struct Pair64 {
  int i;
  float2 a, b;  // entries i and i + 1
};

// Bracket of x in component C of an n-entry row.  On rows that never fall
// (mono) the bracket is unique, so the remembered one and its successor are
// tried first; the third probe may lie one entry past the row (padding or
// the next row) and is ignored there.  Other rows take the plain bisection.
template <int C>
__device__ __forceinline__ Pair64 find64(const float2* g, int n, float x, int h, bool mono) {
  if (mono) {
    h = min(max(h, 0), n - 2);
    const float2 A = __ldg(g + h), B = __ldg(g + h + 1), D = __ldg(g + h + 2);
    const float a = part<C>(A), b = part<C>(B), d = part<C>(D);
    if (a <= x && (x < d || h + 2 >= n - 1)) {
      const bool up = x >= b && h + 2 < n;
      return up ? Pair64{h + 1, B, D} : Pair64{h, A, B};
    }
    const int i = a <= x ? bisect64<C>(g, h + 2, n - 1, x) : bisect64<C>(g, 0, h, x);
    return Pair64{i, __ldg(g + i), __ldg(g + i + 1)};
  }
  const int i = bisect64<C>(g, 0, n - 1, x);
  return Pair64{i, __ldg(g + i), __ldg(g + i + 1)};
}

// intpol_tbl_eps beyond the row's last entry: exponential saturation
__device__ __noinline__ double eps_above(float un, float en, double u) {
  const double a = log((double)(1 - en)) / (double)un;
  return 1 - exp(a * u);
}

// intpol_tbl_u beyond the row's last entry
__device__ __noinline__ double u_above(float un, float en, double e) {
  const double a = log((double)(1 - en)) / (double)un;
  return log(1 - e) / a;
}

// Emissivity of one corner of the cell: EGA intpol_tbl_eps(intpol_tbl_u(e) +
// du), CGA intpol_tbl_eps(du).  ef = round_down_f(e), the row's count and
// end entries come with the row record (EGA {u0, e0, en, n}, {un, ...}; CGA {n,
// ..., u0, e0}).  Slopes between entries are formed in
// single precision, as the reference's LIN macro does on floats.  Where the
// column u_eq + du stays in the bracket that inverts e, the emissivity
// follows from the entries already loaded.
template <bool CGA>
__device__ __forceinline__ double corner64(const TblDev& T, unsigned r, double e, float ef,
                                           double du, int& h, bool& ok) {
  const float2* row = T.ue + (size_t)r * (unsigned)T.tu;
  float u0, e0, un = 0.f, en = 0.f;
  int n;
  if (CGA) {
    const float4 m = __ldg(T.rowmeta + r);
    n = __float_as_int(m.x);
    u0 = m.z;
    e0 = m.w;
  } else {
    const float4 m = __ldg(T.rowmeta + 2 * (size_t)r);
    n = __float_as_int(m.w);
    un = __ldg(reinterpret_cast<const float*>(T.rowmeta + 2 * (size_t)r + 1));
    u0 = m.x;
    e0 = m.y;
    en = m.z;
  }
  const bool mono = !(n & kOddRow);
  n &= ~kOddRow;
  ok = n >= 2;
  if (!ok) return 0.0;
  // Both interpolations are y0 + (y1 - y0) / (x1 - x0) (x - x0): the lanes pick
  // the two entries apart (below the row: the origin and the first entry) and
  // interpolate together, so that divergence costs no FP64 instructions.
  double u = du;
  float2 lo = make_float2(0.f, 0.f), hi = lo;
  int ib = CGA ? h : 0;
  bool inside = false;  // lo, hi: the bracket that inverts e
  if (!CGA) {
    const bool up = above_f(e, ef, en);
    if (ef < e0) {
      hi = make_float2(u0, e0);
    } else if (!up) {
      const Pair64 k = find64<1>(row, n, ef, h, mono);
      ib = h = k.i;
      lo = k.a;
      hi = k.b;
      inside = mono;
    }
    u = f2d_bits(lo.x) + f2d_bits((hi.x - lo.x) / (hi.y - lo.y)) * (e - f2d_bits(lo.y)) + du;
    if (up) {
      u = u_above(un, en, e) + du;
      ib = n - 2;
    }
  }
  const float uf = round_down_f(u);
  bool up = false;
  if (!(inside && uf >= lo.x && uf < hi.x)) {
    if (uf < u0) {
      lo = make_float2(0.f, 0.f);
      hi = make_float2(u0, e0);
    } else {
      if (!CGA) up = above_f(u, uf, un);
      if (CGA && !mono) {
        const float2 last = __ldg(row + n - 1);
        up = above_f(u, uf, last.x);
        un = last.x;
        en = last.y;
      }
      if (!up) {
        const Pair64 k = find64<0>(row, n, uf, ib, mono);
        lo = k.a;
        hi = k.b;
        if (CGA) {
          h = k.i;
          un = hi.x;
          en = hi.y;
          up = mono && k.i == n - 2 && above_f(u, uf, un);
        }
      }
    }
  }
  if (up) return eps_above(un, en, u);
  return f2d_bits(lo.y) + f2d_bits((hi.y - lo.y) / (hi.x - lo.x)) * (u - f2d_bits(lo.x));
}

// ---------------------------------------------------------------------------
// the emitters' paths

template <bool CGA, int LPR>
__global__ void __launch_bounds__(128) k_gas64(CtlDev c, TblDev T, BatchDev b, LosDev L,
                                               Path64 P) {
  const int lane = threadIdx.x & 31;
  const int ng = c.ng, ndc = P.id1 - P.id0;
  long long w = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int idl = (int)(w % ndc);
  w /= ndc;
  const int g = (int)(w % ng);
  w /= ng;
  const int part8 = LPR == 4 ? (int)(w & 3) : 0;  // 8 of the tile's rays
  const int tl = (int)(LPR == 4 ? w >> 2 : w);
  if (tl >= P.tile1 - P.tile0) return;
  const int tile = P.tile0 + tl, id = P.id0 + idl;
  const long long dg = (long long)id * ng + g;
  const int np = T.np[dg];
  if (np < 30) return;  // no table: k_seg64 leaves this emitter out
  const int rl = LPR == 4 ? part8 * 8 + (lane >> 2) : lane;
  const int corner = lane & 3;
  int r = P.perm[tile * 32 + rl];
  if (r >= 0 && b.obs_skip && b.obs_skip[b.ray_obs[r]]) r = -1;
  if (r >= 0 && b.skip_masked && b.mask[(long long)id * b.nray + r]) r = -1;
  const int n = r >= 0 ? L.count[r] : 0;
  const int nmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
  const Fields64 F = fields64(c);
  const long long lp0 = P.toff[tile] - P.pt0;
  const double* fd = P.fd + (lp0 * F.nfd + F.g0 + kGas64 * g) * 32 + rl;
  const unsigned* fu = P.fu + (lp0 * F.nfu + 1 + g) * 32 + rl;
  double* out = P.om + ((lp0 * ndc + idl) * ng + g) * 32 + rl;
  const long long ostep = (long long)ndc * ng * 32;
  const bool cell = (P.shared >> g) & 1u;
  const unsigned rb = (unsigned)dg * (unsigned)(T.tp * T.tt);
  int h[4] = {0, 0, 0, 0};
  double tau = 1.0;
  int stop = n;
  // the next point's column and rows are loaded ahead of this point's chain
  double nu = 0;
  unsigned nrows = kNoCell;
  auto fetch = [&](int ip) {
    if (ip >= n) return;
    nu = fd[(long long)ip * F.nfd * 32];
    if (cell) nrows = fu[(long long)ip * F.nfu * 32];
  };
  fetch(0);
  for (int ip = 0; ip < nmax; ip++) {
    bool on = ip < n && stop == n;
    if (on && less_pos(tau, 1e-9)) {  // saturated from here on (the reference's tau_path < 1e-9)
      stop = ip;
      on = false;
    }
    if (!__any_sync(0xffffffffu, on)) break;
    const double du = nu;
    const unsigned rows = nrows;
    fetch(ip + 1);
    const double* f = fd + (long long)ip * F.nfd * 32;
    unsigned ra = 0, rc = 0;
    bool have = on, logp = false;
    Lin64 lp{}, la{}, lb{};
    if (on && cell) {
      have = rows != kNoCell;
      logp = rows & kLogP;
      ra = rb + (rows & 0x7fffu);
      rc = rb + (rows >> 16);
      if (LPR == 1 || (corner & 2) == 0) la = Lin64{f[4 * 32], f[5 * 32], f[6 * 32]};
      if (LPR == 1 || (corner & 2)) lb = Lin64{f[7 * 32], f[8 * 32], f[9 * 32]};
      lp = Lin64{f[1 * 32], f[2 * 32], f[3 * 32]};
    } else if (on) {
      const Cell64 k = cell64<CGA>(T, dg, np, f[1 * 32], f[2 * 32]);
      have = k.ra >= 0;
      logp = k.logp;
      ra = rb + (unsigned)k.ra;
      rc = rb + (unsigned)k.rc;
      lp = k.p;
      la = k.a;
      lb = k.b;
    }
    const double e = 1 - tau;  // the path's emissivity
    const float ef = CGA ? 0.f : round_down_f(e);
    bool ok = false;
    double ea = 0, eb = 0;
    if (LPR == 4) {
      double mine = 0.0;
      if (have)
        mine = corner64<CGA>(T, ((corner & 2) ? rc : ra) + (corner & 1), e, ef, du, h[0], ok);
      ok = ((__ballot_sync(0xffffffffu, ok) >> (lane & ~3)) & 15u) == 15u;
      const double ox = __shfl_xor_sync(0xffffffffu, mine, 1);
      const double lo = (corner & 1) ? ox : mine, hi = (corner & 1) ? mine : ox;
      const double et = lin64(lo, hi, (corner & 2) ? lb : la);
      const double oy = __shfl_xor_sync(0xffffffffu, et, 2);
      ea = (corner & 2) ? oy : et;
      eb = (corner & 2) ? et : oy;
    } else if (have) {
      bool k0, k1, k2, k3;
      const double e00 = corner64<CGA>(T, ra, e, ef, du, h[0], k0);
      const double e01 = corner64<CGA>(T, ra + 1, e, ef, du, h[1], k1);
      const double e10 = corner64<CGA>(T, rc, e, ef, du, h[2], k2);
      const double e11 = corner64<CGA>(T, rc + 1, e, ef, du, h[3], k3);
      ok = k0 && k1 && k2 && k3;
      ea = lin64(e00, e01, la);
      eb = lin64(e10, e11, lb);
    }
    double om = 1.0;  // segment transmittance 1 - eps
    if (ok) {
      const double v = CGA && logp ? ea + div_by((eb - ea) * lp.d, lp.w, lp.r) : lin64(ea, eb, lp);
      const double eps = 1 - (1 - clamp01(v)) / tau;
      om = 1 - eps;
    }
    if (on) {
      tau *= om;
      if (LPR == 1 || corner == 0) out[ip * ostep] = om;
    }
  }
  if (r >= 0 && (LPR == 1 || corner == 0))
    P.stop[((long long)(tl * ndc + idl) * ng + g) * 32 + rl] = stop;
}

// ---------------------------------------------------------------------------
// segments: src * eps and 1 - eps of every (point, channel)

__global__ void __launch_bounds__(128) k_seg64(CtlDev c, TblDev T, ChanDev ch, BatchDev b,
                                               LosDev L, Path64 P) {
  const int lane = threadIdx.x & 31;
  const int ng = c.ng, ndc = P.id1 - P.id0;
  const int nchb = (ndc + 3) / 4;
  const int idl = (int)(blockIdx.x % nchb) * 4 + (threadIdx.x >> 5);
  const int ip = (int)(blockIdx.x / nchb);
  const int tl = (int)blockIdx.y, tile = P.tile0 + tl;
  if (idl >= ndc) return;
  const int id = P.id0 + idl;
  const int r = P.perm[tile * 32 + lane];
  if (r < 0 || ip >= L.count[r]) return;
  const int o = b.ray_obs[r];
  if (b.obs_skip && b.obs_skip[o]) return;
  if (b.skip_masked && b.mask[(long long)id * b.nray + r]) return;
  const Fields64 F = fields64(c);
  const long long lp = P.toff[tile] - P.pt0 + ip;
  const double* fd = P.fd + lp * F.nfd * 32 + lane;
  double* se = P.se + (lp * ndc + idl) * 2 * 32 + lane;
  const double* om = P.om + (lp * ndc + idl) * ng * 32 + lane;
  const int* st = P.stop + (long long)(tl * ndc + idl) * ng * 32 + lane;
  double tau_gas = 1;
  for (int g = 0; g < ng; g++) {
    if (T.np[(long long)id * ng + g] < 30) continue;
    tau_gas = ip < st[g * 32] ? tau_gas * om[g * 32] : 0.0;
    if (tau_gas == 0) break;
  }
  if (!(tau_gas > 0)) {  // saturated: the segment adds nothing
    se[0] = 0.0;
    se[32] = 1.0;
    return;
  }
  const double* cc = ch.ctm + (long long)id * kCtmStride;
  const double ds = fd[F.ds * 32];
  double beta = c.nw > 0 ? fd[(F.kw0 + ch.window[id]) * 32] : 0.0;
  if (c.ncl > 0) {
    const double* s = b.scal + (long long)o * b.nscal;
    if (s[1] > 0) {
      const double nu = ch.nu[id];
      const int icl = bracket_irr(ch.clnu, c.ncl, nu);
      beta += fd[F.aux * 32] * lin(ch.clnu[icl], s[2 + icl], ch.clnu[icl + 1], s[2 + icl + 1], nu);
    }
  }
  if (c.ctm_co2 && c.ig_co2 >= 0 && cc[0] != 0) {
    const double* f = fd + F.co2 * 32;
    const double ctw = f[32] * cc[3] - f[64] * cc[2] + f[96] * cc[1];
    beta += div_by(f[0] * ctw, ds, fd[F.rds * 32]);
  }
  if (c.ctm_h2o && c.ig_h2o >= 0 && cc[4] != 0) {
    const double* f = fd + F.h2o * 32;
    const double nu = ch.nu[id], x = f[32], lc = cc[14];  // log(cc[6]), NaN: no logarithm
    const double self = cc[5] * (lc == lc ? pow_of_log(lc, cc[15], x) : pow(cc[6], x));
    beta = fma(nu * tanh(f[0] * nu), fma(f[64], self, f[96] * cc[7]), beta);
  }
  if ((c.ctm_n2 && cc[8] != 0) || (c.ctm_o2 && cc[11] != 0)) {
    const double* f = fd + F.n2 * 32;
    if (c.ctm_n2 && cc[8] != 0) beta = fma(f[64] * cc[9], exp(cc[10] * f[0]), beta);
    if (c.ctm_o2 && cc[11] != 0) beta = fma(f[32] * (0.21 * cc[12]), exp(cc[13] * f[0]), beta);
  }
  const unsigned it = P.fu[lp * F.nfu * 32 + lane];
  // source function: value and slope of the table interval
  const double2 sv = T.srd[(long long)id * kNS + it];
  const double src = sv.x + sv.y * fd[F.ws * 32];
  const double eps = 1 - tau_gas * exp(-beta * ds);
  se[0] = src * eps;
  se[32] = 1 - eps;
}

// ---------------------------------------------------------------------------
// radiance: the sums along the path, then surface emission, reflection and
// solar term (jurassic.c:3264-3328), BT conversion and mask (3026-3071)

__global__ void __launch_bounds__(128) k_scan64(CtlDev c, TblDev T, ChanDev ch, BatchDev b,
                                                LosDev L, Path64 P) {
  const int lane = threadIdx.x & 31;
  const int ng = c.ng, ndc = P.id1 - P.id0;
  const long long w = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int idl = (int)(w % ndc);
  const int tl = (int)(w / ndc);
  if (tl >= P.tile1 - P.tile0) return;
  const int tile = P.tile0 + tl, id = P.id0 + idl;
  const int r = P.perm[tile * 32 + lane];
  if (r < 0) return;
  const int o = b.ray_obs[r];
  if (b.obs_skip && b.obs_skip[o]) return;
  const long long nray = b.nray, oi = (long long)id * nray + r;
  int n = b.skip_masked && b.mask[oi] ? 0 : L.count[r];
  const int* st = P.stop + (long long)(tl * ndc + idl) * ng * 32 + lane;
  for (int g = 0; g < ng; g++)  // past the first saturated emitter nothing adds
    if (n > 0 && T.np[(long long)id * ng + g] >= 30) n = min(n, st[g * 32]);
  const long long lp0 = P.toff[tile] - P.pt0;
  const double* se = P.se + (lp0 * ndc + idl) * 2 * 32 + lane;
  const long long step = (long long)ndc * 2 * 32;
  double rad = 0, tau = 1;
  constexpr int U = 8;  // loads in flight ahead of the sums
  int ip = 0;
  for (; ip + U <= n; ip += U) {
    double v[U], m[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      v[k] = se[(ip + k) * step];
      m[k] = se[(ip + k) * step + 32];
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      rad += v[k] * tau;
      tau *= m[k];
    }
  }
  for (; ip < n; ip++) {
    rad += se[ip * step] * tau;
    tau *= se[ip * step + 32];
  }
  const double nu = ch.nu[id];
  const double sft = L.sft[r];
  if (c.sftype >= 1 && sft > 0) {
    double sfeps = 1.0;
    if (c.nsf > 0) {
      const double* s = b.scal + (long long)o * b.nscal + 5 + c.ncl;
      const int isf = bracket_irr(ch.sfnu, c.nsf, nu);
      sfeps = lin(ch.sfnu[isf], s[isf], ch.sfnu[isf + 1], s[isf + 1], nu);
    }
    const int it = bracket_reg(T.st, kNS, sft);
    rad += sfeps * lin(T.st[it], T.sr[(long long)it * c.nd + id], T.st[it + 1],
                       T.sr[(long long)(it + 1) * c.nd + id], sft) * tau;
    if (c.sftype >= 2 && sfeps < 1) {
      double tau_refl = 1;
      for (ip = n - 1; ip >= 0; ip--) {
        rad += se[ip * step] * tau_refl * tau * (1 - sfeps);
        tau_refl *= se[ip * step + 32];
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
  if (c.fov) {  // pencil beam only: FOV convolution, BT and mask follow in k_fov
    b.rad[oi] = rad;
    b.tau[oi] = tau;
    return;
  }
  if (c.write_bbt) rad = kC2 * nu / log1p(kC1 * (nu * nu * nu) / rad);
  b.rad[oi] = b.mask[oi] ? __longlong_as_double(0x7ff8000000000000LL) : rad;
  b.tau[oi] = tau;
}

// source function, channel-major: value and slope (the division of LIN) of
// every interval
__global__ void k_src_channel_major(int nd, const double* st, const double* sr, double2* srd) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nd * kNS) return;
  const int it = gid % kNS, id = gid / kNS;
  const double s0 = sr[(long long)it * nd + id];
  const double s1 = it + 1 < kNS ? sr[(long long)(it + 1) * nd + id] : s0;
  srd[gid] = make_double2(s0, it + 1 < kNS ? (s1 - s0) / (st[it + 1] - st[it]) : 0.0);
}

}  // namespace

void path64_point_bytes(const CtlDev& c, size_t* fd, size_t* fu) {
  const Fields64 F = fields64(c);
  *fd = sizeof(double) * 32 * (size_t)F.nfd;
  *fu = sizeof(unsigned) * 32 * (size_t)F.nfu;
}

void launch_src_channel_major(int nd, const double* st, const double* sr, double2* srd,
                              cudaStream_t s) {
  k_src_channel_major<<<(nd * kNS + 255) / 256, 256, 0, s>>>(nd, st, sr, srd);
}

void launch_prep64(const CtlDev& c, const TblDev& T, const LosDev& L, const Path64& P,
                   int longest, cudaStream_t s) {
  const dim3 grid((unsigned)((longest + 3) / 4), (unsigned)(P.tile1 - P.tile0));
  if (c.formod == 0)
    k_prep64<true><<<grid, 128, 0, s>>>(c, T, L, P);
  else
    k_prep64<false><<<grid, 128, 0, s>>>(c, T, L, P);
}

void launch_path64(const CtlDev& c, const TblDev& T, const ChanDev& ch, const BatchDev& b,
                   const LosDev& L, const Path64& P, int longest, int lanes_per_ray,
                   cudaStream_t s) {
  const long long nt = P.tile1 - P.tile0, ndc = P.id1 - P.id0;
  if (c.ng > 0) {
    const long long warps = nt * ndc * c.ng * (lanes_per_ray == 4 ? 4 : 1);
    const unsigned nblk = (unsigned)((warps + 3) / 4);
    if (c.formod == 0) {
      if (lanes_per_ray == 4) k_gas64<true, 4><<<nblk, 128, 0, s>>>(c, T, b, L, P);
      else k_gas64<true, 1><<<nblk, 128, 0, s>>>(c, T, b, L, P);
    } else {
      if (lanes_per_ray == 4) k_gas64<false, 4><<<nblk, 128, 0, s>>>(c, T, b, L, P);
      else k_gas64<false, 1><<<nblk, 128, 0, s>>>(c, T, b, L, P);
    }
  }
  const long long nchb = (ndc + 3) / 4;
  k_seg64<<<dim3((unsigned)(nchb * longest), (unsigned)nt), 128, 0, s>>>(c, T, ch, b, L, P);
  k_scan64<<<(unsigned)((nt * ndc + 3) / 4), 128, 0, s>>>(c, T, ch, b, L, P);
}

}  // namespace jgb
