// Mixed-precision forward model: FP32 path loop with compensated sums.
//
// Work decomposition: rays are sorted by LOS length and grouped into tiles
// of 32 (one ray per lane), so all lanes of a warp read the same emissivity
// table (same channel, emitter) at neighbouring rows and the same LOS plane
// entries (one 128-byte line per field and point).  A batch runs through
// three kernels: k_gas_m walks the points for one (tile, channel, emitter)
// per warp, k_seg_m joins the emitters' segments of every (point, channel)
// with the continua, k_scan_m sums them along the rays.  Resumed
// finite-difference perturbations start in the middle of a path, from the
// states that their base rays saved there.
//
// Numerics (same algorithm as intpol_tbl_ega/cga, jurassic.c:3710-3891, and
// formod_pencil, 3196-3338):
//  * each (channel, emitter) carries its path transmittance t and path
//    emissivity e = 1 - t as two floats, each accurate where it is small,
//    so that neither 1 - t nor 1 - e is ever formed from a rounded value;
//  * segment emissivities are combined as E <- E + (1 - E) eps_g (no
//    cancellation for small eps), the continuum as -expm1(-beta ds);
//  * the radiance sum is Kahan-compensated.
#include <type_traits>

#include "jgb_common.cuh"
#include "jgb_internal.h"

namespace jgb {

// Field indices of a tile plane: the point's p, t, ds, q_H2O and cloud
// factor, the extinction per window, then one block of kEmitterFields(CGA)
// fields per emitter, emitter g's at g0 + g * es + k (k constant, so that a
// warp addresses them from one base):
//   EGA: u, {br, pw, wa, wb};  CGA: u, cgp, cgt, cgu, {br, pw, wa, wb},
// the braces 16 bytes per lane (one load).
// For emitters whose p-T grids are shared by all channels, the
// channel-independent part of the table interpolation is done once per LOS
// point: br holds the rows of the point's p-T cell within a (channel,
// emitter) table, ipr * tt + it0 | ((ipr + 1) * tt + it1) << 16
// (kNoBracket: no table, kNoBracket | 2: no temperature rows at that
// pressure; tp * tt < 2^15), pw the pressure interpolation weight in that
// bracket (linear in EGA, log-linear in CGA), wa and wb the temperature
// weights at the lower and upper pressure of the bracket.
struct Fields {
  int p, t, ds, qh2o, aux, kw0, g0, es, n;
};
constexpr int kFU = 0;  // column of the segment (EGA) / of the path (continua)
constexpr int kFCgp = 1, kFCgt = 2, kFCgu = 3;  // CGA means
__host__ __device__ constexpr int kEmitterFields(bool cga) { return cga ? 8 : 5; }
__host__ __device__ constexpr int kFBr(bool cga) { return cga ? 4 : 1; }  // then pw, wa, wb

__host__ __device__ inline Fields fields_of(const CtlDev& c) {
  Fields f;
  f.p = 0;
  f.t = 1;
  f.ds = 2;
  f.qh2o = 3;
  f.aux = 4;
  f.kw0 = 5;
  f.g0 = 5 + c.nw;
  f.es = kEmitterFields(c.formod == 0);
  f.n = f.g0 + c.ng * f.es;
  return f;
}

int mixed_nfield(const CtlDev& c) { return fields_of(c).n; }

constexpr unsigned kNoBracket = 0x80000000u;

// ---------------------------------------------------------------------------
// float table access with hinted searches
//
// Along a path the column density of every (channel, emitter) only grows
// and pressure/temperature change slowly, so the bracket found at one LOS
// point is almost always the bracket (or its neighbour) at the next point.
// Each search therefore first tests the remembered bracket and the next one
// with independent loads (one round trip) and falls back to bisection
// only on a miss.  Any valid bracket gives the same interpolated value, so
// the result does not depend on the hint.

// Row r = (dg * tp + ip) * tt + it from its record; 32-bit row arithmetic
// (the table upload checks that rows x TU < 2^32).  EGA records are 32
// bytes, {u[0], eps[0], eps[n-1], n} and {u[n-1], a, 0, 0}, where a = log(1 -
// eps[n-1]) / u[n-1]: the first half places the path emissivity against the
// row before any search (it starts below the rows and saturates above them),
// the second is read where a column leaves the row.  CGA records are 16
// bytes, {n, 0, u[0], eps[0]}: a column above a row brackets at n-2, and the
// search brings the row's last entries.
// kOddRow in n marks a row that falls somewhere or whose columns reach 2^125:
// such rows take corner_odd (full-range divisions, no assumption on the
// order), the others divide by __fdividef, which gives the bits of the
// full-range division for divisors below 2^126 in a quarter of its
// instructions.
// Where results of several kernels must agree to the bit, sums of products
// name their fused form; left to the compiler it depends on the block that a
// value is used in.

// A bracket index i with the grid values at i and i + 1.
struct Bracket {
  int i;
  float a, b;
};

// Bracket i of x in component C (0: u, 1: eps) of an interleaved ascending
// row of n entries with C[0] <= x <= C[n-1], from hint h (locate_tbl
// semantics, jurassic.c:4152-4170), with both components at i and i + 1
// (reused from the probe loads on a hit).
struct Bracket2 {
  int i;
  float2 a, b;
};

template <int C>
__device__ __forceinline__ float comp(const float2 v) {
  return C == 0 ? v.x : v.y;
}

template <int C>
__device__ __forceinline__ int bisect2(const float2* g, int lo, int hi, float x) {
  const float* gc = reinterpret_cast<const float*>(g) + C;
  while (hi > lo + 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(gc + 2 * mid) > x) hi = mid; else lo = mid;
  }
  return lo;
}

// The third probe g[h+2] is read even where h + 2 = n (the next row's first
// entry, or the one-entry pad after the last row) and then ignored.
template <int C>
__device__ __forceinline__ Bracket2 hunt2(const float2* g, int n, float x, int h) {
  h = min(h, n - 2);
  const float2 A = __ldg(g + h), B = __ldg(g + h + 1), D = __ldg(g + h + 2);
  const float a = comp<C>(A), b = comp<C>(B), c = comp<C>(D);
  // bracket h or h + 1: every x >= a when the probes reach the row's end
  // (h >= n - 3; x at or above g[n-1] keeps n - 2, and h + 1 <= n - 2 is the
  // last bracket there), else x < g[h+2]
  const bool tail = h + 2 >= n - 1;
  if (a <= x && (x < c || tail)) {
    const bool up = x >= b && h + 2 < n;
    return up ? Bracket2{h + 1, B, D} : Bracket2{h, A, B};
  }
  const int i = a <= x ? bisect2<C>(g, h + 2, n - 1, x) : bisect2<C>(g, 0, h, x);
  return Bracket2{i, __ldg(g + i), __ldg(g + i + 1)};
}

// Emissivity between the entries a and b {u, eps} at column u (LIN).
__device__ __forceinline__ float between(float2 a, float2 b, float u) {
  return __fmaf_rn(__fdividef(__fsub_rn(b.y, a.y), __fsub_rn(b.x, a.x)), __fsub_rn(u, a.x), a.y);
}

// Emissivity of one table row (corner of the p-T cell) for the extended
// path: EGA u = intpol_tbl_u(e_path) + du, CGA u = ucg; then
// intpol_tbl_eps(u) (jurassic.c:3799-3891, 3895-3967).  In EGA the bracket
// that inverts e_path also brackets u_eq in the column row (the rows are
// monotone), and u_eq + du usually stays inside it: then the emissivity is
// interpolated from the entries already loaded, with no second search.
// The bracket is the same either way, so the value is too.  h is the
// search hint carried along the path: of the emissivity-row search in EGA,
// of the column-row search in CGA (EGA's column search starts from the
// emissivity bracket, or from the row start below the table).  m: the first
// half of the row's record.
template <bool CGA>
__device__ __forceinline__ float corner_eps(const TblDev& T, unsigned r, const float4 m,
                                            float e_path, float du, float ucg,
                                            int& h) {
  const float2* row = T.ue + r * (unsigned)T.tu;
  if (CGA) {  // intpol_tbl_eps(ucg), the row's last entries from the search
    const int n = __float_as_int(m.x);
    const float uc = ucg;
    if (uc < m.z) return __fdividef(m.w, m.z) * uc;
    const Bracket2 k = hunt2<0>(row, n, uc, h);
    h = k.i;
    if (uc > k.b.x) {
      const float a = __fdividef(log1pf(-k.b.y), k.b.x);
      return -expm1f(a * uc);
    }
    return between(k.a, k.b, uc);
  }
  const float2* rec = reinterpret_cast<const float2*>(T.rowmeta + 2 * r + 1);  // {u[n-1], a}
  const int n = __float_as_int(m.w);
  float uq;
  int ib = 0;
  if (e_path < m.y) {
    uq = __fadd_rn(__fmul_rn(__fdividef(m.x, m.y), e_path), du);
    if (uq < m.x) return __fdividef(m.y, m.x) * uq;
  } else if (e_path > m.z) {
    uq = __fadd_rn(__fdividef(log1pf(-e_path), __ldg(rec).y), du);
  } else {
    const Bracket2 k = hunt2<1>(row, n, e_path, h);
    h = k.i;
    ib = k.i;
    uq = __fadd_rn(__fmaf_rn(__fdividef(__fsub_rn(k.b.x, k.a.x), __fsub_rn(k.b.y, k.a.y)),
                             __fsub_rn(e_path, k.a.y), k.a.x), du);
    if (uq >= k.a.x && uq < k.b.x)
      return between(k.a, k.b, uq);
  }
  if (uq < m.x) return __fdividef(m.y, m.x) * uq;
  const float2 top = __ldg(rec);
  if (uq > top.x) return -expm1f(top.y * uq);
  const Bracket2 k = hunt2<0>(row, n, uq, ib);
  return between(k.a, k.b, uq);
}

// The same for a row marked kOddRow; the hint comes and goes by value (a
// pointer to it would keep the hints of every row in local memory).
struct OddCorner {
  float e;
  int h;
};
template <bool CGA>
__device__ __noinline__ OddCorner corner_odd(const float2* row, int n, float e_path, float du,
                                             float ucg, int h) {
  n &= ~kOddRow;
  const float2 first = __ldg(row), last = __ldg(row + n - 1);
  if (CGA) {
    if (ucg < first.x) return OddCorner{first.y / first.x * ucg, h};
    const Bracket2 k = hunt2<0>(row, n, ucg, h);
    if (ucg > k.b.x) {
      const float a = log1pf(-k.b.y) / k.b.x;
      return OddCorner{-expm1f(a * ucg), k.i};
    }
    return OddCorner{k.a.y + (k.b.y - k.a.y) / (k.b.x - k.a.x) * (ucg - k.a.x), k.i};
  }
  float uq, u_lo = 0.f, u_hi = 0.f, e_lo = 0.f, e_hi = 0.f;
  int ib = -1;
  if (e_path < first.y) {
    uq = __fmul_rn(first.x / first.y, e_path);
  } else if (e_path > last.y) {
    const float a = log1pf(-last.y) / last.x;
    uq = log1pf(-e_path) / a;
  } else {
    const Bracket2 k = hunt2<1>(row, n, e_path, h);
    h = ib = k.i;
    e_lo = k.a.y;
    e_hi = k.b.y;
    u_lo = k.a.x;
    u_hi = k.b.x;
    uq = u_lo + (u_hi - u_lo) / (e_hi - e_lo) * (e_path - e_lo);
  }
  uq = __fadd_rn(uq, du);
  if (uq < first.x) return OddCorner{first.y / first.x * uq, h};
  if (uq > last.x) {
    const float a = log1pf(-last.y) / last.x;
    return OddCorner{-expm1f(a * uq), h};
  }
  if (ib >= 0 && uq >= u_lo && uq < u_hi)
    return OddCorner{e_lo + (e_hi - e_lo) / (u_hi - u_lo) * (uq - u_lo), h};
  const Bracket2 k = hunt2<0>(row, n, uq, max(ib, 0));
  return OddCorner{k.a.y + (k.b.y - k.a.y) / (k.b.x - k.a.x) * (uq - k.a.x), h};
}

// One corner of the cell from its record, whichever kind of row it is.  FAST
// kernels run where no row is odd and every emitter's grids are shared by all
// channels: the calls and the search for the cell cost registers even where
// they are not taken.
template <bool CGA, bool FAST>
__device__ __forceinline__ float corner_any(const TblDev& T, unsigned r, const float4 m, int n,
                                            float e_path, float du, float ucg,
                                            int& h) {
  if (!FAST && (n & kOddRow)) {
    const OddCorner o = corner_odd<CGA>(T.ue + r * (unsigned)T.tu, n, e_path, du, ucg, h);
    h = o.h;
    return o.e;
  }
  return corner_eps<CGA>(T, r, m, e_path, du, ucg, h);
}

__device__ __forceinline__ int bracket_regf(const float* g, int n, float x) {
  const float g0 = __ldg(g), g1 = __ldg(g + 1);
  const int i = (int)((x - g0) / (g1 - g0));
  return i < 0 ? 0 : (i > n - 2 ? n - 2 : i);
}

__device__ __forceinline__ int bracket_irrf(const float* g, int n, float x) {
  int lo = 0, hi = n - 1, mid = (lo + hi) >> 1;
  const bool up = __ldg(g + mid) < __ldg(g + mid + 1);
  while (hi > lo + 1) {
    mid = (lo + hi) >> 1;
    const float v = __ldg(g + mid);
    const bool go_low = up ? (v > x) : (v <= x);
    if (go_low) hi = mid; else lo = mid;
  }
  return lo;
}

// One thread per (tile, point, lane) converts the FP64 LOS to float tiles.
__global__ void k_pack_tiles(CtlDev c, TblDev T, LosDev L, MixedPlan P, long long total) {
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= total * 32) return;
  const int lane = (int)(gid & 31);
  const long long tp = gid >> 5;  // tile-point
  // locate the tile by binary search over tile offsets
  int lo = 0, hi = P.ntile;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (P.toff[mid] <= tp) lo = mid; else hi = mid;
  }
  const int tile = lo;
  const int ip = (int)(tp - P.toff[tile]);
  const int r = P.perm[tile * 32 + lane];
  const Fields F = fields_of(c);
  float* out = P.data + tp * (long long)F.n * 32 + lane;
  if (r < 0 || ip >= L.count[r] || (P.start && ip < P.start[r])) return;  // never read
  const long long q = L.off[r] + ip;
  const LosDev::F32& Lf = L.f;
  out[F.p * 32] = Lf.p[q];
  out[F.t * 32] = Lf.t[q];
  out[F.ds * 32] = Lf.ds[q];
  out[F.qh2o * 32] = c.ig_h2o >= 0 ? Lf.qh2o[q] : 0.f;
  out[F.aux * 32] = Lf.aux[q];
  for (int w = 0; w < c.nw; w++) out[(F.kw0 + w) * 32] = Lf.kw[w * L.cap + q];
  const bool cgaf = c.formod == 0;
  for (int g = 0; g < c.ng; g++) {
    float* og = out + (F.g0 + g * F.es) * 32;
    og[kFU * 32] = Lf.u[g * L.cap + q];
    if (cgaf) {
      og[kFCgp * 32] = Lf.cgp[g * L.cap + q];
      og[kFCgt * 32] = Lf.cgt[g * L.cap + q];
      og[kFCgu * 32] = Lf.cgu[g * L.cap + q];
    }
  }
  // p-T brackets and interpolation weights on the grids of channel 0
  // (identical for every channel)
  for (int g = 0; P.brmask && g < c.ng; g++) {
    unsigned wd = kNoBracket;  // no table (np < 30)
    float pw = 0.f, wa = 0.f, wb = 0.f;
    const int np = __ldg(T.np + g);
    if (((P.brmask >> g) & 1u) && np >= 30) {
      const float pq = c.formod == 0 ? Lf.cgp[g * L.cap + q] : Lf.p[q];
      const float tq = c.formod == 0 ? Lf.cgt[g * L.cap + q] : Lf.t[q];
      const int ipr = bracket_irrf(T.pf + (long long)g * T.tp, np, pq);
      const int nt0 = __ldg(T.nt + (long long)g * T.tp + ipr);
      const int nt1 = __ldg(T.nt + (long long)g * T.tp + ipr + 1);
      wd = kNoBracket | 2u;      // temperature rows missing at this pressure
      if (nt0 >= 2 && nt1 >= 2) {
        const float* t0g = T.tf + ((long long)g * T.tp + ipr) * T.tt;
        const int it0 = bracket_regf(t0g, nt0, tq);
        const int it1 = bracket_regf(t0g + T.tt, nt1, tq);
        wd = (unsigned)(ipr * T.tt + it0) | ((unsigned)((ipr + 1) * T.tt + it1) << 16);
        // temperature weights at both pressures (LIN in T of
        // intpol_tbl_ega / intpol_tbl_cga)
        wa = (tq - t0g[it0]) / (t0g[it0 + 1] - t0g[it0]);
        wb = (tq - t0g[T.tt + it1]) / (t0g[T.tt + it1 + 1] - t0g[T.tt + it1]);
        // pressure weight: linear in EGA, log-linear in CGA
        const float* pg = T.pf + (long long)g * T.tp;
        const float pa = pg[ipr], pb = pg[ipr + 1];
        if (c.formod == 0 && pq / pa > 0.f && pb / pa > 0.f)
          pw = __logf(pq / pa) / __logf(pb / pa);
        else
          pw = (pq - pa) / (pb - pa);
      }
    }
    float* og = P.data + (tp * F.n + F.g0 + g * F.es + kFBr(cgaf)) * 32;
    reinterpret_cast<float4*>(og)[lane] = make_float4(__uint_as_float(wd), pw, wa, wb);
  }
}

// Pressure bracket with a hint: keeps ipr while p lies inside its interval
// (or beyond the grid end it is clamped to), else bisects; with the grid
// values at ipr and ipr + 1.
__device__ __forceinline__ Bracket pbracket_f(const float* g, int n, float x, int ipr) {
  if (ipr >= 0) {
    const float a = __ldg(g + ipr), b = __ldg(g + ipr + 1);
    const float lo = fminf(a, b), hi = fmaxf(a, b);
    const bool low_end = (ipr == 0) && ((a < b) ? (x < a) : (x > a));
    const bool high_end = (ipr == n - 2) && ((a < b) ? (x >= b) : (x <= b));
    if ((x >= lo && x < hi) || low_end || high_end) return Bracket{ipr, a, b};
  }
  const int i = bracket_irrf(g, n, x);
  return Bracket{i, __ldg(g + i), __ldg(g + i + 1)};
}

constexpr int kStateWords = 5;  // t, e, ipr, 2 words of 16-bit corner hints
constexpr float kTauStop = 1e-12f;  // path transmittance below which the walk stops
constexpr int kChanConsts = 16;  // constants of a warp's channel
constexpr int kPathThreads = 128;  // threads of a path block

// Per (channel, emitter) state carried along the path: transmittance t and
// emissivity e of the extended path (each accurate where it is small), the
// pressure bracket and the search hints of the four table corners (below 2^16).
struct GasState {
  float t, e;
  int ipr;
  int h[4];
};

// Interpolations of the cell's corners in temperature and pressure.
__device__ __forceinline__ float mix_f(float y0, float y1, float w) {
  return __fmaf_rn(__fsub_rn(y1, y0), w, y0);
}

// The path's emissivity becomes e: the segment's emissivity; *sat is set where
// the reference's segment transmittance becomes zero.
__device__ __forceinline__ float extend_f(float e, GasState& s, bool& sat) {
  e = fminf(fmaxf(e, 0.f), 1.f);
  const float te = __fsub_rn(1.f, e);  // exact for e >= 0.5
  const float rt = __fdividef(1.f, s.t);
  const float eps = (s.e < 0.5f) ? __fmul_rn(__fsub_rn(e, s.e), rt) : __fmaf_rn(-te, rt, 1.f);
  if (e >= 1.f) sat = true;
  s.t = te;
  s.e = e;
  return eps;
}

// The p-T cell of one LOS point in table dg: rows ra, ra + 1 at the lower
// pressure, rc, rc + 1 at the upper one, and the weights in pressure (w) and
// temperature (a, b).
struct CellF {
  unsigned ra, rc;
  float w, a, b;
  bool ok;
};

// From the precomputed words (grids shared by all channels) ...
__device__ __forceinline__ float4 cell_words(const float* block, int lane) {
  return reinterpret_cast<const float4*>(block - lane)[lane];
}
__device__ __forceinline__ float4 no_cell() {
  return make_float4(__uint_as_float(kNoBracket | 1u), 0.f, 0.f, 0.f);
}
__device__ __forceinline__ CellF cell_packed(const TblDev& T, long long dg, const float4 cw) {
  const unsigned rb = (unsigned)dg * (unsigned)(T.tp * T.tt), brw = __float_as_uint(cw.x);
  return CellF{rb + (brw & 0xffffu), rb + (brw >> 16), cw.y, cw.z, cw.w, (brw & kNoBracket) == 0u};
}

// ... or found here, the pressure bracket from the last one (ipr).  The
// temperature interpolation is then e00 + (e01 - e00) / (t1 - t0) (t - t0).
struct CellFind {
  CellF k;
  float ta, tb, tc, td;
};
template <bool CGA>
__device__ __forceinline__ CellFind cell_find(const TblDev& T, long long dg, int np, float pq,
                                              float tq, int& ipr) {
  CellFind f{};
  const Bracket pb = pbracket_f(T.pf + dg * T.tp, np, pq, ipr);
  ipr = pb.i;
  const int* ntg = T.nt + dg * T.tp;
  const int nt0 = __ldg(ntg + ipr), nt1 = __ldg(ntg + ipr + 1);
  if (nt0 < 2 || nt1 < 2) return f;
  const int it0 = bracket_regf(T.tf + (dg * T.tp + ipr) * T.tt, nt0, tq);
  const int it1 = bracket_regf(T.tf + (dg * T.tp + ipr + 1) * T.tt, nt1, tq);
  const unsigned rp = (unsigned)dg * (unsigned)T.tp + (unsigned)ipr;
  f.k.ra = rp * (unsigned)T.tt + (unsigned)it0;
  f.k.rc = (rp + 1u) * (unsigned)T.tt + (unsigned)it1;
  f.k.ok = true;
  f.ta = __ldg(T.tf + f.k.ra);
  f.tb = __ldg(T.tf + f.k.ra + 1);
  f.tc = __ldg(T.tf + f.k.rc);
  f.td = __ldg(T.tf + f.k.rc + 1);
  if (CGA && pq / pb.a > 0.f && pb.b / pb.a > 0.f)
    f.k.w = __logf(pq / pb.a) / __logf(pb.b / pb.a);
  else
    f.k.w = (pq - pb.a) / (pb.b - pb.a);
  return f;
}

// Temperature interpolation with the division in place.
__device__ __forceinline__ float mix_t(float y0, float y1, float t0, float t1, float t) {
  return __fmaf_rn(__fsub_rn(y1, y0) / __fsub_rn(t1, t0), __fsub_rn(t, t0), y0);
}

template <bool CGA>
__device__ __forceinline__ float4 row_record(const TblDev& T, unsigned r) {
  return __ldg(T.rowmeta + (CGA ? r : 2 * r));
}
template <bool CGA>
__device__ __forceinline__ int row_count(const float4 m) {
  return __float_as_int(CGA ? m.x : m.w);
}

// One (channel, emitter) at one LOS point (intpol_tbl_ega / intpol_tbl_cga,
// jurassic.c:3710-3891).  Returns the segment emissivity; *sat is set where
// the reference's segment transmittance becomes zero.
// cw: the cell's rows and interpolation weights precomputed for the LOS point
// (grids shared by all channels), or no_cell() to search here.
template <bool CGA, bool FAST>
__device__ __forceinline__ float gas_eps_f(const TblDev& T, long long dg, float pq,
                                           float tq, float du, float ucg, const float4 cw,
                                           GasState& s, bool& sat) {
  const unsigned brw = __float_as_uint(cw.x);
  const float wta = cw.z, wtb = cw.w;
  const bool pre = FAST || brw != (kNoBracket | 1u);
  if (pre && brw == kNoBracket) return 0.f;   // np < 30
  int np = 0;
  if (!pre) {
    np = __ldg(T.np + dg);
    if (np < 30) return 0.f;
  }
  if (s.t < 1e-9f) {
    s.t = 0.f;
    s.e = 1.f;
    sat = true;
    return 1.f;
  }
  CellFind f{};
  if (pre) f.k = cell_packed(T, dg, cw);
  else f = cell_find<CGA>(T, dg, np, pq, tq, s.ipr);
  if (!f.k.ok) return 0.f;                    // nt < 2 at this pressure
  const unsigned ra = f.k.ra, rc = f.k.rc;
  // one pressure's pair of rows after the other (four records at a time cost
  // more registers than their overlap gains)
  float ea, eb;
  {
    const float4 m0 = row_record<CGA>(T, ra), m1 = row_record<CGA>(T, ra + 1u);
    const int n0 = row_count<CGA>(m0), n1 = row_count<CGA>(m1);
    if (min(n0, n1) < 2) return 0.f;
    const float e0 = corner_any<CGA, FAST>(T, ra, m0, n0, s.e, du, ucg, s.h[0]);
    const float e1 = corner_any<CGA, FAST>(T, ra + 1u, m1, n1, s.e, du, ucg, s.h[1]);
    ea = pre ? mix_f(e0, e1, wta) : mix_t(e0, e1, f.ta, f.tb, tq);
  }
  {
    const float4 m0 = row_record<CGA>(T, rc), m1 = row_record<CGA>(T, rc + 1u);
    const int n0 = row_count<CGA>(m0), n1 = row_count<CGA>(m1);
    if (min(n0, n1) < 2) return 0.f;
    const float e0 = corner_any<CGA, FAST>(T, rc, m0, n0, s.e, du, ucg, s.h[2]);
    const float e1 = corner_any<CGA, FAST>(T, rc + 1u, m1, n1, s.e, du, ucg, s.h[3]);
    eb = pre ? mix_f(e0, e1, wtb) : mix_t(e0, e1, f.tc, f.td, tq);
  }
  return extend_f(mix_f(ea, eb, f.k.w), s, sat);
}

// Per-channel constants of the path in FP32 (chanf[id * kChanConsts]): nu,
// CO2 296/260/230 K, H2O 296 K, log of its 260/296 K ratio, foreign, N2 B and
// beta, O2 B and beta, then the continua of the channel as bits (1 CO2, 2 H2O,
// 4 N2, 8 O2) and the window.
constexpr int kChanSwitches = 11, kChanWindow = 12;

__global__ void k_chan_consts(CtlDev c, ChanDev ch, float* out) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= c.nd) return;
  const double* cc = ch.ctm + (long long)id * kCtmStride;
  float* k = out + id * kChanConsts;
  k[0] = (float)ch.nu[id];
  k[1] = (float)cc[1];
  k[2] = (float)cc[2];
  k[3] = (float)cc[3];
  k[4] = (float)cc[5];
  k[5] = (float)log(cc[6] > 0 ? cc[6] : 1.0);
  k[6] = (float)cc[7];
  k[7] = (float)cc[9];
  k[8] = (float)cc[10];
  k[9] = (float)cc[12];
  k[10] = (float)cc[13];
  const int on = (c.ig_co2 >= 0 && cc[0] != 0 ? 1 : 0) | (c.ig_h2o >= 0 && cc[4] != 0 ? 2 : 0) |
                 (cc[8] != 0 ? 4 : 0) | (cc[11] != 0 ? 8 : 0);
  k[kChanSwitches] = __int_as_float(on);
  k[kChanWindow] = __int_as_float(c.nw > 0 ? ch.window[id] : 0);
}

// The channel's continua that the control set has on.
__device__ __forceinline__ int continua_on(const CtlDev& c, float bits) {
  return __float_as_int(bits) & ((c.ctm_co2 ? 1 : 0) | (c.ctm_h2o ? 2 : 0) | (c.ctm_n2 ? 4 : 0) |
                                 (c.ctm_o2 ? 8 : 0));
}

// Extinction of a segment by the continua (ctmco2, ctmh2o, ctmn2, ctmo2)
// added to beta; kc: the channel's constants, f: the point's fields.
template <typename K>
__device__ __forceinline__ float continua_f(const CtlDev& c, const Fields& F, K kc, int on,
                                            const float* f, float p, float t, float ds,
                                            float beta) {
  const float pr = p / (float)kP0;
  if (on & 1) {
    const float co2_296 = kc[1], co2_260 = kc[2], co2_230 = kc[3];
    const float d230 = t - 230.f, d260 = t - 260.f, d296 = t - 296.f;
    const float ctw = d260 * 5.050505e-4f * d296 * co2_230 - d230 * 9.259259e-4f * d296 * co2_260 +
                      d230 * 4.208754e-4f * d260 * co2_296;
    const float uco2 = f[(F.g0 + c.ig_co2 * F.es + kFU) * 32];
    beta += __fdividef(uco2, ds) * (float)(1.0 / (kNA * 1000.0)) * pr * ctw;
  }
  if (on & 2) {
    const float q = f[F.qh2o * 32];
    const float uh = f[(F.g0 + c.ig_h2o * F.es + kFU) * 32];
    const float nu = kc[0], h2o_s296 = kc[4], h2o_lr = kc[5], h2o_frn = kc[6];
    const float self = h2o_s296 * __expf(h2o_lr * (296.f - t) * (1.f / 36.f));
    const float a1 = nu * (__fdividef(uh, ds) * 1e-20f) * tanhf(__fdividef(.7193876f, t) * nu);
    beta += a1 * __fdividef(296.f, t) * pr * (q * self + (1.f - q) * h2o_frn);
  }
  if (on & 12) {
    const float n2_b = kc[7], n2_beta = kc[8], o2_b = kc[9], o2_beta = kc[10];
    const float x = __fdividef(pr * 273.f, t);
    const float x2 = 0.1f * x * x;
    if (on & 4)
      beta += x2 * __expf(n2_beta * (1.f / 296.f - 1.f / t)) * 0.79f * n2_b *
              (0.79f + 0.21f * (1.294f - 0.4545f * t / 296.f));
    if (on & 8) beta += x2 * __expf(o2_beta * (1.f / 296.f - 1.f / t)) * 0.21f * o2_b;
  }
  return beta;
}

// Source function (formod_srcfunc) of a channel's table at temperature t.
__device__ __forceinline__ float source_f(const float* srf, float t) {
  const float st0 = (float)kTMIN, sdt = (float)((kTMAX - kTMIN) / (kNS - 1.0));
  const float xs = (t - st0) / sdt;
  int is = (int)xs;
  is = is < 0 ? 0 : (is > kNS - 2 ? kNS - 2 : is);
  const float s0 = __ldg(srf + is), s1 = __ldg(srf + is + 1);
  return s0 + (s1 - s0) * (xs - (float)is);
}

// Emissivity of a segment from the emitters' E, the extinction beta and the
// length.
__device__ __forceinline__ float segment_f(float E, float beta, float ds) {
  return E + (1.f - E) * (-expm1f(-beta * ds));
}

// E of a segment joined with another emitter's emissivity.
__device__ __forceinline__ float join_f(float E, float eg) {
  return __fmaf_rn(__fsub_rn(1.f, E), eg, E);
}

// One segment (v = src * eps, m = 1 - eps) added to the Kahan-compensated
// radiance sum and the path transmittance.
__device__ __forceinline__ void add_f(float v, float m, float& rad, float& comp, float& tau) {
  const float y = __fmaf_rn(v, tau, -comp);
  const float sum = __fadd_rn(rad, y);
  comp = __fsub_rn(__fsub_rn(sum, rad), y);
  rad = sum;
  tau = __fmul_rn(tau, m);
}

// Cloud extinction and surface emissivity of a (ray, channel).
__device__ __forceinline__ float cloud_of(const CtlDev& c, const ChanDev& ch, const BatchDev& b,
                                          int r, int id, bool* has) {
  const double* s = b.scal + (long long)b.ray_obs[r] * b.nscal;
  *has = c.ncl > 0 && s[1] > 0;
  if (!*has) return 0.f;
  const double nu = ch.nu[id];
  const int icl = bracket_irr(ch.clnu, c.ncl, nu);
  return (float)lin(ch.clnu[icl], s[2 + icl], ch.clnu[icl + 1], s[2 + icl + 1], nu);
}

__device__ __forceinline__ float sfeps_of(const CtlDev& c, const ChanDev& ch, const BatchDev& b,
                                          int r, int id) {
  if (c.nsf <= 0) return 1.f;
  const double* se = b.scal + (long long)b.ray_obs[r] * b.nscal + 5 + c.ncl;
  const double nu = ch.nu[id];
  const int isf = bracket_irr(ch.sfnu, c.nsf, nu);
  return (float)lin(ch.sfnu[isf], se[isf], ch.sfnu[isf + 1], se[isf + 1], nu);
}

// Surface emission, reflection and solar term (jurassic.c:3264-3328), BT
// conversion and mask.  seg: the n segments {src * eps, 1 - eps} step apart
// where the surface reflects, else nullptr.
__device__ __forceinline__ void write_radiance(const CtlDev& c, const TblDev& T, const ChanDev& ch,
                                               const BatchDev& b, const LosDev& L, int id, int r,
                                               float rad, float tau, const float* seg,
                                               long long step, int n) {
  const double nu = ch.nu[id];
  double radd = (double)rad;
  const double sft = L.sft[r];
  if (c.sftype >= 1 && sft > 0) {
    const float sfeps = sfeps_of(c, ch, b, r, id);
    const float ssf = source_f(T.srf + (long long)id * kNS, (float)sft);
    radd += (double)(sfeps * ssf * tau);
    if (seg) {
      float tr = 1.f;
      double acc = 0;
      for (int ip = n - 1; ip >= 0; ip--) {
        acc += (double)(seg[ip * step] * tr);
        tr *= seg[ip * step + 32];
      }
      radd += acc * (double)tau * (double)(1.f - sfeps);
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
          radd += 6.764e-5 / (2. * kPI) * planck(kTSUN, nu) * tr * (1 - sfeps) * tau * rcos;
        }
      }
    }
  }
  const long long oi = (long long)id * b.nray + r;
  if (c.fov) {  // pencil beam only: FOV convolution, BT and mask follow in k_fov
    b.rad[oi] = radd;
    b.tau[oi] = (double)tau;
    return;
  }
  if (c.write_bbt) radd = kC2 * nu / log1p(kC1 * (nu * nu * nu) / radd);
  b.rad[oi] = b.mask[oi] ? __longlong_as_double(0x7ff8000000000000LL) : radd;
  b.tau[oi] = (double)tau;
}

// Does perturbed ray r take emitter g from its base ray?
__device__ __forceinline__ bool shared_gas(const MixedPlan& P, int r, int g) {
  if (!P.reuse) return false;
  const int2 ru = P.reuse[r];
  return ru.x >= 0 && ru.y != g;
}

// ---------------------------------------------------------------------------
// opaque rays
//
// Behind a thick cloud or window extinction a ray's path adds nothing (kTauStop),
// but the emitters' kernel does not know the other factors of the ray's
// transmittance.  The extinctions' optical depth depends on no emitter, and the
// emitters' transmittances are at most 1: from the point where it reaches
// kOpaqueDepth the transmittance is below 1e-13 (the CO2 continuum's
// extrapolation to 100 K could take 0.1 off the depth, two segments that are
// opaque by themselves and round to 1 a factor of 4), so that k_scan_m would have
// stopped there or before.  8000 nadir observations x 50 channels x 5 emitters, 5
// per km below 80, 40 and 20 km: 31.6, 31.3 and 31.5 ms without these ends, 8.6,
// 20.3 and 27.0 with them; the kernel that held all emitters of a channel in a
// warp and left at kTauStop took 11.1, 26.9 and 37.1, and 43.8 on clear scenes
// (31.5 here).
constexpr float kOpaqueDepth = 30.f;

// Sums along every ray, a warp per ray: extinction x length of every window, then
// cloud factor x length; -infinity where a value is negative (such a ray keeps
// all its points).
__global__ void __launch_bounds__(128) k_ext_sums(CtlDev c, LosDev L, int nray, float* out) {
  const int lane = threadIdx.x & 31;
  const long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (r >= nray) return;
  const int n = L.count[r];
  const long long base = L.off[r];
  for (int w = 0; w <= c.nw; w++) {
    const float* k = (w < c.nw ? L.f.kw + w * L.cap : L.f.aux) + base;
    float sum = 0.f;
    bool negative = false;
    if (w < c.nw || c.ncl > 0)
      for (int ip = lane; ip < n; ip += 32) {
        const float v = k[ip];
        sum += v * L.f.ds[base + ip];
        negative |= v < 0.f;
      }
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    negative = __any_sync(0xffffffffu, negative);
    if (lane == 0) out[(long long)w * nray + r] = negative ? __int_as_float(0xff800000) : sum;
  }
}

// Does the surface of ray r reflect in channel id?  Its sum needs every point.
__device__ __forceinline__ bool reflects(const CtlDev& c, const ChanDev& ch, const BatchDev& b,
                                         const LosDev& L, int r, int id) {
  return c.sftype >= 2 && c.nsf > 0 && L.sft[r] > 0 && sfeps_of(c, ch, b, r, id) < 1.f;
}

// P.ends of a chunk, a warp per (tile, channel): the points that a lane walks, 0
// where it is empty, skipped or masked.  A perturbed ray (RES 2) sums from its
// start point on, and needs no point beyond it where its base was opaque there.
template <int RES>
__global__ void __launch_bounds__(128) k_path_ends(CtlDev c, TblDev T, ChanDev ch, BatchDev b,
                                                   LosDev L, MixedPlan P) {
  const int lane = threadIdx.x & 31, ndc = P.id1 - P.id0;
  const long long w = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int idl = (int)(w % ndc), tl = (int)(w / ndc);
  if (tl >= P.tile1 - P.tile0) return;
  const int tile = P.tile0 + tl, id = P.id0 + idl;
  const int r = P.perm[tile * 32 + lane];
  const int n = r >= 0 && !(b.obs_skip && b.obs_skip[b.ray_obs[r]]) &&
                        !(b.skip_masked && b.mask[(long long)id * b.nray + r])
                    ? L.count[r] : 0;
  int start = 0, end = n;
  if (RES == 2 && n > 0) {
    start = P.start[r];
    if (start > 0 && P.snap_sums[((long long)r * P.gndc + (id - P.gid0)) * 3 + 2] < kTauStop) end = start;
  }
  bool walk = false;
  float cl = 0.f;
  const Fields F = fields_of(c);
  const int win = c.nw > 0 ? __float_as_int(T.chanf[id * kChanConsts + kChanWindow]) : -1;
  if (P.ext_sum && n > 0 && end == n) {
    if (P.cloud) cl = P.cloud[(long long)id * b.nray + r];
    const float depth = (win >= 0 ? P.ext_sum[(long long)win * b.nray + r] : 0.f) +
                        cl * P.ext_sum[(long long)c.nw * b.nray + r];
    walk = depth >= kOpaqueDepth && !(cl < 0.f) && (RES != 0 || !reflects(c, ch, b, L, r, id));
  }
  if (__any_sync(0xffffffffu, walk)) {
    const float* f = P.data + P.toff[tile] * (long long)F.n * 32 + lane;
    const int kw = win >= 0 ? (F.kw0 + win) * 32 : -1;
    float depth = 0.f;
    int ip = (int)__reduce_min_sync(0xffffffffu, walk ? (unsigned)start : 0x7fffffffu);
    const int last = (int)(P.toff[tile + 1] - P.toff[tile]) - 1;
    const bool cloudy = P.cloud != nullptr;
    constexpr int U = 8;  // points in flight: every lane loads, the walking ones use them
    for (; __any_sync(0xffffffffu, walk); ip += U) {
      float v[U], a[U], ds[U];
#pragma unroll
      for (int k = 0; k < U; k++) {
        const float* q = f + (long long)min(ip + k, last) * F.n * 32;
        v[k] = kw >= 0 ? q[kw] : 0.f;
        a[k] = cloudy ? q[F.aux * 32] : 0.f;
        ds[k] = q[F.ds * 32];
      }
#pragma unroll
      for (int k = 0; k < U; k++) {
        if (ip + k >= start && ip + k < n) depth += (v[k] + a[k] * cl) * ds[k];
        if (walk && depth >= kOpaqueDepth) {
          end = min(ip + k + 1, n);
          walk = false;
        }
      }
      walk = walk && ip + U < n;
    }
  }
  P.ends[(long long)w * 32 + lane] = end;
}

// ---------------------------------------------------------------------------
// the path of a batch, in three kernels
//
// k_gas_m: the emitters' paths are independent (one tau_path per emitter in
// intpol_tbl_ega / intpol_tbl_cga), so a warp walks a tile's points for one
// (channel, emitter) with the state in registers and writes the segment
// emissivities.  LPR = 4 gives each ray four lanes, one per corner of the p-T
// cell, for batches that leave the device idle.  shape 1: the warps of a
// block take consecutive tiles of one (channel, emitter), whose rows they
// share in L1; shape 0: consecutive channels of one tile.
// Bound by instruction issue and the L1 data pipe together (77 % and 70 %
// busy on 62 nadir tiles x 100 channels x 5 emitters, 354 instructions per
// point and emitter, DRAM 5 %): 12.1 ms for those 3.1e7 warp steps, against
// 17 ms in a kernel that held all emitters of a channel in a warp (527
// instructions, state in shared memory).  What the register count costs
// shows in the variants: 12.8 to 14.7 ms.
//
// RES: 1 the base rays of resumed perturbations, which leave their state
// before every start point of their perturbations; 2 the perturbations, which
// walk on from there, and not at all for an emitter they share with the base.
// 48 nadir observations x 405 perturbations, 150 channels, 4 emitters: 29 ms
// here and 17 ms in k_seg_m (6.8e7 and 3.8e7 warp points; bound by issue as
// above, with 1.5 times the plain batch's time per point since a warp's rays
// come from several observations and share fewer rows), against 64 ms in a
// kernel that held all emitters of a channel in a warp and joined the shared
// ones there.
template <bool CGA, int LPR, int MINB, bool FAST, int RES = 0>
__global__ void __launch_bounds__(kPathThreads, MINB) k_gas_m(CtlDev c, TblDev T, BatchDev b,
                                                              LosDev L, MixedPlan P, int shape) {
  constexpr int W = kPathThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ng = c.ng, ndc = P.id1 - P.id0;
  int tl, idl, g, part8 = 0;
  if (LPR == 4 || shape == 0) {
    long long w = (long long)blockIdx.x * W + warp;
    idl = (int)(w % ndc);
    w /= ndc;
    g = (int)(w % ng);
    w /= ng;
    if (LPR == 4) {
      part8 = (int)(w & 3);
      w >>= 2;
    }
    tl = (int)w;
  } else {
    const unsigned per = (unsigned)(ndc * ng);
    tl = (int)(blockIdx.x / per) * W + warp;
    const unsigned rem = blockIdx.x % per;
    idl = (int)(rem / ng);
    g = (int)(rem % ng);
  }
  if (tl >= P.tile1 - P.tile0) return;
  const int tile = P.tile0 + tl, id = P.id0 + idl;
  const long long dg = (long long)id * ng + g;
  const int np = __ldg(T.np + dg);
  if (np < 30) return;  // no table: k_seg_m leaves this emitter out
  const int rl = LPR == 4 ? part8 * 8 + (lane >> 2) : lane, corner = lane & 3;
  int r = 0, n = 0;
  if (LPR == 1 && RES != 1) {
    n = P.ends[(long long)(tl * ndc + idl) * 32 + rl];
    if (RES == 2) r = P.perm[tile * 32 + rl];
  } else {
    r = P.perm[tile * 32 + rl];
    if (r >= 0 && b.obs_skip && b.obs_skip[b.ray_obs[r]]) r = -1;
    if (r >= 0 && b.skip_masked && b.mask[(long long)id * b.nray + r]) r = -1;
    n = r >= 0 ? L.count[r] : 0;
  }
  if (RES == 2 && n > 0 && shared_gas(P, r, g)) n = 0;
  const Fields F = fields_of(c);
  constexpr int es = kEmitterFields(CGA), kb = kFBr(CGA);
  const float* f = P.data + P.toff[tile] * (long long)F.n * 32 + rl;
  const float* fg = f + (F.g0 + g * es) * 32;
  const int fstep = F.n * 32;
  const long long lp0 = P.toff[tile] - P.pt0;
  float* out = P.seg + ((lp0 * ndc + idl) * P.nseg + (RES == 2 ? g * P.gstep : g)) * 32 + rl;
  const long long ostep = (long long)ndc * P.nseg * 32;
  const bool brg = FAST || ((P.brmask >> g) & 1u);
  GasState st;
  st.t = 1.f;
  st.e = 0.f;
  st.ipr = -1;
#pragma unroll
  for (int k = 0; k < 4; k++) st.h[k] = 0;
  int stop = n;  // the first point that is saturated: all later ones are too
  // resumed perturbations: the state before a start point
  int sn = 0, se = 0;
  auto state_of = [&](int ray) {
    return P.snap + (((long long)ray * P.gndc + (id - P.gid0)) * ng + g) * kStateWords;
  };
  auto save = [&](int target) {
    if (shared_gas(P, target, g)) return;
    unsigned* q = state_of(target);
    if (LPR == 1 || corner == 0) {
      q[0] = __float_as_uint(st.t);
      q[1] = __float_as_uint(st.e);
      q[2] = (unsigned)st.ipr;
    }
    unsigned short* h = reinterpret_cast<unsigned short*>(q + 3);
    if (LPR == 4) h[corner] = (unsigned short)st.h[0];
    else
#pragma unroll
      for (int k = 0; k < 4; k++) h[k] = (unsigned short)st.h[k];
  };
  if (RES == 1 && n > 0) {
    sn = P.snap_off[r];
    se = P.snap_off[r + 1];
  }
  int next = RES == 1 && sn < se ? P.snap_ip[sn] : 0x7fffffff;
  auto save_at = [&](int ip) {
    while (next == ip) {
      save(P.snap_ray[sn]);
      next = ++sn < se ? P.snap_ip[sn] : 0x7fffffff;
    }
  };
  if (LPR == 1) {
    int start = 0, ip = 0;
    if (RES == 2) {
      start = n > 0 ? P.start[r] : 0x7fffffff;
      ip = (int)__reduce_min_sync(0xffffffffu, (unsigned)start);
      if (ip == 0x7fffffff) return;  // no lane walks
      if (n > 0 && start > 0) {
        const unsigned* q = state_of(r);
        st.t = __uint_as_float(q[0]);
        st.e = __uint_as_float(q[1]);
        st.ipr = (int)q[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
          st.h[2 * k] = (int)(q[3 + k] & 0xffffu);
          st.h[2 * k + 1] = (int)(q[3 + k] >> 16);
        }
      }
      out += ip * ostep;
      f += (long long)ip * fstep;
      fg += (long long)ip * fstep;
    }
    for (; ip < n; ip++) {
      if (RES == 2 && ip < start) {  // one row of the tile for all lanes
        out += ostep;
        f += fstep;
        fg += fstep;
        continue;
      }
      if (RES == 1) save_at(ip);
      const float du = CGA ? 0.f : fg[kFU * 32];
      const float pq = CGA ? fg[kFCgp * 32] : brg ? 0.f : f[F.p * 32];
      const float tq = CGA ? fg[kFCgt * 32] : brg ? 0.f : f[F.t * 32];
      const float ucg = CGA ? fg[kFCgu * 32] : 0.f;
      const float4 cw = brg ? cell_words(fg + kb * 32, rl) : no_cell();
      bool sat = false;
      const float eg = gas_eps_f<CGA, FAST>(T, dg, pq, tq, du, ucg, cw, st, sat);
      if (sat) {
        stop = ip;
        break;
      }
      *out = eg;
      out += ostep;
      f += fstep;
      fg += fstep;
    }
    // beyond the walk's end a perturbation starts saturated, as its base ended
    if (RES == 1)
      for (; sn < se; sn++) save(P.snap_ray[sn]);
    if (r >= 0) P.stop[((long long)(tl * ndc + idl) * ng + g) * 32 + rl] = stop;
    return;
  }
  const int nmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
  // the next point's fields are loaded ahead of this point's chain
  float nu = 0.f, npq = 0.f, ntq = 0.f;
  float4 ncw = no_cell();
  auto fetch = [&](int ip) {
    if (ip >= n) return;
    const float* q = fg + (long long)ip * fstep;
    nu = CGA ? q[kFCgu * 32] : q[kFU * 32];
    if (brg) {
      ncw = cell_words(q + kb * 32, rl);
    } else {
      npq = CGA ? q[kFCgp * 32] : f[(long long)ip * fstep + F.p * 32];
      ntq = CGA ? q[kFCgt * 32] : f[(long long)ip * fstep + F.t * 32];
    }
  };
  fetch(0);
  for (int ip = 0; ip < nmax; ip++) {
    if (RES == 1) save_at(ip);
    bool on = ip < n && stop == n;
    if (on && st.t < 1e-9f) {
      stop = ip;
      on = false;
    }
    if (!__any_sync(0xffffffffu, on)) break;
    const float u = nu, pq = npq, tq = ntq;
    CellFind cf{};
    if (brg) cf.k = cell_packed(T, dg, ncw);
    else if (on) cf = cell_find<CGA>(T, dg, np, pq, tq, st.ipr);
    fetch(ip + 1);
    float mine = 0.f;
    int cnt = 0;
    if (on && cf.k.ok) {
      const unsigned row = ((corner & 2) ? cf.k.rc : cf.k.ra) + (corner & 1);
      const float4 m = row_record<CGA>(T, row);
      cnt = row_count<CGA>(m);
      if (cnt >= 2) mine = corner_any<CGA, FAST>(T, row, m, cnt, st.e, u, u, st.h[0]);
    }
    const bool ok = ((__ballot_sync(0xffffffffu, cnt >= 2) >> (lane & ~3)) & 15u) == 15u;
    const float ox = __shfl_xor_sync(0xffffffffu, mine, 1);
    const float lo = (corner & 1) ? ox : mine, hi = (corner & 1) ? mine : ox;
    const float et = brg ? mix_f(lo, hi, (corner & 2) ? cf.k.b : cf.k.a)
                         : (corner & 2) ? mix_t(lo, hi, cf.tc, cf.td, tq)
                                        : mix_t(lo, hi, cf.ta, cf.tb, tq);
    const float oy = __shfl_xor_sync(0xffffffffu, et, 2);
    const float ea = (corner & 2) ? oy : et, eb = (corner & 2) ? et : oy;
    if (on) {
      bool sat = false;
      const float eg = ok ? extend_f(mix_f(ea, eb, cf.k.w), st, sat) : 0.f;
      if (sat) stop = ip;
      else if (corner == 0) out[ip * ostep] = eg;
    }
  }
  if (RES == 1)
    for (; sn < se; sn++) save(P.snap_ray[sn]);
  if (r >= 0 && corner == 0) P.stop[((long long)(tl * ndc + idl) * ng + g) * 32 + rl] = stop;
}

// k_seg_m: joins the emitters' segments with the continua, clouds and
// extinction and leaves src * eps and 1 - eps in the first two of the point's
// entries.  Nothing here depends on the path, so a warp takes a run of
// kSegRun points of its (tile, channel): long enough that the channel's
// constants and the rays' limits are read once per run, short enough to
// spread a small batch (a warp per point took 398 instructions for what takes
// 212 here; 3.3 -> 1.8 ms for 6.2e6 warp points, 5.5 GB of DRAM traffic).
constexpr int kSegRun = 16;
// Cloud extinction of a ray without a cloud: -0 (an extinction of -0 is kept as 0,
// and one that is not a number stays one).  Tested per lane: a test of the batch
// alone, hoisted, costs k_seg_m 48 instead of 40 registers (20000 limb rays:
// 1.55 instead of 1.14 ms).
constexpr unsigned kNoCloud = 0x80000000u;

template <int RES>
__global__ void __launch_bounds__(kPathThreads) k_seg_m(CtlDev c, TblDev T, BatchDev b, LosDev L,
                                                        MixedPlan P) {
  const int lane = threadIdx.x & 31;
  const int ng = c.ng, ndc = P.id1 - P.id0, nchb = (ndc + 3) / 4;
  const int idl = (int)(blockIdx.x % nchb) * 4 + (threadIdx.x >> 5);
  const int ip0 = (int)(blockIdx.x / nchb) * kSegRun;
  const int tl = (int)blockIdx.y, tile = P.tile0 + tl;
  if (idl >= ndc) return;
  const int id = P.id0 + idl;
  const int r = P.perm[tile * 32 + lane];
  if (r < 0 || (b.obs_skip && b.obs_skip[b.ray_obs[r]])) return;
  if (b.skip_masked && b.mask[(long long)id * b.nray + r]) return;
  // the run ends at the first saturated emitter, where k_scan_m stops
  int n = min(L.count[r], ip0 + kSegRun);
  const int* st = P.stop + (long long)(tl * ndc + idl) * ng * 32 + lane;
  unsigned has = 0, own = ~0u;  // emitters with a table; of this ray, not of its base
  const float* bseg = nullptr;
  long long bstep = 0;
  int start = 0;
  const int* bst = nullptr;
  if (RES == 2) {
    start = P.start[r];
    const int2 ru = P.reuse ? P.reuse[r] : make_int2(-1, -1);
    if (ru.x >= 0) {
      const int slot = P.base_slot[ru.x], bt = slot >> 5, gidl = id - P.gid0;
      own = ru.y >= 0 ? 1u << ru.y : 0u;
      bst = P.base_stop + (long long)(bt * P.gndc + gidl) * ng * 32 + (slot & 31);
      bstep = (long long)P.gndc * P.base_nseg * 32;
      bseg = P.base_seg + (P.toff[bt] + ip0) * bstep + (long long)gidl * P.base_nseg * 32 + (slot & 31);
    }
  }
  for (int g = 0; g < ng; g++)
    if (__ldg(T.np + (long long)id * ng + g) >= 30) {
      has |= 1u << g;
      n = min(n, RES == 2 && !((own >> g) & 1u) ? bst[g * 32] : st[g * 32]);
    }
  if (RES != 1 && P.ends) n = min(n, P.ends[(long long)(tl * ndc + idl) * 32 + lane]);
  if (RES == 2 && n <= start) return;
  const Fields F = fields_of(c);
  const long long pt = P.toff[tile] + ip0;
  const float* f = P.data + pt * F.n * 32 + lane;
  float* seg = P.seg + ((pt - P.pt0) * ndc + idl) * (long long)P.nseg * 32 + lane;
  const long long sstep = (long long)ndc * P.nseg * 32;
  float kc[kChanWindow];
  for (int k = 0; k < kChanWindow; k++) kc[k] = T.chanf[id * kChanConsts + k];
  const int on = continua_on(c, kc[kChanSwitches]);
  const int kw = c.nw > 0 ? (F.kw0 + __float_as_int(T.chanf[id * kChanConsts + kChanWindow])) * 32 : -1;
  const float cl = P.cloud ? P.cloud[(long long)id * b.nray + r] : __uint_as_float(kNoCloud);
  const float* srf = T.srf + (long long)id * kNS;
  const int po = RES == 1 ? ng * 32 : 0;  // a base ray's emitters stay for its perturbations
  for (int ip = ip0; ip < n; ip++, f += F.n * 32, seg += sstep) {
    float E = 0.f;
    if (RES == 2 && ip < start) {
      bseg += bstep;
      continue;
    }
    for (int g = 0; g < ng; g++)
      if ((has >> g) & 1u)
        E = join_f(E, RES != 2 ? seg[g * 32] : (own >> g) & 1u ? seg[g * P.gstep * 32] : bseg[g * 32]);
    if (RES == 2) bseg += bstep;
    const float p = f[F.p * 32], t = f[F.t * 32], ds = f[F.ds * 32];
    float beta = kw >= 0 ? f[kw] : 0.f;
    if (__float_as_uint(cl) != kNoCloud) beta = __fmaf_rn(f[F.aux * 32], cl, beta);
    beta = continua_f(c, F, kc, on, f, p, t, ds, beta);
    const float src = source_f(srf, t);
    const float eps = segment_f(E, beta, ds);
    seg[po] = __fmul_rn(src, eps);
    seg[po + 32] = __fsub_rn(1.f, eps);
  }
}

// Cloud extinction of every (channel, ray), kNoCloud without a cloud.
__global__ void k_cloud_m(CtlDev c, ChanDev ch, BatchDev b, float* out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)c.nd * b.nray) return;
  bool has = false;
  const float v = cloud_of(c, ch, b, (int)(i % b.nray), (int)(i / b.nray), &has);
  out[i] = has ? v + 0.f : __uint_as_float(kNoCloud);
}

// k_scan_m: one thread per (ray, channel) sums the segments along the path.
// It stops at the first saturated emitter (nothing adds after it) and, without
// surface reflection, once the path transmittance is below kTauStop: the rest
// adds at most max(src) tau, below 1e-10 of the radiance.
template <int RES>
__global__ void __launch_bounds__(kPathThreads) k_scan_m(CtlDev c, TblDev T, ChanDev ch, BatchDev b,
                                                         LosDev L, MixedPlan P) {
  const int lane = threadIdx.x & 31;
  const int ng = c.ng, ndc = P.id1 - P.id0;
  const long long w = (long long)blockIdx.x * (kPathThreads / 32) + (threadIdx.x >> 5);
  const int idl = (int)(w % ndc), tl = (int)(w / ndc);
  if (tl >= P.tile1 - P.tile0) return;
  const int tile = P.tile0 + tl, id = P.id0 + idl;
  const int r = P.perm[tile * 32 + lane];
  const bool idle = r < 0 || (b.obs_skip && b.obs_skip[b.ray_obs[r]]);
  if (RES != 2 && idle) return;
  int n = idle || (b.skip_masked && b.mask[(long long)id * b.nray + r]) ? 0 : L.count[r];
  const int* st = P.stop + (long long)(tl * ndc + idl) * ng * 32 + lane;
  float rad = 0.f, comp = 0.f, tau = 1.f;
  int ip = 0, start = 0, sn = 0, se = 0;
  const int* bst = nullptr;
  unsigned own = ~0u;
  auto sums_of = [&](int ray) { return P.snap_sums + ((long long)ray * P.gndc + (id - P.gid0)) * 3; };
  if (RES == 2) {  // on from the base's sums, one row of the tile for all lanes
    start = n > 0 ? P.start[r] : 0x7fffffff;
    ip = (int)__reduce_min_sync(0xffffffffu, (unsigned)start);
    if (idle) return;
    if (n > 0) {
      const int2 ru = P.reuse ? P.reuse[r] : make_int2(-1, -1);
      if (ru.x >= 0) {
        const int slot = P.base_slot[ru.x];
        own = ru.y >= 0 ? 1u << ru.y : 0u;
        bst = P.base_stop + (long long)((slot >> 5) * P.gndc + (id - P.gid0)) * ng * 32 + (slot & 31);
      }
      if (start > 0) {
        const float* q = sums_of(r);
        rad = q[0];
        comp = q[1];
        tau = q[2];
      }
    }
  }
  if (RES != 1 && P.ends && n > 0) n = min(n, P.ends[(long long)(tl * ndc + idl) * 32 + lane]);
  for (int g = 0; g < ng; g++)
    if (n > 0 && __ldg(T.np + (long long)id * ng + g) >= 30)
      n = min(n, RES == 2 && !((own >> g) & 1u) ? bst[g * 32] : st[g * 32]);
  if (RES == 1 && !(b.skip_masked && b.mask[(long long)id * b.nray + r])) {
    sn = P.snap_off[r];
    se = P.snap_off[r + 1];
  }
  int next = sn < se ? P.snap_ip[sn] : 0x7fffffff;
  auto save = [&]() {
    float* q = sums_of(P.snap_ray[sn]);
    q[0] = rad;
    q[1] = comp;
    q[2] = tau;
    next = ++sn < se ? P.snap_ip[sn] : 0x7fffffff;
  };
  const float* seg = P.seg + ((P.toff[tile] - P.pt0) * ndc + idl) * (long long)P.nseg * 32 + lane +
                     (RES == 1 ? ng * 32 : 0);
  const long long step = (long long)ndc * P.nseg * 32;
  const bool refl = RES == 0 && reflects(c, ch, b, L, r, id);
  constexpr int U = 8;  // loads in flight ahead of the sums
  for (; ip < n; ip += U) {
    if (tau < kTauStop && !refl) break;
    float v[U], m[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      const bool in = ip + k < n && (RES != 2 || ip + k >= start);
      v[k] = in ? seg[(ip + k) * step] : 0.f;
      m[k] = in ? seg[(ip + k) * step + 32] : 1.f;
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      if (RES == 1 && ip + k < n)
        while (next == ip + k) save();
      if (ip + k < n && (RES != 2 || ip + k >= start) && (refl || !(tau < kTauStop)))
        add_f(v[k], m[k], rad, comp, tau);
    }
  }
  while (RES == 1 && sn < se) save();
  write_radiance(c, T, ch, b, L, id, r, rad, tau, refl ? seg : nullptr, step, n);
}

// Row records (layouts above); rows with fewer than two entries are never
// interpolated and get zeros.
__global__ void k_rowmeta(long long nrow, int tu, const int* nu, const float* u, const float* e,
                          int cga, float4* meta) {
  const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrow) return;
  const int n = nu[r];
  const float* ur = u + r * tu;
  const float* er = e + r * tu;
  const float nf = __int_as_float(n);
  if (cga) {
    meta[r] = n >= 2 ? make_float4(nf, 0.f, ur[0], er[0]) : make_float4(nf, 0.f, 0.f, 0.f);
    return;
  }
  float4 m = make_float4(0.f, 0.f, 0.f, nf), m2 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (n >= 2) {
    m = make_float4(ur[0], er[0], er[n - 1], nf);
    m2 = make_float4(ur[n - 1], log1pf(-er[n - 1]) / ur[n - 1], 0.f, 0.f);
  }
  meta[2 * r] = m;
  meta[2 * r + 1] = m2;
}

// The rows interleaved {u[i], eps[i]}: a probe of one brings the other; marks
// odd rows (kOddRow, from the entry that shows it).
__global__ void k_interleave(long long n, int tu, const int* nu, const float* u, const float* e,
                             int cga, float2* ue, float4* meta, int* any_odd) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float a = u[i], b = e[i];
  ue[i] = make_float2(a, b);
  const long long r = i / tu;
  const int k = (int)(i - r * tu), cnt = nu[r];
  if (cnt < 2 || k >= cnt) return;
  const bool fine = fabsf(a) < 4.2535296e37f && fabsf(b) < 4.2535296e37f &&  // 2^125
                    (k + 1 >= cnt || (a <= u[i + 1] && b <= e[i + 1]));
  if (!fine) {
    atomicOr(reinterpret_cast<int*>(cga ? &meta[r].x : &meta[2 * r].w), kOddRow);
    *any_odd = 1;
  }
}

void launch_rowmeta(long long nrow, int tu, const int* nu, const float* u, const float* e, int cga,
                    float4* meta, float2* ue, int* any_odd, cudaStream_t s) {
  const int bs = 256;
  if (nrow > 0) {
    k_rowmeta<<<(unsigned)((nrow + bs - 1) / bs), bs, 0, s>>>(nrow, tu, nu, u, e, cga, meta);
    const long long n = nrow * tu;
    k_interleave<<<(unsigned)((n + bs - 1) / bs), bs, 0, s>>>(n, tu, nu, u, e, cga, ue, meta,
                                                               any_odd);
  }
}

__global__ void k_src_to_float(int nd, const double* sr, float* srf) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nd * kNS) return;
  const int id = gid / kNS, it = gid % kNS;
  srf[gid] = (float)sr[(long long)it * nd + id];
}

void launch_pack_tiles_n(const CtlDev& c, const TblDev& T, const LosDev& L, const MixedPlan& P,
                         long long total_tile_points, cudaStream_t s) {
  const long long nth = total_tile_points * 32;
  const int bs = 256;
  k_pack_tiles<<<(unsigned)((nth + bs - 1) / bs), bs, 0, s>>>(c, T, L, P, total_tile_points);
}

// The resumed kernels take at most 64 registers (16 observations x 405 elements, emitters'
// kernel: 24.6 ms; 48, 40 and 32 registers 24.8, 25.1 and 26.6).
// Variants of k_gas_m with one lane per ray, chosen by the autotuner: block
// shape (v / 4) and minimum resident blocks per SM (v % 4: 8, 10, 12, 16, i.e.
// at most 64, 48, 40 and 32 registers).
int path_gas_variants() { return 8; }

template <bool CGA>
void launch_gas_v(const CtlDev& c, const TblDev& T, const BatchDev& b, const LosDev& L,
                  const MixedPlan& P, int lanes_per_ray, int variant, int res, cudaStream_t s) {
  const long long nt = P.tile1 - P.tile0, ndc = P.id1 - P.id0;
  constexpr int W = kPathThreads / 32;
  const int shape = lanes_per_ray == 4 ? 0 : variant / 4;
  const unsigned nblk =
      (unsigned)(lanes_per_ray == 4 ? (nt * ndc * c.ng * 4 + W - 1) / W
                 : shape ? (nt + W - 1) / W * ndc * c.ng : (nt * ndc * c.ng + W - 1) / W);
  auto go = [&](auto kern) { kern<<<nblk, kPathThreads, 0, s>>>(c, T, b, L, P, shape); };
  if (res == 1) {
    if (lanes_per_ray == 4) return P.fast ? go(k_gas_m<CGA, 4, 8, true, 1>) : go(k_gas_m<CGA, 4, 8, false, 1>);
    return P.fast ? go(k_gas_m<CGA, 1, 8, true, 1>) : go(k_gas_m<CGA, 1, 8, false, 1>);
  }
  if (res == 2) return P.fast ? go(k_gas_m<CGA, 1, 8, true, 2>) : go(k_gas_m<CGA, 1, 8, false, 2>);
  if (lanes_per_ray == 4) return P.fast ? go(k_gas_m<CGA, 4, 8, true>) : go(k_gas_m<CGA, 4, 8, false>);
  if (!P.fast) return go(k_gas_m<CGA, 1, 8, false>);
  switch (variant % 4) {
    case 0: go(k_gas_m<CGA, 1, 8, true>); break;
    case 1: go(k_gas_m<CGA, 1, 10, true>); break;
    case 2: go(k_gas_m<CGA, 1, 12, true>); break;
    default: go(k_gas_m<CGA, 1, 16, true>); break;
  }
}

void launch_gas_m(const CtlDev& c, const TblDev& T, const BatchDev& b, const LosDev& L,
                  const MixedPlan& P, int lanes_per_ray, int variant, int res, cudaStream_t s) {
  if (c.ng <= 0) return;
  if (c.formod == 0) launch_gas_v<true>(c, T, b, L, P, lanes_per_ray, variant, res, s);
  else launch_gas_v<false>(c, T, b, L, P, lanes_per_ray, variant, res, s);
}

void launch_seg_scan_m(const CtlDev& c, const TblDev& T, const ChanDev& ch, const BatchDev& b,
                       const LosDev& L, const MixedPlan& P, int longest, int res, cudaStream_t s) {
  const long long nt = P.tile1 - P.tile0, ndc = P.id1 - P.id0, nchb = (ndc + 3) / 4;
  const long long runs = (longest + kSegRun - 1) / kSegRun;
  const dim3 gs((unsigned)(nchb * runs), (unsigned)nt);
  const unsigned gn = (unsigned)((nt * ndc + 3) / 4);
  if (res == 1) {
    k_seg_m<1><<<gs, kPathThreads, 0, s>>>(c, T, b, L, P);
    k_scan_m<1><<<gn, kPathThreads, 0, s>>>(c, T, ch, b, L, P);
  } else if (res == 2) {
    k_seg_m<2><<<gs, kPathThreads, 0, s>>>(c, T, b, L, P);
    k_scan_m<2><<<gn, kPathThreads, 0, s>>>(c, T, ch, b, L, P);
  } else {
    k_seg_m<0><<<gs, kPathThreads, 0, s>>>(c, T, b, L, P);
    k_scan_m<0><<<gn, kPathThreads, 0, s>>>(c, T, ch, b, L, P);
  }
}

void launch_cloud_m(const CtlDev& c, const ChanDev& ch, const BatchDev& b, float* out,
                    cudaStream_t s) {
  const long long n = (long long)c.nd * b.nray;
  k_cloud_m<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(c, ch, b, out);
}

void launch_ext_sums(const CtlDev& c, const LosDev& L, int nray, float* out, cudaStream_t s) {
  k_ext_sums<<<(unsigned)((nray + 3) / 4), 128, 0, s>>>(c, L, nray, out);
}

void launch_path_ends(const CtlDev& c, const TblDev& T, const ChanDev& ch, const BatchDev& b,
                      const LosDev& L, const MixedPlan& P, int res, cudaStream_t s) {
  const long long warps = (long long)(P.tile1 - P.tile0) * (P.id1 - P.id0);
  const unsigned nblk = (unsigned)((warps + 3) / 4);
  if (res == 2) k_path_ends<2><<<nblk, 128, 0, s>>>(c, T, ch, b, L, P);
  else k_path_ends<0><<<nblk, 128, 0, s>>>(c, T, ch, b, L, P);
}

void launch_chan_consts(const CtlDev& c, const ChanDev& ch, float* out, cudaStream_t s) {
  k_chan_consts<<<(c.nd + 127) / 128, 128, 0, s>>>(c, ch, out);
}

size_t chan_const_bytes(const CtlDev& c) { return sizeof(float) * kChanConsts * (size_t)c.nd; }

size_t gas_state_bytes() { return sizeof(unsigned) * kStateWords; }

void launch_src_to_float(int nd, const double* sr, float* srf, cudaStream_t s) {
  const int n = nd * kNS, bs = 256;
  k_src_to_float<<<(n + bs - 1) / bs, bs, 0, s>>>(nd, sr, srf);
}

}  // namespace jgb
