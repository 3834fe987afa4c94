// Batched inverses of symmetric positive-definite matrices in FP64
// (gsl_linalg_cholesky_decomp and gsl_linalg_cholesky_invert as used by
// matrix_invert, retrieval.c:373-399), blocked in tiles of 32 x 32:
//
//   for every panel k: k_chol_diag   L_kk and its inverse, one warp
//                      k_chol_panel  L_ik = (A - S)_ik L_kk^-T, a tile per block
//                      k_chol_update S_ij += L_ik L_jk^T, a tile per block
//   k_tri_inverse      W = L^-1, one block per block column
//   k_gram             A^-1 = W^T W, a tile pair per block, both triangles
//
// and invert_small for matrices of a tile or less, a warp each.
//
// What bounds it: n^3 / 2 FP64 multiply-adds per matrix at 19 cycles of an SM
// per warp instruction (the tensor form of FP64 runs at the same rate).  A
// block per matrix left 56 of 152 SMs idle for 96 matrices and spent two
// instructions per multiply-add, 1.7 n^3 in all, with a block-wide barrier
// twice per column; tiles spread every matrix over the device, a thread keeps
// 4 x 4 sums in registers, and 32 x 32 tiles waste little on the diagonals.
// 96 matrices of up to 405 x 405 (48 of them smaller): 44.6 -> 7.9 ms, of
// which k_tri_inverse 2.8 (its longest column is 1.5), k_gram 1.8,
// k_chol_update 1.5, k_chol_diag 1.1 (13 panels, a warp's chain of roots),
// k_chol_panel 0.7; the multiply-adds alone are 4.1 ms.
//
// Rounding: sums are formed apart and subtracted once, a tile's products apart
// from the sum over the tiles, quotients are correctly rounded.  Error against
// inverses refined in long double, over the error of a block per matrix that
// subtracted whole sums (geometric means, n from 12 to 405): covariances 1.02,
// Gauss-Newton matrices 0.74.
#include <algorithm>

#include "../../include/jurassic_gb300.h"
#include "jgb_cholinv.cuh"

namespace jgb {
namespace {

constexpr int kB = 32;            // tile edge
constexpr int kT = 64;            // threads of a tile block, 4 x 4 sums each
constexpr int kPad = kB + 2;      // shared row stride (16-byte aligned rows)

struct Mat {
  int n;
  double* L;  // factor, row-major n x n, lower triangle
  double* W;  // inverse of the factor
};

__device__ __forceinline__ bool mat_at(const InvertDesc* d, const int* full, const int* status,
                                       double* Lall, double* Wall, int i, Mat& m) {
  if (!full[i] || status[i] || d[i].n <= kB) return false;
  m.n = d[i].n;
  m.L = Lall + d[i].off;
  m.W = Wall + d[i].off;
  return true;
}

// Tile (bi, bj) of a row-major n x n matrix into shared memory, zero outside;
// TR: transposed (s[column][row]).  LOWER: entries above the diagonal are zero.
template <bool TR, bool LOWER>
__device__ __forceinline__ void load_tile(const double* M, int n, int bi, int bj,
                                          double (*s)[kPad]) {
  for (int e = threadIdx.x; e < kB * kB; e += kT) {
    const int r = e / kB, c = e % kB;
    const int row = bi * kB + r, col = bj * kB + c;
    const bool in = row < n && col < n && (!LOWER || col <= row);
    const double v = in ? M[(long long)row * n + col] : 0.0;
    if (TR) s[c][r] = v; else s[r][c] = v;
  }
}

// acc += a^T b over the 32 rows of a and b (a[k][i], b[k][j]); thread t holds
// rows 4 (t / 8) .. and columns 4 (t % 8) .. of the tile.
__device__ __forceinline__ void tile_fma(const double (*a)[kPad], const double (*b)[kPad],
                                         double (&acc)[4][4]) {
  const int i0 = 4 * (threadIdx.x >> 3), j0 = 4 * (threadIdx.x & 7);
#pragma unroll 8
  for (int k = 0; k < kB; k++) {
    const double2 a0 = *reinterpret_cast<const double2*>(&a[k][i0]);
    const double2 a1 = *reinterpret_cast<const double2*>(&a[k][i0 + 2]);
    const double2 b0 = *reinterpret_cast<const double2*>(&b[k][j0]);
    const double2 b1 = *reinterpret_cast<const double2*>(&b[k][j0 + 2]);
    const double av[4] = {a0.x, a0.y, a1.x, a1.y}, bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][j] = fma(av[i], bv[j], acc[i][j]);
  }
}

__device__ __forceinline__ void tile_add(double (&acc)[4][4], const double (&part)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] += part[i][j];
}

// a / w from the reciprocal r of w > 0: quotient, exact remainder, one correction
// (Markstein, IBM J. Res. Dev. 34, 1990); 0 for an infinite w.
__device__ __forceinline__ double quotient(double a, double w, double r) {
  const double q = a * r;
  return __double2hiint(w) == 0x7ff00000 ? q : fma(fma(-q, w, a), r, q);
}

// Cholesky factor of an n x n tile (n <= kB) by a warp: l holds the lower triangle of
// A and receives the factor, rec its reciprocal diagonal; lane r holds row r.  An entry
// is (A - sum) / L_jj with its sum formed apart and subtracted once: the sum over the
// columns before the tile (s, if SUMS) and over the tile's own.  Taking the products
// off A one by one rounds at the size of A every time and made covariances' inverses
// 2.4 times as wrong.  The loops end at n: the FP64 instructions of a column (root,
// reciprocal, products) are what a tile costs.  False: not positive definite.
template <bool SUMS>
__device__ __forceinline__ bool factor_tile(double (*l)[kB + 1], const double (*s)[kB + 1], int n,
                                            double* rec) {
  const int lane = threadIdx.x & 31;
  double sum[kB];
#pragma unroll
  for (int c = 0; c < kB; c++) sum[c] = 0.0;
#pragma unroll
  for (int j = 0; j < kB; j++) {
    if (j >= n) break;
    double v = 0.0;
    if (lane >= j && lane < n) v = l[lane][j] - (SUMS ? s[lane][j] + sum[j] : sum[j]);
    const double dj = __shfl_sync(0xffffffffu, v, j);
    if (!(dj > 0)) return false;
    const double lj = sqrt(dj), rj = 1 / lj;
    const double mine = lane > j ? quotient(v, lj, rj) : 0.0;
    if (lane >= j) l[lane][j] = lane == j ? lj : mine;
    if (lane == j) rec[j] = rj;
#pragma unroll
    for (int c = j + 1; c < kB; c++) {
      if (c >= n) break;
      sum[c] = fma(mine, __shfl_sync(0xffffffffu, mine, c), sum[c]);
    }
  }
  __syncwarp();
  return true;
}

// L x = e_c for lane c.
__device__ __forceinline__ void forward_tile(const double (*l)[kB + 1], const double* rec, int n,
                                             double (&x)[kB]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < kB; r++) {
    if (r >= n) break;
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < r; q++) t = fma(l[r][q], x[q], t);
    x[r] = quotient((r == lane ? 1.0 : 0.0) - t, l[r][r], rec[r]);
  }
}

// Inverse of a matrix of one tile or less by a warp: lane c solves for column c, and
// the two triangles are averaged.  20000 matrices of 2 x 2, 8 x 8 and 32 x 32: 0.18,
// 0.45 and 2.41 ms; by the kernels for several tiles, whose columns beyond the matrix
// cost as much as its own then, 1.80, 3.02 and 3.24, with a block per matrix 0.82,
// 2.57 and 14.3.
__device__ __forceinline__ void invert_small(double* A, int n, double (*l)[kB + 1], double* rec,
                                             int* status) {
  const int lane = threadIdx.x;
  for (int r = 0; r < n; r++) l[r][lane] = lane <= r ? A[r * n + lane] : 0.0;
  __syncwarp();
  if (!factor_tile<false>(l, nullptr, n, rec)) {
    if (lane == 0) *status = 1;
    return;
  }
  double x[kB];
  forward_tile(l, rec, n, x);
#pragma unroll
  for (int r = kB - 1; r >= 0; r--) {  // L^T x = y
    if (r >= n) continue;
    double t = 0.0;
#pragma unroll
    for (int q = r + 1; q < kB; q++) {
      if (q >= n) break;
      t = fma(l[q][r], x[q], t);
    }
    x[r] = quotient(x[r] - t, l[r][r], rec[r]);
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < kB; r++) {
    if (r >= n) break;
    l[r][lane] = x[r];
  }
  __syncwarp();
  if (lane < n)
    for (int r = 0; r < n; r++) A[r * n + lane] = 0.5 * (l[r][lane] + l[lane][r]);
}

__global__ void __launch_bounds__(32) k_invert_small(const InvertDesc* d, const int* full,
                                                     int* status, double* Aall) {
  __shared__ double l[kB][kB + 1], rec[kB];
  const int i = blockIdx.x;
  if (full[i]) invert_small(Aall + d[i].off, d[i].n, l, rec, status + i);
}

// Diagonal tile of panel k, a warp per matrix; S, the sums over the panels before,
// lies where the factor goes.  The first panel's launch inverts the small matrices.
__global__ void __launch_bounds__(32) k_chol_diag(const InvertDesc* d, const int* full, int* status,
                                                  double* Aall, double* Lall, double* Wall, int k) {
  __shared__ double l[kB][kB + 1], s[kB][kB + 1], rec[kB];
  const int i = blockIdx.x, lane = threadIdx.x;
  if (k == 0 && full[i] && d[i].n <= kB) {
    invert_small(Aall + d[i].off, d[i].n, l, rec, status + i);
    return;
  }
  Mat m;
  if (!mat_at(d, full, status, Lall, Wall, i, m)) return;
  const int base = k * kB;
  if (base >= m.n) return;
  const int nb = min(kB, m.n - base);
  const double* A = Aall + d[i].off + (long long)base * (m.n + 1);
  double* L = m.L + (long long)base * (m.n + 1);
  double* W = m.W + (long long)base * (m.n + 1);
#pragma unroll 16
  for (int r = 0; r < nb; r++) {
    l[r][lane] = lane <= r ? A[(long long)r * m.n + lane] : 0.0;
    s[r][lane] = lane <= r && k > 0 ? L[(long long)r * m.n + lane] : 0.0;
  }
  __syncwarp();
  if (!factor_tile<true>(l, s, nb, rec)) {
    if (lane == 0) status[i] = 1;
    return;
  }
  double x[kB];
  forward_tile(l, rec, nb, x);
  for (int r = 0; r < nb; r++)
    if (lane <= r) L[(long long)r * m.n + lane] = l[r][lane];
  if (lane < nb)
#pragma unroll
    for (int r = 0; r < kB; r++)
      if (r < nb && r >= lane) W[(long long)r * m.n + lane] = x[r];
}

// L_ik = (A - S)_ik L_kk^-T below the diagonal tile (L_kk^-1 in W; S, the sum over
// the panels before, where L_ik goes).
__global__ void __launch_bounds__(kT) k_chol_panel(const InvertDesc* d, const int* full,
                                                   const int* status, const double* Aall,
                                                   double* Lall, double* Wall, int k) {
  Mat m;
  if (!mat_at(d, full, status, Lall, Wall, blockIdx.y, m)) return;
  const int bi = k + 1 + (int)blockIdx.x;
  if (bi * kB >= m.n) return;
  __shared__ __align__(16) double a[kB][kPad], b[kB][kPad];
  const double* A = Aall + d[blockIdx.y].off;
  for (int e = threadIdx.x; e < kB * kB; e += kT) {  // a[q][i] = (A - S)_iq
    const int r = e / kB, c = e % kB, row = bi * kB + r;
    const long long g = (long long)row * m.n + k * kB + c;  // panel k lies whole in the matrix
    a[c][r] = row < m.n ? (k > 0 ? A[g] - m.L[g] : A[g]) : 0.0;
  }
  load_tile<true, true>(m.W, m.n, k, k, b);    // b[q][j] = (L_kk^-1)_jq
  __syncthreads();
  double acc[4][4] = {};
  tile_fma(a, b, acc);
  const int i0 = bi * kB + 4 * (threadIdx.x >> 3), j0 = k * kB + 4 * (threadIdx.x & 7);
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < 4; j++)
      if (i0 + i < m.n && j0 + j < m.n) m.L[(long long)(i0 + i) * m.n + j0 + j] = acc[i][j];
}

// Tile pair (ti, tj), ti >= tj, of the g-th entry of a lower triangle.
__device__ __forceinline__ void tri_pair(int g, int& ti, int& tj) {
  ti = (int)((sqrtf(8.f * g + 1.f) - 1.f) * 0.5f);
  while ((ti + 1) * (ti + 2) / 2 <= g) ti++;
  while (ti * (ti + 1) / 2 > g) ti--;
  tj = g - ti * (ti + 1) / 2;
}

// S_ij += L_ik L_jk^T for the tiles behind panel k (the first panel writes S).
__global__ void __launch_bounds__(kT) k_chol_update(const InvertDesc* d, const int* full,
                                                    const int* status, double* Lall, double* Wall,
                                                    int k) {
  Mat m;
  if (!mat_at(d, full, status, Lall, Wall, blockIdx.y, m)) return;
  int bi, bj;
  tri_pair((int)blockIdx.x, bi, bj);
  bi += k + 1;
  bj += k + 1;
  if (bi * kB >= m.n) return;
  __shared__ __align__(16) double a[kB][kPad], b[kB][kPad];
  load_tile<true, false>(m.L, m.n, bi, k, a);
  if (bi != bj) load_tile<true, false>(m.L, m.n, bj, k, b);
  __syncthreads();
  double acc[4][4] = {};
  tile_fma(a, bi != bj ? b : a, acc);
  const int i0 = bi * kB + 4 * (threadIdx.x >> 3), j0 = bj * kB + 4 * (threadIdx.x & 7);
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < 4; j++)
      if (i0 + i < m.n && j0 + j <= i0 + i) {
        double* p = m.L + (long long)(i0 + i) * m.n + j0 + j;
        *p = k > 0 ? *p + acc[i][j] : acc[i][j];
      }
}

// Block column j of W = L^-1: W_ij = -L_ii^-1 sum_(k=j..i-1) L_ik W_kj down
// the column (the diagonal tiles of W are there).  The long columns start
// first.
__global__ void __launch_bounds__(kT) k_tri_inverse(const InvertDesc* d, const int* full,
                                                    const int* status, double* Lall, double* Wall) {
  Mat m;
  if (!mat_at(d, full, status, Lall, Wall, blockIdx.x, m)) return;
  const int nt = (m.n + kB - 1) / kB, bj = (int)blockIdx.y;
  if (bj >= nt) return;
  __shared__ __align__(16) double a[kB][kPad], b[kB][kPad];
  const int i0 = 4 * (threadIdx.x >> 3), j0 = 4 * (threadIdx.x & 7);
  for (int bi = bj + 1; bi < nt; bi++) {
    double acc[4][4] = {};  // a tile's products apart, then the tiles: fewer roundings
    for (int k = bj; k < bi; k++) {
      double part[4][4] = {};
      __syncthreads();
      load_tile<true, false>(m.L, m.n, bi, k, a);  // a[q][i] = L_iq
      if (k == bj) load_tile<false, true>(m.W, m.n, k, bj, b);
      else load_tile<false, false>(m.W, m.n, k, bj, b);  // b[q][j] = W_qj
      __syncthreads();
      tile_fma(a, b, part);
      tile_add(acc, part);
    }
    __syncthreads();
    load_tile<true, true>(m.W, m.n, bi, bi, a);  // a[q][i] = (L_ii^-1)_iq
    for (int i = 0; i < 4; i++)
      for (int j = 0; j < 4; j++) b[i0 + i][j0 + j] = -acc[i][j];
    __syncthreads();
    double out[4][4] = {};
    tile_fma(a, b, out);
    for (int i = 0; i < 4; i++)
      for (int j = 0; j < 4; j++) {
        const int row = bi * kB + i0 + i, col = bj * kB + j0 + j;
        if (row < m.n && col < m.n) m.W[(long long)row * m.n + col] = out[i][j];
      }
  }
}

// Tiles (i, j) and (j, i) of A^-1 = W^T W: the rows of W from tile row i on.
__global__ void __launch_bounds__(kT) k_gram(const InvertDesc* d, const int* full,
                                             const int* status, double* Lall, double* Wall,
                                             double* A) {
  Mat m;
  if (!mat_at(d, full, status, Lall, Wall, blockIdx.y, m)) return;
  const int nt = (m.n + kB - 1) / kB;
  int bi, bj;
  tri_pair((int)blockIdx.x, bi, bj);
  if (bi >= nt) return;
  __shared__ __align__(16) double a[kB][kPad], b[kB][kPad];
  double acc[4][4] = {};
  for (int k = bi; k < nt; k++) {
    double part[4][4] = {};
    __syncthreads();
    if (k == bi) load_tile<false, true>(m.W, m.n, k, bi, a);
    else load_tile<false, false>(m.W, m.n, k, bi, a);
    if (bi != bj) load_tile<false, false>(m.W, m.n, k, bj, b);
    __syncthreads();
    tile_fma(a, bi != bj ? b : a, part);
    tile_add(acc, part);
  }
  double* out = A + d[blockIdx.y].off;
  const int i0 = bi * kB + 4 * (threadIdx.x >> 3), j0 = bj * kB + 4 * (threadIdx.x & 7);
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < 4; j++)
      if (i0 + i < m.n && j0 + j < m.n && j0 + j <= i0 + i) {
        out[(long long)(i0 + i) * m.n + j0 + j] = acc[i][j];
        out[(long long)(j0 + j) * m.n + i0 + i] = acc[i][j];
      }
}

}  // namespace

void matrix_invert_blocked(int nret, int nmax, const InvertDesc* d, const int* full, int* status,
                           double* A, double* L, double* W, cudaStream_t s) {
  if (nmax <= kB) {
    k_invert_small<<<nret, 32, 0, s>>>(d, full, status, A);
    return;
  }
  const int nt = (nmax + kB - 1) / kB;
  for (int k = 0; k < nt; k++) {
    const int below = nt - 1 - k;
    k_chol_diag<<<nret, 32, 0, s>>>(d, full, status, A, L, W, k);
    if (below > 0) {
      k_chol_panel<<<dim3(below, nret), kT, 0, s>>>(d, full, status, A, L, W, k);
      k_chol_update<<<dim3(below * (below + 1) / 2, nret), kT, 0, s>>>(d, full, status, L, W, k);
    }
  }
  k_tri_inverse<<<dim3(nret, nt - 1), kT, 0, s>>>(d, full, status, L, W);
  k_gram<<<dim3(nt * (nt + 1) / 2, nret), kT, 0, s>>>(d, full, status, L, W, A);
}

}  // namespace jgb
