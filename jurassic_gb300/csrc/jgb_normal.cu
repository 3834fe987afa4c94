// Normal-equation products of the optimal-estimation retrieval:
//   A = K^T W K  and  b = K^T W dy,   W = diag(w^2)
// (matrix_product, retrieval.c:403-444, and the gsl_blas_dgemv of
// retrieval.c:573-577), batched over retrievals of different sizes.
//
// Mixed precision: 3xTF32 on the 5th-generation tensor cores (tcgen05, FP32
// accumulators in tensor memory).  Every operand x = sqrt(W)K is split into
// a TF32 head and a TF32 residual (x = hi + lo); the product uses
// hi*hi + hi*lo + lo*hi with FP32 accumulation, which recovers ~FP32
// accuracy from TF32 inputs.  dy is appended to K as column n so that b is
// the last row of the same product.  Only the lower triangle of output
// tiles is computed; the upper one is mirrored.
//
// FP64: the same products on the FP64 pipes (the plain reference arithmetic).
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "../../include/jurassic_gb300.h"
#include "jgb_common.cuh"
#include "jgb_ctx.h"
#include "jgb_internal.h"

namespace jgb {

namespace {

constexpr int kTile = 128;  // output tile (kTile x kTile) per block
constexpr int kChunk = 16;  // rows of X per shared-memory stage
constexpr int kPlaneBytes = kTile * kChunk * 4;  // one operand plane of a stage (8 KB)
constexpr int kBlockFloats = 2 * kTile * kChunk;   // head + residual plane of one (tile, chunk)
constexpr int kStageBytes = 4 * kPlaneBytes;     // A hi, A lo, B hi, B lo
constexpr int kStages = 2;                       // operand stages in flight
constexpr int kStageArea = kStages * kStageBytes;             // 64 KB
constexpr int kEpiCols = kTile / 2;                           // columns per epilogue pass
constexpr int kEpiPad = kEpiCols + 4;  // staging row stride: 16-byte rows, no bank conflicts
constexpr int kStileFloats = kTile * kEpiPad;                 // epilogue staging tile
constexpr int kBarOff = kStageArea + kStileFloats * 4;        // mbarriers
constexpr int kNumBars = 2 * kStages + 4;        // full, empty, accumulator full / empty
constexpr int kTcSmem = kBarOff + kNumBars * 8 + 16;          // + TMEM address
constexpr int kEpiThreads = 512;                 // sixteen epilogue warps
constexpr int kNeThreads = 64 + kEpiThreads;     // + copy warp, MMA warp

struct NeDesc {
  int m, n;                 // rows of K, columns of K (state size)
  long long koff, moff, aoff, boff;
  long long xoff;           // offset (floats) of the problem's operand blocks
  long long tile0;          // index of the problem's first output tile
};

__device__ __forceinline__ unsigned tf32_of(float x) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Byte offset of element (row, k) in a 128 x kChunk K-major operand plane of
// 8-row x 16-byte core matrices: [k / 8][row / 8][k % 8 / 4][row % 8][k % 4];
// one MMA (K = 8 TF32) reads a [row / 8][2 core matrices] slice of 4 KB.
__device__ __forceinline__ int tc_off(int row, int k) {
  return (k >> 3) * 4096 + (row >> 3) * 256 + ((k & 7) >> 2) * 128 + (row & 7) * 16 + (k & 3) * 4;
}

// Shared-memory matrix descriptor of such a slice (no swizzle): start
// address >> 4, leading byte offset 128 (the two core matrices along K),
// stride byte offset 256 (8-row groups), descriptor version 0b001 at bit 46.
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(128u >> 4) << 16) |
         ((uint64_t)(256u >> 4) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of kind::tf32: FP32 accumulator, TF32 A and B, both
// K-major, N = M = kTile.
constexpr uint32_t kTcIdesc = (1u << 4) | (2u << 7) | (2u << 10) |
                              ((uint32_t)(kTile >> 3) << 17) | ((uint32_t)(kTile >> 4) << 24);

__device__ __forceinline__ void tc_mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(kTcIdesc), "r"(acc));
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr unsigned long long kWaitLimitNs = 1000000000ull;  // one second

// Bounded wait for phase `parity` of an mbarrier: gives up after about a
// second of the global timer (checked every 64 polls; a poll may suspend the
// thread for a while), or after 2^30 polls should the timer not advance.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  const unsigned long long t0 = global_ns();
  for (int it = 0; it < (1 << 30); it++) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((it & 63) == 63 && global_ns() - t0 > kWaitLimitNs) return false;
  }
  return false;
}

// Self-test of mbar_wait: one thread initialises an mbarrier for one
// arrival and waits for its first phase; with arrive != 0 it arrives first
// (the wait succeeds at once), otherwise nothing ever arrives and the wait
// must give up.  Records the outcome and the waiting time.
__global__ void k_wait_selftest(int arrive, unsigned long long* out) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x != 0) return;
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar)));
  asm volatile("fence.mbarrier_init.release.cluster;");
  if (arrive)
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bar)) : "memory");
  const unsigned long long t0 = global_ns();
  const bool ok = mbar_wait(smem_u32(&bar), 0);
  out[0] = ok ? 0ull : 1ull;
  out[1] = global_ns() - t0;
}

// X = sqrt(W)[K | dy] of every problem, formed once in FP64 and split into
// a TF32 high part and a TF32-rounded remainder, written in the operand
// layout of the tensor-core product: per (column tile ti, chunk c of kChunk
// rows) one block of kBlockFloats, the head plane then the residual plane,
// each 128 columns x kChunk rows in the core-matrix order of tc_off, zero
// outside m x (n + 1).  Block bi = ti * nch + c of a problem starts at
// xoff + bi * kBlockFloats (16 KB apart: whole blocks go to shared memory
// with one bulk copy).  A thread takes a column of a block: its kChunk loads,
// lanes along a row, are in flight together, and four rows of a column are 16
// bytes of a plane, eight columns' 128 bytes, so the stores go straight to
// memory.  512 problems of 150 x 405: 63 us (0.5 GB, 47 us at the
// measured bandwidth); assembled in shared memory by 4-byte stores, with two
// barriers per block, 97 us.
__global__ void __launch_bounds__(128) k_split_x(const NeDesc* desc, const double* Kall,
                                                 const double* wall, const double* dyall,
                                                 float* xbuf) {
  const NeDesc d = desc[blockIdx.y];
  const int na = d.n + 1;
  const int nt = (na + kTile - 1) / kTile, nch = (d.m + kChunk - 1) / kChunk;
  const int tid = threadIdx.x;
  for (int bi = blockIdx.x; bi < nt * nch; bi += gridDim.x) {
    const int ti = bi / nch, c = bi - ti * nch;
    const int col = ti * kTile + tid, row0 = c * kChunk;
    // column n of the augmented matrix is dy, contiguous
    const double* src = col < d.n ? Kall + d.koff + (long long)row0 * d.n + col : dyall + d.moff + row0;
    const int step = col < d.n ? d.n : 1;
    const double* w = wall + d.moff + row0;
    const int nrow = col < na ? min(d.m - row0, kChunk) : 0;
    double v[kChunk];
#pragma unroll
    for (int k = 0; k < kChunk; k++) v[k] = k < nrow ? src[(long long)k * step] : 0.0;
    float* dst = xbuf + d.xoff + (long long)bi * kBlockFloats;
#pragma unroll
    for (int k = 0; k < kChunk; k += 4) {
      float hi[4], lo[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float x = k + j < nrow ? d2f_bits(v[k + j] * w[k + j]) : 0.f;
        hi[j] = __uint_as_float(tf32_of(x));
        lo[j] = __uint_as_float(tf32_of(x - hi[j]));
      }
      const int o = tc_off(tid, k) >> 2;
      *reinterpret_cast<float4*>(dst + o) = make_float4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<float4*>(dst + kTile * kChunk + o) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}

// Output tile g of the concatenated lower-triangular tile lists: problem
// (last with tile0 <= g) and tile pair (ti, tj), ti >= tj.
__device__ __forceinline__ int tile_of(const NeDesc* desc, int nsel, long long g, int& ti,
                                       int& tj) {
  int lo = 0, hi = nsel - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (desc[mid].tile0 <= g) lo = mid; else hi = mid - 1;
  }
  int t = (int)(g - desc[lo].tile0);
  ti = 0;
  while (t > ti) {
    t -= ti + 1;
    ti++;
  }
  tj = t;
  return lo;
}

// AND of a flag over the epilogue warps (named barrier 1): all of them take
// the same branch after it.
__device__ __forceinline__ bool epi_all(bool v) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, 1, %2, p;\n"
      " selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "n"(kEpiThreads)
      : "memory");
  return r != 0;
}

__device__ __forceinline__ void epi_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
}

// C = X^T X over the augmented columns for every output tile of every
// problem, as a persistent kernel: one CTA per SM walks tiles blockIdx.x,
// blockIdx.x + gridDim.x, ... with three roles that meet only at mbarriers.
//  * copy warp (one lane): per chunk of kChunk rows, bulk copies of the
//    operand blocks (already in the core-matrix layout; B = A on a diagonal
//    tile) into one of kStages stages, completing on the stage's "full"
//    barrier, after the stage's "empty" barrier says its MMAs are done;
//  * MMA warp (one lane; it also owns the tensor memory): the 3 x 2
//    tcgen05.mma of each chunk (3xTF32: lo*hi + hi*lo + hi*hi) into one of
//    two 128 x 128 FP32 accumulators in tensor memory, committed to the
//    stage's "empty" barrier, and after a tile's last chunk to the
//    accumulator's "full" barrier;
//  * sixteen epilogue warps, four per tensor-memory lane quarter (warp w
//    reads lanes 32 (w % 4) ...), in two passes of 64 columns, 16 columns
//    per warp and pass: tcgen05.ld of the accumulator, mirrored FP64 entries
//    written straight from registers (lanes along a column of the upper
//    triangle), the direct entries through a shared staging tile with lanes
//    along rows; after the second pass's loads the accumulator is handed
//    back ("empty").
// So the copies, the MMAs of one tile and the epilogue of the previous one
// overlap.  The epilogue sets the pace (without its stores the kernel runs
// in about half the time, and four stages instead of two change nothing; with
// two columns per lane in the direct entries, half a sector per store, 512
// problems of 150 x 405 took 185 us, 152 now), so
// the CTA keeps two stages and a 64-column staging tile, 97 KB of shared
// memory, and two CTAs share an SM (32 epilogue warps, all 512 columns of
// tensor memory).  Every wait is bounded; one that gives up flags the error, the
// epilogue warps leave together (epi_all), the copy lane waits (bounded) for
// its copies in flight and the MMA lane for its last commit, and the tensor
// memory is freed.
__global__ void __launch_bounds__(kNeThreads, 2) k_normal_tc(const NeDesc* desc, int nsel,
                                                             long long ntiles, const float* xbuf,
                                                             double* Aall, double* ball,
                                                             unsigned* err) {
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint64_t* full = reinterpret_cast<uint64_t*>(tc_smem + kBarOff);  // [kStages]
  uint64_t* empty = full + kStages;                                  // [kStages]
  uint64_t* acc_full = empty + kStages;                              // [2]
  uint64_t* acc_empty = acc_full + 2;                                // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tc_smem + kBarOff + kNumBars * 8);
  float* stile = reinterpret_cast<float*>(tc_smem + kStageArea);     // [kTile][kEpiPad]
  if (tid == 0) {
    for (int i = 0; i < 2 * kStages + 2; i++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[i])));
    for (int i = 0; i < 2; i++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&acc_empty[i])),
                   "r"(kEpiThreads));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(2 * kTile));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  const uint32_t sbase = smem_u32(tc_smem);
  bool ok = true;

  if (warp == 0 && lane == 0) {  // copies
    long long it = 0;  // chunks issued by this CTA
    for (long long g = blockIdx.x; g < ntiles && ok; g += gridDim.x) {
      int ti, tj;
      const NeDesc d = desc[tile_of(desc, nsel, g, ti, tj)];
      const int nch = (d.m + kChunk - 1) / kChunk;
      const bool diag = ti == tj;
      const float* XA = xbuf + d.xoff + (long long)ti * nch * kBlockFloats;
      const float* XB = xbuf + d.xoff + (long long)tj * nch * kBlockFloats;
      const uint32_t bytes = diag ? 2u * kPlaneBytes : 4u * kPlaneBytes;
      for (int c = 0; c < nch; c++) {
        const int st = (int)(it % kStages);
        const uint32_t ph = (uint32_t)((it / kStages) & 1);
        if (!mbar_wait(smem_u32(&empty[st]), ph ^ 1u)) {  // a fresh stage passes at once
          ok = false;
          break;
        }
        const uint32_t fb = smem_u32(&full[st]);
        const uint32_t dst = sbase + st * kStageBytes;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(bytes)
                     : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                dst),
            "l"(XA + (long long)c * kBlockFloats), "r"(2 * kPlaneBytes), "r"(fb)
            : "memory");
        if (!diag)
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                  dst + 2 * kPlaneBytes),
              "l"(XB + (long long)c * kBlockFloats), "r"(2 * kPlaneBytes), "r"(fb)
              : "memory");
        it++;
      }
    }
    // the last copy of every stage has landed before the CTA exits
    for (int st = 0; st < kStages; st++)
      if (it > st) {
        const long long last = st + ((it - 1 - st) / kStages) * kStages;
        mbar_wait(smem_u32(&full[st]), (uint32_t)((last / kStages) & 1));
      }
  } else if (warp == 1 && lane == 0) {  // MMAs
    long long it = 0;
    int lt = 0;
    uint32_t last_bar = 0, last_par = 0;  // barrier and phase of the last commit
    for (long long g = blockIdx.x; g < ntiles && ok; g += gridDim.x, lt++) {
      int ti, tj;
      const NeDesc d = desc[tile_of(desc, nsel, g, ti, tj)];
      const int nch = (d.m + kChunk - 1) / kChunk;
      const bool diag = ti == tj;
      const int acc = lt & 1;
      if (!mbar_wait(smem_u32(&acc_empty[acc]), (uint32_t)((lt >> 1) & 1) ^ 1u)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t dt = tmem + (uint32_t)(acc * kTile);
      for (int c = 0; c < nch; c++, it++) {
        const int st = (int)(it % kStages);
        const uint32_t ph = (uint32_t)((it / kStages) & 1);
        if (!mbar_wait(smem_u32(&full[st]), ph)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t a0 = sbase + st * kStageBytes;
        const uint32_t b0 = diag ? a0 : a0 + 2 * kPlaneBytes;
#pragma unroll
        for (int s = 0; s < kChunk / 8; s++) {
          const uint64_t ah = tc_desc(a0 + s * 4096), al = tc_desc(a0 + kPlaneBytes + s * 4096);
          const uint64_t bh = tc_desc(b0 + s * 4096), bl = tc_desc(b0 + kPlaneBytes + s * 4096);
          tc_mma(dt, al, bh, (c | s) != 0);
          tc_mma(dt, ah, bl, 1u);
          tc_mma(dt, ah, bh, 1u);
        }
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_u32(&empty[st])));
        last_bar = smem_u32(&empty[st]);
        last_par = ph;
      }
      if (!ok) break;
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              smem_u32(&acc_full[acc])));
      last_bar = smem_u32(&acc_full[acc]);
      last_par = (uint32_t)((lt >> 1) & 1);
    }
    // every MMA issued is complete before the tensor memory can be freed
    if (last_bar && !mbar_wait(last_bar, last_par)) ok = false;
  } else if (warp >= 2) {  // epilogue
    const int q = warp & 3;          // tensor-memory lane quarter of this warp
    const int r = q * 32 + lane;     // accumulator row (tile-local column ti of X)
    const int ew = warp - 2;         // 0 .. 15
    const int cq = (ew >> 2) * 16;   // this warp's 16 columns within a pass
    int lt = 0;
    for (long long g = blockIdx.x; g < ntiles; g += gridDim.x, lt++) {
      int ti, tj;
      const NeDesc d = desc[tile_of(desc, nsel, g, ti, tj)];
      const int acc = lt & 1;
      const bool w = mbar_wait(smem_u32(&acc_full[acc]), (uint32_t)((lt >> 1) & 1));
      if (!epi_all(w)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      double* A = Aall + d.aoff;
      double* bv = ball + d.boff;
      const int row = ti * kTile + r;
      const bool mrow = row < d.n;
      for (int h = 0; h < 2; h++) {
        const int c0 = h * kEpiCols + cq;  // accumulator columns c0 ... c0 + 15
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
              "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * kTile + c0)));
        asm volatile("tcgen05.wait::ld.sync.aligned;");
        if (h == 1) {  // accumulator read: hand it back to the MMA warp
          asm volatile("tcgen05.fence::before_thread_sync;");
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[acc]))
                       : "memory");
        }
        float4* srow = reinterpret_cast<float4*>(stile + r * kEpiPad + cq);
#pragma unroll
        for (int k = 0; k < 4; k++)
          srow[k] = make_float4(__uint_as_float(v[4 * k]), __uint_as_float(v[4 * k + 1]),
                                __uint_as_float(v[4 * k + 2]), __uint_as_float(v[4 * k + 3]));
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const int col = tj * kTile + c0 + j;
          // mirrored entry (col, row) of the upper triangle: lanes along rows
          if (mrow && col < row && col < d.n)
            A[(long long)col * d.n + row] = f2d_bits(__uint_as_float(v[j]));
        }
        epi_sync();
        // direct entries, rows >= columns (and b, the augmented row n): lanes
        // along the row, so that a store covers whole sectors
        const int col0 = tj * kTile + h * kEpiCols;
        const int rows = col0 < d.n ? min(kTile, d.n + 1 - ti * kTile) : 0;
        for (int rr = ew; rr < rows; rr += kEpiThreads / 32) {
          const int row2 = ti * kTile + rr;
          double* dst = row2 == d.n ? bv : A + (long long)row2 * d.n;
#pragma unroll
          for (int k = 0; k < kEpiCols; k += 32) {
            const int col = col0 + k + lane;
            if (col < d.n && col <= row2) dst[col] = f2d_bits(stile[rr * kEpiPad + k + lane]);
          }
        }
        epi_sync();  // the staging tile is free for the next pass
      }
    }
  }
  if (!ok) atomicOr(err, 1u);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kTile));
}

// FP64 products, A = (w K)^T (w K) and b = K^T (w^2 dy), summed over the rows in
// the order of matrix_product.  A block takes a 32 x 32 tile of the lower
// triangle, a thread 2 x 2 entries; the rows come 32 at a time through shared
// memory, already weighted, so that a term is one multiply-add (a thread per
// entry formed both weighted factors for every term, four FP64 instructions, and
// read them from L2).  The tile is small so that one problem of 405 elements
// still spreads over the SMs (91 blocks).  The blocks behind the tiles take b, a
// thread per element.  512 problems of up to 150 x 405 take 7.5
// ms instead of 28.0, one 0.074 instead of 0.175 (bound by the FP64 pipe).
// Problems of up to kNe64 columns take k_normal_fp64_small.
constexpr int kNe64 = 32, kNe64Threads = 256;

__global__ void __launch_bounds__(kNe64Threads) k_normal_fp64(const NeDesc* desc, const double* Kall,
                                                              const double* wall, const double* dyall,
                                                              double* Aall, double* ball) {
  __shared__ double xi[kNe64][kNe64 + 1], xj[kNe64][kNe64 + 1];
  const NeDesc d = desc[blockIdx.y];
  if (d.n <= kNe64) return;
  const int nt = (d.n + kNe64 - 1) / kNe64, ntri = nt * (nt + 1) / 2;
  const int nb = (d.n + kNe64Threads - 1) / kNe64Threads, tid = threadIdx.x;
  const double* K = Kall + d.koff;
  const double* w = wall + d.moff;
  for (int tile = blockIdx.x; tile < ntri + nb; tile += gridDim.x) {
    if (tile >= ntri) {
      const int j = (tile - ntri) * kNe64Threads + tid;
      const double* dy = dyall + d.moff;
      double s = 0;
      if (j < d.n) {
        for (int k = 0; k < d.m; k++) s += K[(long long)k * d.n + j] * (dy[k] * (w[k] * w[k]));
        ball[d.boff + j] = s;
      }
      continue;
    }
    int ti = 0, tj = tile;
    while (tj > ti) tj -= ++ti;
    const int tx = tid & 15, ty = tid >> 4;
    double s[2][2] = {};
    for (int k0 = 0; k0 < d.m; k0 += kNe64) {
      __syncthreads();
      for (int e = tid; e < kNe64 * kNe64; e += kNe64Threads) {
        const int k = k0 + (e >> 5), c = e & 31, ci = ti * kNe64 + c, cj = tj * kNe64 + c;
        const double wk = k < d.m ? w[k] : 0.0;
        xi[e >> 5][c] = k < d.m && ci < d.n ? wk * K[(long long)k * d.n + ci] : 0.0;
        xj[e >> 5][c] = k < d.m && cj < d.n ? wk * K[(long long)k * d.n + cj] : 0.0;
      }
      __syncthreads();
      const int kn = min(kNe64, d.m - k0);
      for (int k = 0; k < kn; k++) {
        const double a0 = xi[k][ty], a1 = xi[k][ty + 16], b0 = xj[k][tx], b1 = xj[k][tx + 16];
        s[0][0] = fma(a0, b0, s[0][0]);
        s[0][1] = fma(a0, b1, s[0][1]);
        s[1][0] = fma(a1, b0, s[1][0]);
        s[1][1] = fma(a1, b1, s[1][1]);
      }
    }
    double* A = Aall + d.aoff;
    for (int p = 0; p < 2; p++)
      for (int q = 0; q < 2; q++) {
        const int i = ti * kNe64 + ty + 16 * p, j = tj * kNe64 + tx + 16 * q;
        if (i < d.n && j <= i) {
          A[(long long)i * d.n + j] = s[p][q];
          A[(long long)j * d.n + i] = s[p][q];
        }
      }
  }
}

// The same for problems of one tile or less: a block per problem, a thread per entry
// of the lower triangle and of b, so that few columns cost few multiply-adds (the
// tile above forms all 1024).  Rows of [w K | K | w^2 dy] come kNe64 at a time
// through shared memory.  1000 problems of 300 x 8 and 3000 x 3: 0.11 and 0.64 ms; in
// tiles 0.69 and 6.57, with a thread per entry that read both factors from L2 0.27
// and 1.63.  At the line: 200 x 32 here 0.23, 200 x 33 in tiles 0.70.
__host__ __device__ inline int small_entries(int n) { return n * (n + 1) / 2 + n; }

__global__ void k_normal_fp64_small(const NeDesc* desc, const double* Kall, const double* wall,
                                    const double* dyall, double* Aall, double* ball) {
  __shared__ double rows[kNe64 * (2 * kNe64 + 1)];
  const NeDesc d = desc[blockIdx.x];
  const int n = d.n, tid = threadIdx.x, stride = 2 * n + 1;
  if (n > kNe64) return;
  const double* K = Kall + d.koff;
  const double* w = wall + d.moff;
  const double* dy = dyall + d.moff;
  const int ntri = n * (n + 1) / 2;
  int i = (int)((sqrtf(8.f * tid + 1.f) - 1.f) * 0.5f);
  if ((i + 1) * (i + 2) / 2 <= tid) i++;
  if (i * (i + 1) / 2 > tid) i--;
  const int j = tid < ntri ? tid - i * (i + 1) / 2 : tid - ntri;
  double s = 0;
  for (int k0 = 0; k0 < d.m; k0 += kNe64) {
    const int kn = min(kNe64, d.m - k0);
    __syncthreads();
    for (int e = tid; e < kn * n; e += blockDim.x) {
      const int k = e / n, c = e - k * n;
      const double v = K[(long long)k0 * n + e];
      rows[k * stride + c] = w[k0 + k] * v;
      rows[k * stride + n + c] = v;
    }
    for (int k = tid; k < kn; k += blockDim.x)
      rows[k * stride + 2 * n] = dy[k0 + k] * (w[k0 + k] * w[k0 + k]);
    __syncthreads();
    if (tid < ntri)
      for (int k = 0; k < kn; k++) s = fma(rows[k * stride + i], rows[k * stride + j], s);
    else if (tid < ntri + n)
      for (int k = 0; k < kn; k++) s += rows[k * stride + n + j] * rows[k * stride + 2 * n];
  }
  if (tid < ntri) {
    double* A = Aall + d.aoff;
    A[i * n + j] = s;
    A[j * n + i] = s;
  } else if (tid < ntri + n) {
    ball[d.boff + j] = s;
  }
}

}  // namespace

int normal_equations_dev(int nret, const int* m, const int* n, const double* K, const double* w,
                         const double* dy, double* A, double* b, int precision, const int* sel,
                         void* desc_dev, DevBuf& split, cudaStream_t s) {
  // descriptors of the selected problems (host -> device scratch provided by
  // the caller); offsets follow the concatenation of all nret problems
  // (one more entry holds the tensor-core kernel's error word)
  std::vector<NeDesc> hd(nret + 1);
  long long ko = 0, mo = 0, ao = 0, bo = 0, xo = 0, ntiles = 0;
  int maxn = 0, maxsmall = 0, maxblk = 0, nsel = 0;  // maxsmall: largest n up to kNe64
  for (int i = 0; i < nret; i++) {
    if (!sel || sel[i]) {
      hd[nsel++] = NeDesc{m[i], n[i], ko, mo, ao, bo, xo, ntiles};
      const int nt = (n[i] + 1 + kTile - 1) / kTile;
      const int nblk = nt * ((m[i] + kChunk - 1) / kChunk);
      xo += (long long)nblk * kBlockFloats;
      ntiles += (long long)nt * (nt + 1) / 2;
      maxblk = nblk > maxblk ? nblk : maxblk;
      maxn = n[i] > maxn ? n[i] : maxn;
      if (n[i] <= kNe64) maxsmall = n[i] > maxsmall ? n[i] : maxsmall;
    }
    ko += (long long)m[i] * n[i];
    mo += m[i];
    ao += (long long)n[i] * n[i];
    bo += n[i];
  }
  if (nsel == 0) return JGB_OK;
  if (nsel > 65535) return JGB_ERR_ARG;
  hd[nsel] = NeDesc{};
  // pageable memory: staged by the time the call returns
  if (cudaMemcpyAsync(desc_dev, hd.data(), sizeof(NeDesc) * (nsel + 1), cudaMemcpyHostToDevice, s) !=
      cudaSuccess)
    return JGB_ERR_CUDA;
  if (precision == JGB_MIXED) {
    // operand blocks in the context's buffer (its calls run one after another)
    if (split.reserve(sizeof(float) * (size_t)xo) != cudaSuccess) return JGB_ERR_CUDA;
    float* xbuf = split.as<float>();
    const NeDesc* dd = static_cast<const NeDesc*>(desc_dev);
    k_split_x<<<dim3((unsigned)(maxblk < 4096 ? maxblk : 4096), nsel), 128, 0, s>>>(dd, K, w, dy,
                                                                                      xbuf);
    cudaFuncSetAttribute(k_normal_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem);
    unsigned* err = reinterpret_cast<unsigned*>(static_cast<NeDesc*>(desc_dev) + nsel);
    // persistent: two CTAs per SM (or one per tile when there are fewer)
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      return JGB_ERR_CUDA;
    const unsigned grid = (unsigned)(ntiles < 2LL * sms ? ntiles : 2LL * sms);
    k_normal_tc<<<grid, kNeThreads, kTcSmem, s>>>(dd, nsel, ntiles, xbuf, A, b, err);
    unsigned herr = 0;
    cudaMemcpyAsync(&herr, err, sizeof(herr), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess || herr) return JGB_ERR_CUDA;
  } else {
    const NeDesc* dd = static_cast<const NeDesc*>(desc_dev);
    if (maxsmall > 0)
      k_normal_fp64_small<<<nsel, (small_entries(maxsmall) + 31) / 32 * 32, 0, s>>>(dd, K, w, dy, A, b);
    if (maxn > kNe64) {
      const long long nt = (maxn + kNe64 - 1) / kNe64;
      const long long nblk = nt * (nt + 1) / 2 + (maxn + kNe64Threads - 1) / kNe64Threads;
      dim3 grid((unsigned)(nblk < 4096 ? nblk : 4096), nsel);
      k_normal_fp64<<<grid, kNe64Threads, 0, s>>>(dd, K, w, dy, A, b);
    }
  }
  return cudaGetLastError() == cudaSuccess ? JGB_OK : JGB_ERR_CUDA;
}

size_t normal_desc_bytes(int nret) { return sizeof(NeDesc) * ((size_t)nret + 1); }

int wait_selftest(int device, int arrive, int* timed_out, double* seconds) {
  if (!timed_out || !seconds) return JGB_ERR_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return JGB_ERR_CUDA;
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 2 * sizeof(unsigned long long)) != cudaSuccess) return JGB_ERR_CUDA;
  unsigned long long h[2] = {2, 0};
  k_wait_selftest<<<1, 32>>>(arrive, d);
  int rc = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess &&
                   cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) == cudaSuccess
               ? JGB_OK
               : JGB_ERR_CUDA;
  cudaFree(d);
  *timed_out = (int)h[0];
  *seconds = (double)h[1] * 1e-9;
  return rc;
}

}  // namespace jgb

using namespace jgb;

extern "C" int jgb_selftest_bounded_wait(int device, int arrive, int* timed_out, double* seconds) {
  return wait_selftest(device, arrive, timed_out, seconds);
}

// Host-buffer entry point: copies in, computes, copies out.
extern "C" int jgb_normal_equations(jgb_ctx* x, int nret, const int* m, const int* n,
                                    const double* K, const double* w, const double* dy,
                                    double* A, double* b, int precision) {
  jgb::CtxLock lock(x);
  if (!x || nret <= 0 || !m || !n || !K || !w || !dy || !A || !b)
    return ctx_fail(x, JGB_ERR_ARG, "bad arguments");
  CtxView v;
  int rc = ctx_view(x, &v);  // tables are not needed here: only device and stream
  if (rc != JGB_OK && rc != JGB_ERR_STATE) return rc;
  cudaSetDevice(v.device);
  long long sk = 0, sm = 0, sa = 0, sb = 0;
  for (int i = 0; i < nret; i++) {
    if (m[i] <= 0 || n[i] <= 0) return ctx_fail(x, JGB_ERR_ARG, "empty retrieval");
    sk += (long long)m[i] * n[i];
    sm += m[i];
    sa += (long long)n[i] * n[i];
    sb += n[i];
  }
  void* buf = nullptr;
  const size_t bytes = sizeof(double) * (size_t)(sk + 2 * sm + sa + sb) + normal_desc_bytes(nret) + 64;
  if (cudaMalloc(&buf, bytes) != cudaSuccess) return ctx_fail(x, JGB_ERR_CUDA, "cudaMalloc failed");
  double* dK = static_cast<double*>(buf);
  double* dw = dK + sk;
  double* ddy = dw + sm;
  double* dA = ddy + sm;
  double* db = dA + sa;
  void* ddesc = db + sb;
  cudaStream_t s = v.stream;
  cudaMemcpyAsync(dK, K, sizeof(double) * sk, cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(dw, w, sizeof(double) * sm, cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(ddy, dy, sizeof(double) * sm, cudaMemcpyHostToDevice, s);
  rc = normal_equations_dev(nret, m, n, dK, dw, ddy, dA, db, precision, nullptr, ddesc, x->ne_split, s);
  if (rc == JGB_OK) {
    cudaMemcpyAsync(A, dA, sizeof(double) * sa, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(b, db, sizeof(double) * sb, cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) rc = JGB_ERR_CUDA;
  }
  cudaFree(buf);
  return rc ? ctx_fail(x, rc, "normal-equation kernel failed") : JGB_OK;
}

// Device-buffer entry point: K, w, dy, A, b on the device, m and n on the
// host; runs on the context's stream and returns when the products are
// done.  *kernel_ms (optional) receives the CUDA-event time of the kernel.
extern "C" int jgb_normal_equations_dev(jgb_ctx* x, int nret, const int* m, const int* n,
                                        const double* K, const double* w, const double* dy,
                                        double* A, double* b, int precision, float* kernel_ms) {
  jgb::CtxLock lock(x);
  if (!x || nret <= 0 || !m || !n || !K || !w || !dy || !A || !b)
    return ctx_fail(x, JGB_ERR_ARG, "bad arguments");
  if (nret > 65535) return ctx_fail(x, JGB_ERR_ARG, "at most 65535 problems per call");
  CtxView v;
  int rc = ctx_view(x, &v);
  if (rc != JGB_OK && rc != JGB_ERR_STATE) return rc;
  cudaSetDevice(v.device);
  for (int i = 0; i < nret; i++)
    if (m[i] <= 0 || n[i] <= 0) return ctx_fail(x, JGB_ERR_ARG, "empty retrieval");
  // descriptors in the context's buffer, under its lock
  if (x->ne_desc.reserve(normal_desc_bytes(nret)) != cudaSuccess)
    return ctx_fail(x, JGB_ERR_CUDA, "cudaMalloc failed");
  void* ddesc = x->ne_desc.p;
  cudaEvent_t e0 = x->ev[0], e1 = x->ev[1];
  cudaStream_t s = v.stream;
  rc = normal_equations_dev(nret, m, n, K, w, dy, A, b, precision, nullptr, ddesc, x->ne_split, s);
  // time a second identical call only when asked: the first one may have grown
  // the buffers
  if (rc == JGB_OK && kernel_ms) {
    cudaEventRecord(e0, s);
    rc = normal_equations_dev(nret, m, n, K, w, dy, A, b, precision, nullptr, ddesc, x->ne_split, s);
    cudaEventRecord(e1, s);
  }
  if (cudaStreamSynchronize(s) != cudaSuccess) rc = JGB_ERR_CUDA;
  if (x->ne_split.n > x->path_limit) x->ne_split.release();  // large scratch is not kept
  if (rc == JGB_OK && kernel_ms) cudaEventElapsedTime(kernel_ms, e0, e1);
  return rc ? ctx_fail(x, rc, "normal-equation kernel failed") : JGB_OK;
}
