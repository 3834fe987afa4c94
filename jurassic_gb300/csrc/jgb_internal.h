// Launch wrappers shared between the translation units of libjurassic_gb300.
#pragma once

#include <cuda_runtime.h>

#include "jgb_common.cuh"

struct jgb_ctx;
struct jgb_engine;

namespace jgb {

struct DevBuf;

// jgb_fp64.cu: ray tracing.  slopes: the level intervals' slopes
// (launch_level_slopes into level_slope_bytes) or nullptr, which forms them
// as the rays go
size_t level_slope_bytes(const CtlDev& c, long long nlev);
void launch_level_slopes(const CtlDev& c, const BatchDev& b, double* slopes, cudaStream_t s);
void launch_trace_count(const CtlDev& c, const BatchDev& b, const LosDev& L, const double* slopes,
                        unsigned* err, cudaStream_t s);
// jgb_fp64.cu: field-of-view convolution + BT + mask of pencil-beam results
void launch_fov(const CtlDev& c, const BatchDev& b, const double* prad, const double* ptau,
                int nfov, const double* fdz, const double* fw, const double* nu, unsigned* err,
                cudaStream_t s);
// jgb_trace_mixed.cu: ray tracing of the mixed-precision forward model
void launch_trace_count_mixed(const CtlDev& c, const BatchDev& b, const LosDev& L, unsigned* err,
                              cudaStream_t s);
void launch_trace_fill_mixed(const CtlDev& c, const BatchDev& b, const LosDev& L, const int* order,
                             unsigned* err, cudaStream_t s);
// Resumed tracing of finite-difference perturbations (EGA).  The fill of the
// base rays (the first nbase rays of the batch) keeps, per LOS point (indexed
// like the LOS planes, bpts points), the walk's FP64 position and direction,
// its raw segment length and its level interval.  A perturbed ray r then
// follows plan[r] = {base ray, m, mode}: mode 2 takes the base's geometry
// whole and recomputes the point values from its own profile (a perturbed
// mixing ratio or extinction: the step rule and refraction see z, p and T
// only; or a perturbed temperature whose levels the ray never comes near);
// mode 1 copies the base's points before m and walks on from the base's
// state at point m (a perturbed temperature, m before the first segment that
// comes near the perturbed levels); mode 0 walks from the start.  Every
// perturbed ray's LOS equals, bit for bit, what a walk from the start writes.
struct TraceResume {
  long long bpts;
  double* xs;        // [3][bpts] positions
  double* es;        // [3][bpts] directions
  float* dsr;        // [bpts] raw segment lengths
  int* lev;          // [bpts] level intervals
  const int4* plan;  // [nray] (perturbed rays)
};
// rays the fill kernel of the perturbed rays holds on the device at once
int trace_fill_resident(int sms);
// rays [r0, r0 + nr) (or order[0, nr)); role 1: the base rays (keep their
// walks in R), role 2: the perturbed rays (follow R.plan)
void launch_trace_fill_resumed(const CtlDev& c, const BatchDev& b, const LosDev& L,
                               const int* order, int r0, int nr, const TraceResume& R, int role,
                               unsigned* err, cudaStream_t s);
void launch_los_bound_mixed(const CtlDev& c, const BatchDev& b, double scale, int* cap,
                            cudaStream_t s);
void launch_trace_fill(const CtlDev& c, const BatchDev& b, const LosDev& L, const int* order,
                       const double* slopes, unsigned* err, cudaStream_t s);
void launch_path_fp64(const CtlDev& c, const TblDev& T, const ChanDev& ch, const BatchDev& b,
                      const LosDev& L, double* refl_scratch, cudaStream_t s);
void launch_srcfunc(int nd, int id0, int nch, const int* fn_off, const double* fnu,
                    const double* f, const double* st, double* sr, cudaStream_t s);
void launch_hydrostatic(const CtlDev& c, const BatchDev& b, double* p_out, cudaStream_t s);
// loads the kernels above onto the current device (JGB_OK or JGB_ERR_CUDA)
int preload_fp64_kernels();

// jgb_noalloc.cu: loads the allocation-free entry point's scratch array and
// kernels onto the device and resolves the array's address there (called by
// jgb_create with the device current; a failure is reported by the entry
// point's first call, which retries)
int noalloc_prepare(int device);

// jgb_mixed.cu
struct MixedPlan {
  int ntile;
  int* perm;            // [ntile*32]
  long long* toff;      // [ntile+1]
  float* data;          // tile planes
  int nfield;
  unsigned brmask;      // emitters with p-T brackets precomputed per LOS point
  bool fast;            // all of them, and no odd row in the tables
  // a chunk of the path (k_gas_m, k_seg_m, k_scan_m): tiles [tile0, tile1)
  // with pt0 = toff[tile0], channels [id0, id1); seg[((point * channels +
  // channel) * nseg + emitter) * 32 + lane] the segment emissivities, stop the
  // point where each (tile, channel, emitter, lane) saturates
  int tile0, tile1;
  long long pt0;
  int id0, id1;
  int nseg;
  float* seg;
  int* stop;
  const float* cloud;   // [nd][nray] cloud extinction (-0: no cloud), nullptr: no clouds
  // opaque rays (k_path_ends): sums along the rays of extinction x length per
  // window and of cloud factor x length ([nw + 1][nray], nullptr: neither), and
  // the points that a (tile, channel, lane) of the chunk walks (one lane per ray
  // only; nullptr otherwise)
  const float* ext_sum;
  int* ends;
  // Resumed forward models (finite-difference perturbations), for channels
  // [gid0, gid0 + gndc): ray r starts at LOS point start[r], where its path
  // equals its base ray's.  A base ray saves its state for the rays snap_ray[k]
  // before its point snap_ip[k], k in [snap_off[r], snap_off[r+1]): every
  // emitter's in snap[((ray * gndc + channel) * ng + emitter) * state words],
  // the sums in snap_sums[(ray * gndc + channel) * 3].  A perturbation of one
  // emitter's mixing ratio (or of an extinction) leaves the other emitters'
  // inputs and path states equal to the base's: a ray with reuse[r] = {base
  // ray, emitter} takes every emitter but that one (< 0: all) from its base's
  // segments, base_seg (entries base_nseg) and base_stop, laid out as seg and
  // stop over the base tiles, the base ray in tile and lane base_slot[ray].
  // nullptr start: no resume; nullptr reuse: nothing shared.
  int gid0, gndc;
  const int* start;
  const int* snap_off;
  const int* snap_ip;
  const int* snap_ray;
  unsigned* snap;
  float* snap_sums;
  const int2* reuse;
  const int* base_slot;
  const float* base_seg;
  const int* base_stop;
  int base_nseg;
  int gstep;  // perturbations: emitter g in entry g * gstep (0: a tile's one emitter)
};
int mixed_nfield(const CtlDev& c);
void launch_pack_tiles_n(const CtlDev& c, const TblDev& T, const LosDev& L, const MixedPlan& P,
                         long long total_tile_points, cudaStream_t s);
// the path of a chunk: the emitters' paths (lanes_per_ray 1 or 4; variant:
// the autotuner's choice for 1), then segments and sums; res 0, or 1 for the
// base rays and 2 (one lane per ray) for the perturbations of a resumed batch
int path_gas_variants();
void launch_gas_m(const CtlDev& c, const TblDev& T, const BatchDev& b, const LosDev& L,
                  const MixedPlan& P, int lanes_per_ray, int variant, int res, cudaStream_t s);
void launch_seg_scan_m(const CtlDev& c, const TblDev& T, const ChanDev& ch, const BatchDev& b,
                       const LosDev& L, const MixedPlan& P, int longest, int res, cudaStream_t s);
void launch_cloud_m(const CtlDev& c, const ChanDev& ch, const BatchDev& b, float* out,
                    cudaStream_t s);
// opaque rays of the mixed path: sums per ray, then P.ends of a chunk
void launch_ext_sums(const CtlDev& c, const LosDev& L, int nray, float* out, cudaStream_t s);
void launch_path_ends(const CtlDev& c, const TblDev& T, const ChanDev& ch, const BatchDev& b,
                      const LosDev& L, const MixedPlan& P, int res, cudaStream_t s);
// FP32 channel constants of the path
size_t chan_const_bytes(const CtlDev& c);
void launch_chan_consts(const CtlDev& c, const ChanDev& ch, float* out, cudaStream_t s);
// bytes of an emitter's saved path state
size_t gas_state_bytes();
void launch_src_to_float(int nd, const double* sr, float* srf, cudaStream_t s);
void launch_rowmeta(long long nrow, int tu, const int* nu, const float* u, const float* e, int cga,
                    float4* meta, float2* ue, int* any_odd, cudaStream_t s);

// jgb_retrieval.cu: frees an engine's device and pinned memory and unties
// it from its context (which is being destroyed); the handle then accepts
// only jgb_engine_destroy, every other call returns JGB_ERR_STATE
void engine_detach(jgb_engine* E);

// jgb_api.cu: read-only view of a context for entry points defined in other
// translation units.  Returns JGB_OK, or an error code with the context's
// message set when tables or source functions are missing.
struct CtxView {
  int device;
  cudaStream_t stream;
  CtlDev c;
  TblDev T;
  ChanDev ch;
};
int ctx_view(jgb_ctx* x, CtxView* out);  // fills *out; returns JGB_ERR_STATE if not ready

// jgb_normal.cu: batched normal-equation products on device buffers.
// Problems are concatenated (K blocks m_i x n_i, A blocks n_i x n_i, ...);
// sel (host, nullptr = all) picks the problems computed, the others' blocks
// are left untouched.  At most 65535 selected problems per call.  split: the
// operand blocks' buffer of the context whose stream s is.
int normal_equations_dev(int nret, const int* m, const int* n, const double* K, const double* w,
                         const double* dy, double* A, double* b, int precision, const int* sel,
                         void* desc_dev, DevBuf& split, cudaStream_t s);
size_t normal_desc_bytes(int nret);
int ctx_fail(jgb_ctx* x, int code, const char* msg);

// jgb_api.cu: reserves a buffer for which the path's workspaces of the context make
// room (fields: also tiles_data, while it holds nothing).
cudaError_t reserve_first(jgb_ctx* x, DevBuf& buf, size_t bytes, bool fields);

// The context's (recursive) lock for the duration of a public call: host
// threads may share a context, and their calls run one after another.
void ctx_lock(jgb_ctx* x);
void ctx_unlock(jgb_ctx* x);
struct CtxLock {
  jgb_ctx* x;
  explicit CtxLock(const jgb_ctx* c) : x(const_cast<jgb_ctx*>(c)) {
    if (x) ctx_lock(x);
  }
  ~CtxLock() {
    if (x) ctx_unlock(x);
  }
  CtxLock(const CtxLock&) = delete;
  CtxLock& operator=(const CtxLock&) = delete;
};

}  // namespace jgb
