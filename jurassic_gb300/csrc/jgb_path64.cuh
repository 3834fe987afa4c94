// FP64 path over tiles of 32 rays (jgb_path64.cu): a chunk of tiles and
// channels and its workspaces.
#pragma once

#include <cuda_runtime.h>

#include "jgb_common.cuh"

namespace jgb {

struct Path64 {
  const int* perm;        // [ntile * 32] ray of (tile, lane), -1 = empty lane
  const long long* toff;  // [ntile + 1] point offsets of the tiles
  int tile0, tile1;       // tiles of this chunk
  long long pt0;          // toff[tile0]
  int id0, id1;           // channels of this chunk
  unsigned shared;        // emitters whose p-T grids are the same for every channel
  int gref[kMaxG];        // a channel with a table of each such emitter
  double* fd;             // per-point fields (k_prep64)
  unsigned* fu;
  double* om;             // segment transmittance of every (point, channel, emitter, lane)
  double* se;             // {src eps, 1 - eps} of every (point, channel, lane)
  int* stop;              // point where (tile, channel, emitter, lane) saturates, else its count
};

// bytes of the per-point fields (32 lanes)
void path64_point_bytes(const CtlDev& c, size_t* fd, size_t* fu);
void launch_src_channel_major(int nd, const double* st, const double* sr, double2* srd,
                              cudaStream_t s);
// longest: points of the chunk's longest tile
void launch_prep64(const CtlDev& c, const TblDev& T, const LosDev& L, const Path64& P,
                   int longest, cudaStream_t s);
void launch_path64(const CtlDev& c, const TblDev& T, const ChanDev& ch, const BatchDev& b,
                   const LosDev& L, const Path64& P, int longest, int lanes_per_ray,
                   cudaStream_t s);

}  // namespace jgb
