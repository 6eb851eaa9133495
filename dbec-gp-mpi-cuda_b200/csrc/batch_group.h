// batch_group.h -- a group of a batch and its step, per real type and mode
// (defined in batch_step.cuh, compiled in batch_*.cu, one translation unit
// each).
#pragma once

#include <cuda_runtime.h>

#include <string>
#include <type_traits>
#include <vector>

#include "batch_kernels.cuh"
#include "gpe.h"
#include "internal.h"

using namespace gpe;

// One group: instances of one (mode, precision), with the aggregated launch
// geometry of its passes.
struct Group {
   bool cplx = false, fp32 = false;
   std::vector<int> members;  // instance indices
   int Ly = 0, Lx = 0;        // FFT tile widths (the narrowest of the members)
   BatchGeom geo{};           // maxima over the members (tiles: sums)
   long long off[kNPass + 1] = {};  // start of each pass's work list in dwork
   BatchDesc *dtab = nullptr;        // device descriptor table
   unsigned *dwork = nullptr;        // device work lists (TileRef packed per tile; the sweeps' are in dtile)
   SweepTile *dtile[3] = {nullptr, nullptr, nullptr};  // device tile records of the sweeps
   int sweep_grid[3] = {0, 0, 0};
   size_t sweep_smem[3] = {0, 0, 0};
   mutable RoomyKernels roomy;  // launched with more dynamic shared memory than the default
   int nbuf[3] = {2, 2, 2};  // table buffers of the sweeps (one where two do not fit: long complex lines)
};

inline gpe_status bfail(gpe_status st, const std::string &m) {
   gpe::set_last_error(m);
   return st;
}

#define BCK(x)                                                                        \
   do {                                                                               \
      cudaError_t e_ = (x);                                                           \
      if (e_ != cudaSuccess) return bfail(GPE_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); \
   } while (0)
#define BCKS(...)                     \
   do {                               \
      gpe_status s_ = (__VA_ARGS__);  \
      if (s_ != GPE_OK) return s_;    \
   } while (0)

// Queues the passes of one batch step of group G on stream st, counting its
// launches; ev (may be null): an event recorded after every pass, index = pass.
template <class R, bool CPLX>
gpe_status batch_step(const Group &G, cudaStream_t st, long long *kernels, cudaEvent_t *ev);
