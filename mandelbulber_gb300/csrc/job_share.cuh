// How the warps of a wavefront stage share its jobs.
#pragma once

#include <cuda_runtime.h>

namespace mbgb {
namespace dev {

__host__ __device__ __forceinline__ unsigned int at_least_one(const unsigned int v) {
#ifdef __CUDA_ARCH__
  return max(1u, v);
#else
  return v > 1u ? v : 1u;
#endif
}

// `lanes`: the lanes of a warp that take jobs; `warps`: the launch's first warps, which do;
// `refill`: idle lanes before a warp claims again, refill_min of 32 in proportion to its lanes.
struct JobShare {
  unsigned int lanes, warps, refill;
  bool idle;   // this lane takes none
};

// The share of lane `lane` of warp `warp`. A stage with fewer jobs than lanes hands each warp only as
// many as let `spread` warps take part, and only the first warps take any (blocks start one per SM, so
// those spread evenly over the SMs and their sub-partitions).
__host__ __device__ __forceinline__ JobShare job_share(const unsigned int jobs, const unsigned int spread,
                                                       const unsigned int refill_min, const unsigned int warp,
                                                       const unsigned int lane) {
  JobShare s;
  s.lanes = jobs >= 32u * spread ? 32u : at_least_one((jobs + spread - 1) / spread);
  s.warps = (jobs + s.lanes - 1) / s.lanes;
  s.refill = at_least_one(s.lanes * refill_min / 32u);
  s.idle = lane >= s.lanes || warp >= s.warps;
  return s;
}

// `spread` of a launch of `warps` warps, from that of the main launches: one of fewer warps, as the
// overflow pass's 64, spreads over those it has. With lanes for 2432 warps a 96x54 Mandelbox whose
// rays all overflow (DE factor 0.01) took 107.8 ms, with lanes for its own 41.2 (FP64: 512 and 298).
inline int launch_spread(const int spread, const int warps) { return spread < warps ? spread : warps; }

}  // namespace dev
}  // namespace mbgb
