// How the warps of a wavefront stage share its jobs.
#pragma once

#include <cuda_runtime.h>

namespace mbgb {
namespace dev {

// `lanes`: the lanes of a warp that take jobs; `warps`: the launch's first warps, which do;
// `refill`: idle lanes before a warp claims again, a quarter of its lanes at most unless it has all.
struct JobShare {
  unsigned int lanes, warps, refill;
};

// A stage with fewer jobs than lanes hands each warp only as many as let `spread` warps take part,
// and only the first warps take any (blocks start one per SM, so those spread evenly over the SMs and
// their sub-partitions). `spread` is the main launches'; a launch of fewer warps, as the overflow
// pass's 64, spreads over those it has: with lanes for 2432 warps a 96x54 Mandelbox whose rays all
// overflow (DE factor 0.01) took 107.8 ms, with lanes for its own 41.2 (FP64: 512 and 298).
__host__ __device__ __forceinline__ JobShare job_share(const unsigned int jobs, const unsigned int spread,
                                                       const unsigned int launched, const unsigned int refill_min) {
  JobShare s;
  const unsigned int over = spread < launched ? spread : launched;
  s.lanes = jobs >= 32u * over ? 32u : (jobs + over - 1) / over;
  if (s.lanes < 1u) s.lanes = 1u;
  s.warps = (jobs + s.lanes - 1) / s.lanes;
  const unsigned int quarter = s.lanes / 4 > 1u ? s.lanes / 4 : 1u;
  s.refill = s.lanes == 32u || refill_min < quarter ? refill_min : quarter;
  return s;
}

}  // namespace dev
}  // namespace mbgb
