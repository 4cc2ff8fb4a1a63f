// incident.h - one step of the 1-D incident grid as a job of another launch.
#pragma once

#include <cuda_runtime.h>

namespace fdtdb {

struct IncidentJob
{
  double *now;                 // level written
  const double *old;           // the same family's previous level
  const double *other;         // E: HInc before its update; H: EInc after its update
  int cells = 0;               // cells 0 .. cells - 1 are updated (0: nothing to do)
  double modifier;
  const double *src;           // E: value of cell 0
};

// E then H of one step.  H at cell i needs the new E at i and i + 1, which the
// job computes again from the old levels instead of waiting for it: the cells
// are independent, any threads of a launch may take them.  (As two launches
// in front of a sweep step they were 6.5 of 58 us per step at 80^3.)
struct IncidentPair
{
  IncidentJob e, h;            // h.other = e.now, e.other = h.old
};

#ifdef __CUDACC__
// (rounded operations: the same bits with and without contraction)
__device__ __forceinline__ double incident_e_cell (const IncidentJob &e, int i)
{
  if (i >= e.cells)
    return e.now[i];           // not updated: both levels hold it
  if (i == 0)
    return *e.src;
  return __dadd_rn (e.old[i], __dmul_rn (__dsub_rn (e.other[i - 1], e.other[i]), e.modifier));
}

__device__ __forceinline__ void incident_pair (const IncidentPair &j, int first, int stride)
{
  for (int i = first; i < max (j.e.cells, j.h.cells); i += stride)
  {
    const double e = incident_e_cell (j.e, i);
    if (i < j.e.cells)
      j.e.now[i] = e;
    if (i < j.h.cells)
      j.h.now[i] =
          __dadd_rn (j.h.old[i], __dmul_rn (__dsub_rn (e, incident_e_cell (j.e, i + 1)), j.h.modifier));
  }
}
#endif

}  // namespace fdtdb
