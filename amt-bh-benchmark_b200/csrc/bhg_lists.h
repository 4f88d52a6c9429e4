// Where the walk keeps a group's dense list, for host and device.
#pragma once

#include <stddef.h>

#if defined(__CUDACC__)
#define BHG_LIST_HD __host__ __device__ __forceinline__
#else
#define BHG_LIST_HD inline
#endif

namespace bhg {

// The dense list of a job on group gi by warp `warp` of the grid; there is one
// list per warp.  With dense jobs (paired: two warps of the grid for each of
// the ngroups groups) the group's own job writes the group's list while its
// dense job reads it.  When the traversal pauses, the dense job learns of it
// only after the cells published so far, so from then on (paused) the group's
// own job writes another list, one of the second half, which no other job
// touches.
BHG_LIST_HD size_t dense_slot(bool paired, bool paused, size_t gi, size_t ngroups, size_t warp) {
  return !paired ? warp : paused ? ngroups + gi : gi;
}

}  // namespace bhg
