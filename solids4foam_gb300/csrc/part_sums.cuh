// Sums of the processor-local preconditioner over the parts, in an order that
// depends on the part count only (kernels_local.cu, kernels_part.cu).
#pragma once

#include "device_common.cuh"
#include "pcg_common.cuh"
#include "sweep.cuh"

namespace s4g {

// Part records in groups of kLocGroup parts: the CTA whose part completes a
// group (the last to arrive on the group's counter) sums the group's records
// in part order by a fixed shuffle tree, and the last CTA of the launch sums
// the group records -- one round trip each instead of one CTA reading every
// part record at the end of the launch.
constexpr int kLocGroup = 32;

__device__ __forceinline__ int locGroupSize(int g, int nParts) {
  const int n = nParts - g * kLocGroup;
  return n < kLocGroup ? n : kLocGroup;
}

// Thread 0: the arrival of `part`'s record (written by this thread) on its
// group's counter; true if it completes the group.
__device__ __forceinline__ bool locArrive(unsigned* gcnt, int part, int nParts) {
  __threadfence();
  const int g = part / kLocGroup;
  return atomicAdd(&gcnt[g], 1u) + 1u == (unsigned)locGroupSize(g, nParts);
}

// One warp: the record (six values) of group g (lane j holds part g*32 + j), and the
// group's counter back to zero for the next launch.
__device__ __forceinline__ void locGroupSum(const double* rec, double* grec, unsigned* gcnt, int g,
                                            int nParts) {
  const int lane = threadIdx.x & 31;
  const int part = g * kLocGroup + lane;
  __threadfence();
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 6; ++k) v[k] = part < nParts ? __ldcg(rec + 8 * (size_t)part + k) : 0.0;
  const double s = warpSpreadSum<8>(v);
  if (lane % 4 == 0 && lane < 24) grec[8 * (size_t)g + lane / 4] = s;
  if (lane == 0) gcnt[g] = 0;
}

// The last CTA: the sum of the group records in group order -- lane v of
// 64 sums groups v, v + 64, ..., then a fixed tree (sum64's).  Value k in lane k of
// warp 0.  red: 6 values.
__device__ __forceinline__ double locGroupsTotal(const double* grec, int nGroups, double* red) {
  const int t = (int)threadIdx.x, lane = t & 31;
  double s = 0;
  if (t < 64) {
    double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int g = t; g < nGroups; g += 64)
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const double x = __ldcg(grec + 8 * (size_t)g + k);
        v[k] = g == t ? x : v[k] + x;
      }
    s = warpSpreadSum<8>(v);
    if (t >= 32 && lane % 4 == 0 && lane < 24) red[lane / 4] = s;
  }
  __syncthreads();
  if (t >= 32) return 0;
  if (lane % 4 == 0 && lane < 24) s += red[lane / 4];
  return __shfl_sync(0xffffffffu, s, lane < 6 ? 4 * lane : 0);
}

// End of a preconditioner launch, after the CTA's last part: thread 0
// reports that part on its group counter (warp 0 sums the group if that
// completes it); the last CTA sums the group records in group order -- lane
// v of 64 sums groups v, v + 64, ..., then a fixed tree -- and decides, per
// component, the residual test of the pending iteration, beta and wArA, and
// whether the loop goes on.  Block size >= 64.
__device__ __forceinline__ void locFinish(const MeshView& mv, const Controls& c, DevState* st,
                                          double* partials, int lastPart, bool anyPend,
                                          double* red, int* sGroup) {
  double* grec = partials + mv.locGrpOff;
  unsigned* gcnt = reinterpret_cast<unsigned*>(grec + 8 * (size_t)mv.locGroups);
  const int t = (int)threadIdx.x;
  if (t == 0)
    *sGroup = (lastPart >= 0 && locArrive(gcnt, lastPart, mv.nParts)) ? lastPart / kLocGroup : -1;
  __syncthreads();
  if (*sGroup >= 0 && t < 32) locGroupSum(partials, grec, gcnt, *sGroup, mv.nParts);
  if (!lastBlockDone(&st->counter[5], gridDim.x)) return;
  const double mine = locGroupsTotal(grec, mv.locGroups, red);
  if (t >= 32) return;
  if (t == 0) {
    st->counter[5] = 0;
    st->locTicket = 0;
  }
  pcgDecideBeta(c, st, mine, anyPend);
}

}  // namespace s4g
