// Deterministic sums over a grid, finished in the launch that computes the terms.
#pragma once

#include "common.cuh"

namespace mw {

// The grid-wide sum of one value per thread: block partials in part[block], and the last block to
// arrive adds them in block order and resets the counter (threadfence + arrival counter).  Called
// once, by every thread, at the end of a kernel.  True for the one thread that holds the sum.
MW_D bool grid_sum(double v, double* part, unsigned* counter, int block, int nblocks, double* sum) {
  __shared__ double sh[32];
  __shared__ bool last;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (wid == 0) {
    v = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) {
      part[block] = v;
      __threadfence();
      last = atomicAdd(counter, 1u) == (unsigned)nblocks - 1;
    }
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double t = 0;
  for (int i = threadIdx.x; i < nblocks; i += blockDim.x) t += ((volatile double*)part)[i];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  if (lane == 0) sh[wid] = t;
  __syncthreads();
  if (threadIdx.x != 0) return false;
  double s = 0;
  for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += sh[k];
  *sum = s;
  *counter = 0u;
  return true;
}

// Where a kernel leaves a sum that the iterations keep by parity: out[*it & 1].
struct ParitySum {
  double* part;
  unsigned* counter;
  double* out;
  const double* it;
};

MW_D void grid_sum_parity(double v, const ParitySum& p, int block, int nblocks) {
  double s;
  if (grid_sum(v, p.part, p.counter, block, nblocks, &s)) p.out[(int)*p.it & 1] = s;
}

}  // namespace mw
