// Deterministic sums over a grid, finished in the launch that computes the terms.
#pragma once

#include "common.cuh"

namespace mw {

// The grid-wide sums of NV values per thread: block partials in part[i * nblocks + block], and the last
// block to arrive adds them in block order and resets the counter (threadfence + arrival counter).
// Called once, by every thread, at the end of a kernel.  True for the one thread that holds the sums.
template <int NV>
MW_D bool grid_sums(double (&v)[NV], double* part, unsigned* counter, int block, int nblocks, double* sum) {
  __shared__ double sh[NV][32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
    if (lane == 0) sh[i][wid] = v[i];
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      v[i] = lane < nw ? sh[i][lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
      if (lane == 0) part[i * nblocks + block] = v[i];
    }
    if (lane == 0) {
      __threadfence();
      last = atomicAdd(counter, 1u) == (unsigned)nblocks - 1;
    }
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double t = 0;
    for (int k = threadIdx.x; k < nblocks; k += blockDim.x) t += ((volatile double*)part)[i * nblocks + k];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) sh[i][wid] = t;
  }
  __syncthreads();
  if (threadIdx.x != 0) return false;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double s = 0;
    for (int k = 0; k < nw; ++k) s += sh[i][k];
    sum[i] = s;
  }
  *counter = 0u;
  return true;
}

MW_D bool grid_sum(double v, double* part, unsigned* counter, int block, int nblocks, double* sum) {
  double a[1] = {v};
  return grid_sums<1>(a, part, counter, block, nblocks, sum);
}
MW_D bool grid_sum2(double v, double w, double* part, unsigned* counter, int block, int nblocks, double* sum) {
  double a[2] = {v, w};
  return grid_sums<2>(a, part, counter, block, nblocks, sum);
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
