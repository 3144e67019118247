// The Stokes operator on a level as one launch of cell tiles (op_apply.cu).
#pragma once

#include "mg_level.cuh"
#include "solve_scalars.cuh"

namespace mw {

template <typename R>
struct OpArgs {
  LevelGeo g;
  const R* u;          // velocity (interleaved u, w); null: zero
  const R* p;          // pressure; null: zero
  const R* eta;        // viscosity of element e at Gauss point q: eta[q * qs + e * es]
  int64_t qs, es;
  const uint8_t* fix;  // Dirichlet flags (2 per node)
  const R* diag;       // diag(K)
  R* yV;               // K u + G p, or with bV the residual bV - (K u + G p); may be null
  R* yP;               // G^T u, or bP - G^T u; may be null
  const R *bV, *bP;
};

// One conjugate-gradient direction and its operator product: p = z + beta p, Ap = K p, (p, Ap).
// p lives in pbuf[iteration & 1], so that a tile's halo can read the old direction while others
// write the new one; rz holds (r, z) by the same parity, beta = rz[k] / rz[k - 1].
template <typename R>
struct PcgDir {
  const R* z;
  R* pbuf[2];
  const double* rz;
  const double* it;    // the iteration, 0 for the first (p = z)
  double *part, *pap;  // partial sums, (p, Ap)
  unsigned* counter;
};

// The FP64 residual (bV, bP) - A (u, p) with its sum of squares, and what follows from it.
struct ResidSum {
  double *part, *sc;
  unsigned* counter;
  int action;
  LoopTest test;
};

int op_ensure_tables();
void op_residual(const OpArgs<double>& a, const ResidSum& r, cudaStream_t s);
template <typename R> void op_apply(const OpArgs<R>& a, cudaStream_t s);
template <typename R> void op_pcg_direction(const OpArgs<R>& a, const PcgDir<R>& d, cudaStream_t s);
// the partial sums the level and direction launches of a level of nx x nz elements need
int cell_partials(int nx, int nz);

}  // namespace mw
