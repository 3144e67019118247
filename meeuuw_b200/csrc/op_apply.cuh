// The Stokes operator on a level as one launch of cell tiles (op_apply.cu).
#pragma once

#include "mg_level.cuh"

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

int op_ensure_tables();
template <typename R> void op_apply(const OpArgs<R>& a, cudaStream_t s);

}  // namespace mw
