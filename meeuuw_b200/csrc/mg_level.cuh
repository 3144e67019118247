// One multigrid level's half of a V-cycle as one launch (mg_level.cu), and the level geometry it
// shares with the operator and solver kernels of stokes.cu.
#pragma once

#include "common.cuh"
#include "reduce.cuh"

namespace mw {

struct LevelGeo {
  int nx, nz;        // elements
  int nnx, nnz;      // Q2 lattice nodes
  double hx, hz;
  double s;          // G scaling eta_ref / L_ref (build_matrix_stokes.py:157)
};

template <typename R> struct Vec2;
template <> struct Vec2<float> { typedef float2 T; };
template <> struct Vec2<double> { typedef double2 T; };

// smoothing steps per sweep the level launches are built for
constexpr int MG_MAXDEG = 2;

// The transfer between a level of nf elements a side and the coarser one of nc along one direction, as
// tables: fine lattice node i takes coarse nodes pj[i] .. pj[i] + 2 with weights pw[3 i ...] (nodes past the
// end with weight zero); coarse node J takes fine nodes ri[J] .. ri[J] + rn[J] - 1 with weights rw[RTAPS J ...].
constexpr int RTAPS = 8;
struct Transfer1D {
  const int* pj;
  const double* pw;
  const int *ri, *rn;
  const double* rw;
};

// Arguments of a level's half cycle.  Velocity vectors are interleaved (u, w) pairs.
template <typename R>
struct MgArgs {
  LevelGeo g, gc;      // this level, the coarser one
  const R* eta;        // viscosity: nine planes of nel values (level 0), or one value per element
  const uint8_t* fix;  // Dirichlet flags (2 per node)
  const R *diag, *dinv;// diag(K) and its rounded reciprocal
  const R* b;          // right-hand side
  const R* xin;        // upward: x before the correction (not the output buffer)
  R* x;                // downward: the smoothed x; upward: the result
  const double* cheb;  // Chebyshev coefficient pairs {c1, c2} per step
  R* bc;               // downward: the restricted residual (fixed coarse entries zero)
  const uint8_t* fixc;
  const R* xc;         // upward: the coarse correction
  Transfer1D tx, tz;   // levels that are not nested: the transfer along each direction
  ParitySum bx;        // upward: (b, x) of the result (part null: not wanted)
};

// The FP64 kernels' basis tables in the constant bank; called before the first level launch.
int mg_ensure_tables();
// Smoothing from a zero guess (`deg` Chebyshev-Jacobi steps), the residual and its restriction.
template <typename R> void mg_down(const MgArgs<R>& a, int deg, bool planes, cudaStream_t s);
// The coarse correction and `deg` smoothing steps.
template <typename R> void mg_up(const MgArgs<R>& a, int deg, bool planes, cudaStream_t s);

// The coarse end of a V-cycle in one launch (mg_tail.cu): `n` smoothed levels of at most MG_TAIL_CELLS cells
// ((nx + 1)(nz + 1)) and the coarsest level's dense inverse.
constexpr int MG_TAIL_CELLS = 384, MG_TAIL_LEVELS = 5;
template <typename R> constexpr int mg_tail_degree() { return sizeof(R) == 4 ? MG_MAXDEG : 1; }   // smoothing steps
template <typename R>
struct MgTailLevel {
  LevelGeo g;
  const R *eta, *diag, *dinv;          // eta: one value per element
  const uint8_t* fix;
  const double* cheb;
  Transfer1D tx, tz;                   // to the next level
};
template <typename R>
struct MgTailArgs {
  MgTailLevel<R> L[MG_TAIL_LEVELS];
  int n, nd;
  LevelGeo gd;                         // the coarsest level: nd unknowns, Ainv
  const uint8_t* fixd;
  const double* Ainv;
  const R* b;                          // the first level's right-hand side ...
  R* x;                                // ... and result
};
int mg_tail_ensure_tables();
// false when the levels' vectors do not fit one CTA's shared memory (nothing is launched)
template <typename R> bool mg_tail(const MgTailArgs<R>& a, int deg, cudaStream_t s);

}  // namespace mw
