// The parts of a multigrid hierarchy's set-up that run over every level at once, or on one SM
// (mg_setup.cu).
#pragma once

#include "mg_level.cuh"

namespace mw {

constexpr int MAXLEV = 12;

// One level of a power iteration v <- D^-1 K v / |v|.
template <typename R>
struct PowerLevel {
  LevelGeo g;
  const R* eta;          // nine planes (qs = nel) or one value per element (qs = 0)
  int64_t qs;
  const uint8_t* fix;
  const R *diag, *dinv;
  const R* vin;
  R* vout;
  double* lam2;          // [0]: |v|^2 after the last iteration; [1], [2]: in between
  double* cheb;          // the last iteration's Chebyshev coefficients for `deg` steps
  int deg;
  int block0, tiles_x;   // its first block of the launch, its tiles along x
  double* part;
  unsigned* counter;
};

template <typename R>
struct PowerArgs {
  int n, it, last;
  double ratio, safety;
  PowerLevel<R> L[MAXLEV];
};

// Chebyshev coefficients from |D^-1 K v|^2 with |v| = 1
MW_D void cheb_coefficients(double lam2, int degree, double ratio, double safety, double* coef) {
  const double lmax = sqrt(fmax(lam2, 1e-300)) * safety;
  const double lmin = lmax / ratio;
  const double theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin), sigma = theta / delta;
  double rho = 1.0 / sigma;
  coef[0] = 0.0;                             // step 0: d = (1/theta) D^-1 r
  coef[1] = 1.0 / theta;
  for (int k = 1; k < degree; ++k) {
    const double rn = 1.0 / (2.0 * sigma - rho);
    coef[2 * k] = rn * rho;                  // c1: d = c1 d + c2 D^-1 r
    coef[2 * k + 1] = 2.0 * rn / delta;
    rho = rn;
  }
}

int setup_ensure_tables();
// blocks (and partial sums) of a level of nx x nz elements in a power step
int power_blocks(int nx, int nz);
int power_tiles_x(int nx);
// one iteration of every level in one launch of `blocks` blocks
template <typename R> void power_step(const PowerArgs<R>& a, int blocks, cudaStream_t s);

// The inverse of the coarsest level's K (Dirichlet-eliminated), nd x nd; false when it is too large
// for the one-CTA kernel.
template <typename R>
bool dense_inverse(const LevelGeo& g, const R* eta, const uint8_t* fix, int nd, double* Ainv, cudaStream_t s);

}  // namespace mw
