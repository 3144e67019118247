// Particle-in-cell helpers shared by the bit-exact kernels (pic.cu: locate, binning,
// projections) and the FMA-contracted ones (advect.cu: interpolation, advection).
#pragma once

#include "common.cuh"

namespace mw {

// x_V / z_V of local node 0 of element e: build_velocity_mesh.py:116-117 computes i*hx/2.
MW_D double xv0(const mw_box& b, int ex) { return ((double)(2 * ex) * b.hx) / 2; }
MW_D double zv0(const mw_box& b, int ez) { return ((double)(2 * ez) * b.hz) / 2; }

// a / h from the rounded reciprocal ih = 1 / h, rounded as the division is (a product corrected twice
// by its exact residual: Markstein, IBM J. Res. Dev. 34, 1990).  Not finite where the product
// overflows: locate refuses such a position either way.
MW_D double quotient_exact(double a, double h, double ih) {
  double q = a * ih;
  q = fma(fma(-h, q, a), ih, q);
  return fma(fma(-h, q, a), ih, q);
}

}  // namespace mw
