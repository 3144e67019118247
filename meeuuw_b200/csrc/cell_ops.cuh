// What the kernels that own the mesh cell by cell share (mg_level.cu, op_apply.cu): the element
// product of K, the division by the diagonal, the basis tables.  A thread of a tile of CELLS x CELLS
// cells owns one element and the four lattice nodes of its lower-left quadrant -- corner, bottom
// midpoint, left midpoint, centre -- and exchanges the rest through shared-memory planes with unit
// stride over the threads.
#pragma once

#include "mg_level.cuh"
#include "q2_ref.cuh"

namespace mw {

namespace {

// FP64 basis values come from the constant bank (an FP64 immediate costs registers and moves)
__constant__ RefTables c_k;

template <typename R, int Q, int K> MW_D R kdr() {
  if constexpr (sizeof(R) == 4) return (float)RefD<Q, K>::r; else return c_k.dr[Q * 9 + K];
}
template <typename R, int Q, int K> MW_D R kdt() {
  if constexpr (sizeof(R) == 4) return (float)RefD<Q, K>::t; else return c_k.dt[Q * 9 + K];
}

template <typename R, int Q> MW_D R kwq() {
  constexpr double w = ref_wq(Q);
  if constexpr (sizeof(R) == 4) return (float)w; else return c_k.wq[Q];
}

template <typename R, int Q, int K> MW_D R knp() {
  constexpr double v = ref_np(Q, K);
  if constexpr (sizeof(R) == 4) return (float)v; else return c_k.NP[Q * 4 + K];
}

constexpr int CELLS = 16;                                   // cells of a tile, per side

MW_D float2 fma2(float s, float2 a, float2 c) { return __ffma2_rn(make_float2(s, s), a, c); }
MW_D double2 fma2(double s, double2 a, double2 c) { return make_double2(fma(s, a.x, c.x), fma(s, a.y, c.y)); }
MW_D float2 pair(float a, float b) { return make_float2(a, b); }
MW_D double2 pair(double a, double b) { return make_double2(a, b); }

// K_el u on one element: the strain rate at each Gauss point, the stress, B^T back onto the nodes
// (element_apply of stokes.cu without the pressure terms).
// PRESSURE: G_el p joins y and G_el^T u goes to yp (s: the scaling of G), with element_apply's terms.
template <bool PRESSURE = false, typename R, typename R2>
MW_D void k_element(R sx, R sz, R jac, const R2 (&u)[9], const R (&eq)[9], R2 (&y)[9], R s = R(0),
                    const R* pe = nullptr, R* yp = nullptr) {
#pragma unroll
  for (int k = 0; k < 9; ++k) y[k] = pair(R(0), R(0));
  if constexpr (PRESSURE) {
#pragma unroll
    for (int k = 0; k < 4; ++k) yp[k] = R(0);
  }
  static_for<9>([&](auto qc) {
    constexpr int Q = qc.value;
    R2 gx = pair(R(0), R(0)), gz = pair(R(0), R(0));
    static_for<9>([&](auto kc) {
      constexpr int K = kc.value;
      if constexpr (RefD<Q, K>::r != 0.0) gx = fma2(kdr<R, Q, K>(), u[K], gx);
      if constexpr (RefD<Q, K>::t != 0.0) gz = fma2(kdt<R, Q, K>(), u[K], gz);
    });
    const R exx = sx * gx.x, ezz = sz * gz.y;
    const R gg = sizeof(R) == 4 ? fma(sx, gx.y, sz * gz.x) : fma(sz, gz.x, sx * gx.y);
    const R jw = jac * kwq<R, Q>();
    const R e = eq[Q] * jw;
    R2 ar, at;
    if constexpr (PRESSURE) {
      R pq = R(0);
      static_for<4>([&](auto kc) { pq += knp<R, Q, kc.value>() * pe[kc.value]; });
      const R sp = s * jw * pq;
      ar = pair((R(2) * e * exx - sp) * sx, e * gg * sx);
      at = pair(e * gg * sz, (R(2) * e * ezz - sp) * sz);
      const R dv = -s * jw * (exx + ezz);
      static_for<4>([&](auto kc) { yp[kc.value] += knp<R, Q, kc.value>() * dv; });
    } else {
      ar = pair((R(2) * e * exx) * sx, e * gg * sx);
      at = pair(e * gg * sz, (R(2) * e * ezz) * sz);
    }
    static_for<9>([&](auto kc) {
      constexpr int K = kc.value;
      if constexpr (RefD<Q, K>::r != 0.0) y[K] = fma2(kdr<R, Q, K>(), ar, y[K]);
      if constexpr (RefD<Q, K>::t != 0.0) y[K] = fma2(kdt<R, Q, K>(), at, y[K]);
    });
  });
}

// a / d from the rounded reciprocal y = 1 / d, correctly rounded as the division is: q = a y is
// within two units, a first correction by the exact residual a - d q makes it faithful, and the
// second rounds it correctly (Markstein, IBM J. Res. Dev. 34, 1990: a faithful quotient corrected
// with a correctly rounded reciprocal).  Five packed multiply-adds for a node's two components in
// place of two divisions.
MW_D float2 div2(float2 a, float2 d, float2 y) {
  const float2 nd = make_float2(-d.x, -d.y);
  float2 q = __fmul2_rn(a, y);
  float2 r = __ffma2_rn(nd, q, a);
  q = __ffma2_rn(r, y, q);
  r = __ffma2_rn(nd, q, a);
  return __ffma2_rn(r, y, q);
}
MW_D double div1(double a, double d, double y) {
  double q = a * y;
  q = fma(fma(-d, q, a), y, q);
  return fma(fma(-d, q, a), y, q);
}
MW_D double2 div2(double2 a, double2 d, double2 y) { return make_double2(div1(a.x, d.x, y.x), div1(a.y, d.y, y.y)); }


// a translation unit's copy of the tables, filled before its first launch
int ensure_cell_tables() {
  static OncePerDevice once;
  return fill_constant(once, c_k, host_ref_tables) ? MW_OK : MW_ERR_CUDA;
}

}  // namespace

}  // namespace mw
