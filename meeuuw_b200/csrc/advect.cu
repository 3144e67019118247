// Particle interpolation and advection for the Cartesian box (sm_100a).
//
// Reference: pic_functions.py (interpolate :85-101, velocity at a point :18-37, advect :180-292)
// and the material hooks experiment0.py:230-264 / experiment1.py:91-113.
//
// Unlike pic.cu (locate, binning and element means, which must round exactly as the reference),
// this file is compiled with FMA contraction: the basis and dot-product arithmetic agrees with the
// reference's unfused arithmetic to a few ulp, and the element index of a velocity evaluation comes
// from the reciprocal of the spacing, falling back to the division wherever the quotient is close
// enough to an integer for its truncation to depend on the last bits -- so the element (and the
// reference's wrap of x == Lx into the next row) is the reference's.
//
// The Q2 basis is used as the product of its one-dimensional functions: a field's value is three row
// sums of three nodes, twelve multiply-adds, and a velocity's two components share the six functions
// (the nine products and eighteen multiply-adds of the basis written out are three times the arithmetic;
// advection is bound by FP64 issue).
#include "pic_common.cuh"

namespace mw {

// the one-dimensional Q2 functions on nodes -1, 0, 1
struct Q2Lines {
  double r[3], t[3];
  MW_D Q2Lines(double x, double z) {
    const double a = 0.5 * x, c = 0.5 * z;
    r[0] = fma(a, x, -a); r[1] = fma(-x, x, 1.0); r[2] = fma(a, x, a);
    t[0] = fma(c, z, -c); t[1] = fma(-z, z, 1.0); t[2] = fma(c, z, c);
  }
  // the field whose lower-left node of the element is *p, lattice rows nnx apart
  MW_D double value(const double* __restrict__ p, int nnx) const {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double* row = p + (int64_t)j * nnx;
      s += t[j] * (r[0] * __ldg(row) + r[1] * __ldg(row + 1) + r[2] * __ldg(row + 2));
    }
    return s;
  }
};

// ------------------------------------------------------------------------------------------
struct FieldSet {
  const double* in[MW_MAX_FIELDS];
  double* out[MW_MAX_FIELDS];
  int n;
};

// V values of T at a time (16 bytes for two doubles)
template <typename T, int V> struct __align__(sizeof(T) * V) Pack { T v[V]; };
template <int V, typename T> MW_D Pack<T, V> load_pack(const T* p, int64_t i) {
  return reinterpret_cast<const Pack<T, V>*>(p)[i];
}
template <int V, typename T> MW_D void store_pack(T* p, int64_t i, const Pack<T, V>& a) {
  if (p) reinterpret_cast<Pack<T, V>*>(p)[i] = a;
}

__global__ void k_interp(mw_box b, int64_t n, const uint8_t* __restrict__ active, const double* __restrict__ r,
                         const double* __restrict__ t, const int32_t* __restrict__ iel, FieldSet fs) {
  const int nnx = 2 * b.nelx + 1;
  const int64_t nel = (int64_t)b.nelx * b.nelz;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int e = iel[i];
    if (!active[i] || e < 0 || e >= nel) {
      for (int f = 0; f < fs.n; ++f) fs.out[f][i] = 0.0;
      continue;
    }
    const Q2Lines q(r[i], t[i]);
    const int ex = e % b.nelx, ez = e / b.nelx;
    const int64_t n0 = (int64_t)(2 * ez) * nnx + 2 * ex;
    for (int f = 0; f < fs.n; ++f) fs.out[f][i] = q.value(fs.in[f] + n0, nnx);
  }
}

// Interpolation of the five nodal fields the time loop needs (meeuuw.py:1118-1125) fused with
// the material model (experiment0.py:254-264 / experiment1.py:104-111).  V particles a thread: two where
// every array is aligned to a pair (16-byte loads and stores and twice the gathers in flight), else one.
// 109 bytes a particle, most of them the eleven results.  4.2 M particles: 158 -> 139 us (70 us at the copy
// rate, about 113 at its write half); four resident CTAs of 64 registers were the fastest (uncapped 184, five
// 153, one particle a thread 148).
template <int V>
__global__ void __launch_bounds__(256, 4) k_interp_material(mw_box b, int64_t n, const uint8_t* __restrict__ active,
                                                         const double* __restrict__ r, const double* __restrict__ t,
                                                         const int32_t* __restrict__ iel,
                                                         const int8_t* __restrict__ mat, mw_nodal5 nodal,
                                                         mw_material m, mw_swarm_props out) {
  const int nnx = 2 * b.nelx + 1;
  const int64_t nel = (int64_t)b.nelx * b.nelz;
  const double* const fl[5] = {nodal.exx, nodal.ezz, nodal.exz, nodal.q, nodal.T};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n / V; i += (int64_t)gridDim.x * blockDim.x) {
    const auto ac = load_pack<V>(active, i);
    const auto rr = load_pack<V>(r, i), tt = load_pack<V>(t, i);
    const auto ee = load_pack<V>(iel, i);
    Pack<int8_t, V> mm;
#pragma unroll
    for (int k = 0; k < V; ++k) mm.v[k] = 0;
    if (m.kind == MW_MATERIAL_TWO && mat) mm = load_pack<V>(mat, i);
    Pack<double, V> v[5];
    bool act[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int e = ee.v[k];
      act[k] = ac.v[k] != 0;
      const Q2Lines q(rr.v[k], tt.v[k]);
      const bool in = act[k] && e >= 0 && e < nel;
      const int ex = in ? e % b.nelx : 0, ez = in ? e / b.nelx : 0;
      const int64_t n0 = (int64_t)(2 * ez) * nnx + 2 * ex;
#pragma unroll
      for (int f = 0; f < 5; ++f) {
        v[f].v[k] = 0.0;
        if (in && fl[f]) v[f].v[k] = q.value(fl[f] + n0, nnx);
      }
    }
    store_pack<V>(out.exx, i, v[0]);
    store_pack<V>(out.ezz, i, v[1]);
    store_pack<V>(out.exz, i, v[2]);
    store_pack<V>(out.p, i, v[3]);
    store_pack<V>(out.T, i, v[4]);
    Pack<double, V> rho, eta, hcond, hcapa, hprod, alpha;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      if (m.kind == MW_MATERIAL_TWO) {
        int id = mm.v[k];
        id = id < 0 ? 0 : (id > 7 ? 7 : id);
        rho.v[k] = act[k] ? m.mat_rho[id] : 0.0;
        eta.v[k] = act[k] ? m.mat_eta[id] : 0.0;
        hcond.v[k] = hcapa.v[k] = hprod.v[k] = alpha.v[k] = 0.0;
      } else {
        const double T = v[4].v[k];
        rho.v[k] = m.rho0 * (1 - m.alphaT * T);
        eta.v[k] = m.fk_gamma != 0.0 ? exp(-m.fk_gamma * T) : m.eta0;
        hcond.v[k] = m.hcond; hcapa.v[k] = m.hcapa; hprod.v[k] = m.hprod; alpha.v[k] = m.alphaT;
      }
    }
    store_pack<V>(out.rho, i, rho);
    store_pack<V>(out.eta, i, eta);
    store_pack<V>(out.hcond, i, hcond);
    store_pack<V>(out.hcapa, i, hcapa);
    store_pack<V>(out.hprod, i, hprod);
    store_pack<V>(out.alpha, i, alpha);
  }
}

// ------------------------------------------------------------------------------------------
// x / h from the reciprocal ih = 1/h (within a few ulp of the rounded quotient); where that lies
// within 2^-48 (relative) of an integer -- close enough for its truncation to depend on the last
// bits -- the quotient itself, so the truncated value is always the reference's int(x / h).
MW_D double quotient(double x, double h, double ih) {
  const double q = x * ih;
  return fabs(q - rint(q)) <= fabs(q) * 0x1p-48 ? x / h : q;
}

// Velocity at a point: pic_functions.py:18-37.  The element index is the reference's, including
// the case x == Lx that wraps into the next row; indices outside the mesh set a flag.
struct Mover {
  const mw_box& b;
  double ihx, ihz;       // the reciprocals of the spacings
  int64_t nel;
  int nnx;
  const double *u, *w;
  int32_t* err;

  MW_D void at(double rp, double tp, int ex, int ez, double* up, double* wp) const {
    const Q2Lines q(rp, tp);
    const int64_t n0 = (int64_t)(2 * ez) * nnx + 2 * ex;
    *up = q.value(u + n0, nnx);
    *wp = q.value(w + n0, nnx);
  }
  // local coordinate of p in element i (exact doubling and halving aside, the reference's roundings)
  MW_D static double local(double p, double i, double h, double ih) {
    return fma(2.0, (p - __dmul_rn(i, h)) * ih, -1.0);
  }
  MW_D static bool outside(const mw_box& b, double x, double z) { return x < 0 || x > b.Lx || z < 0 || z > b.Lz; }

  // The velocity at (x, z); with CHECK false (and nothing evaluated) when the point lies outside the box.
  // The cell from the reciprocals: sure when the product's fraction is at least 2^-20 away from a whole
  // number (its error is below 2^-20 for any index), and then the point is inside.  Everything else --
  // points near a cell's edge, outside, not finite -- goes the reference's way.
  template <bool CHECK>
  MW_D bool velocity(double x, double z, double* up, double* wp) const {
    const double qx = x * ihx, qz = z * ihz;
    const int ix = (int)qx, iz = (int)qz;
    const double fx = (double)ix, fz = (double)iz;
    constexpr double SURE = 0.5 - 0x1p-20;
    if (fabs(qx - fx - 0.5) < SURE && fabs(qz - fz - 0.5) < SURE && (unsigned)ix < (unsigned)b.nelx &&
        (unsigned)iz < (unsigned)b.nelz) {
      at(local(x, fx, b.hx, ihx), local(z, fz, b.hz, ihz), ix, iz, up, wp);
      return true;
    }
    if (CHECK && outside(b, x, z)) return false;
    const double rx = quotient(x, b.hx, ihx), rz = quotient(z, b.hz, ihz);
    int ex = 0, ez = 0;
    bool ok = rx > -2147483648.0 && rx < 2147483647.0 && rz > -2147483648.0 && rz < 2147483647.0;
    if (ok) {
      ex = (int)rx; ez = (int)rz;
      const int64_t e = (int64_t)b.nelx * ez + ex;
      ok = e >= 0 && e < nel;
      if (ok && (ex < 0 || ex >= b.nelx)) { ex = (int)(e % b.nelx); ez = (int)(e / b.nelx); }   // row wrap
    }
    if (!ok) {
      set_flag(err, MW_FLAG_ELEMENT_RANGE);
      *up = 0.0; *wp = 0.0;
      return true;
    }
    at(local(x, (double)ex, b.hx, ihx), local(z, (double)ez, b.hz, ihz), ex, ez, up, wp);
    return true;
  }
};

// Bound by FP64 issue: about 50 FP64 operations a velocity (95 before: basis written out, index checks
// and box tests at every stage), four velocities a particle in RK4.  4.2 M particles, RK4: 197 -> 139 us with
// four resident CTAs of 64 registers (left to itself the compiler took more and ran at 202).
__global__ void __launch_bounds__(256, 4) k_advect(mw_box b, int rk, double dt_host, const double* __restrict__ dt_dev,
                                                int64_t n, double* __restrict__ x, double* __restrict__ z,
                                                uint8_t* __restrict__ active, const double* __restrict__ u,
                                                const double* __restrict__ w, double* __restrict__ up_out,
                                                double* __restrict__ wp_out, int32_t* err) {
  const double dt = dt_dev ? *dt_dev : dt_host, hdt = dt / 2.0;
  const Mover mv{b, 1.0 / b.hx, 1.0 / b.hz, (int64_t)b.nelx * b.nelz, 2 * b.nelx + 1, u, w, err};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double su = 0.0, sw = 0.0;
    bool act = active[i] != 0;
    if (act) {
      const double xA = x[i], zA = z[i];
      double uA, wA;
      mv.velocity<false>(xA, zA, &uA, &wA);
      if (rk == 1) {                                                  // :220-231
        su = uA; sw = wA;
        const double xn = fma(uA, dt, xA), zn = fma(wA, dt, zA);
        x[i] = xn; z[i] = zn;
        if (Mover::outside(b, xn, zn)) act = false;
      } else {
        double uB, wB;                                                // :239-240
        act = mv.velocity<true>(fma(uA, hdt, xA), fma(wA, hdt, zA), &uB, &wB);
        if (act && rk == 2) {                                         // :244-248
          su = uB; sw = wB;
        } else if (act) {
          double uC, wC, uD, wD;                                      // :265-266, :271-272
          act = mv.velocity<true>(fma(uB, hdt, xA), fma(wB, hdt, zA), &uC, &wC) &&
                mv.velocity<true>(fma(uC, dt, xA), fma(wC, dt, zA), &uD, &wD);
          if (act) {
            su = quotient_exact(uA + 2 * uB + 2 * uC + uD, 6.0, 1.0 / 6.0);   // :277-280
            sw = quotient_exact(wA + 2 * wB + 2 * wC + wD, 6.0, 1.0 / 6.0);
          }
        }
        if (act) { x[i] = fma(su, dt, xA); z[i] = fma(sw, dt, zA); }
      }
      if (!act) active[i] = 0;
    }
    if (!act) { x[i] = 0.0; z[i] = 0.0; }                              // :287-290
    if (up_out) up_out[i] = su;
    if (wp_out) wp_out[i] = sw;
  }
}

}  // namespace mw

using namespace mw;

static bool box_ok(const mw_box& b) { return b.nelx > 0 && b.nelz > 0 && b.hx > 0 && b.hz > 0; }

extern "C" {

int mw_interp_q2(mw_box box, int64_t n, const uint8_t* active, const double* r, const double* t, const int32_t* iel,
                 int32_t nfield, const double* const* fields, double* const* out, void* stream) {
  if (!box_ok(box) || n < 0 || nfield < 1 || nfield > MW_MAX_FIELDS) return MW_ERR_BAD_ARG;
  if (n == 0) return MW_OK;
  FieldSet fs;
  fs.n = nfield;
  for (int f = 0; f < nfield; ++f) { fs.in[f] = fields[f]; fs.out[f] = out[f]; }
  k_interp<<<grid_all(n, 256), 256, 0, (cudaStream_t)stream>>>(box, n, active, r, t, iel, fs);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

int mw_interp_material(mw_box box, int64_t n, const uint8_t* active, const double* r, const double* t,
                       const int32_t* iel, const int8_t* mat, mw_nodal5 nodal, mw_material m, mw_swarm_props out,
                       void* stream) {
  if (!box_ok(box) || n < 0 || !out.rho || !out.eta) return MW_ERR_BAD_ARG;
  if (n == 0) return MW_OK;
  // pairs when every array starts on a pair's boundary (each is indexed by the particle)
  const void* const wide[] = {r, t, out.exx, out.ezz, out.exz, out.p, out.T, out.rho, out.eta, out.hcond, out.hcapa,
                              out.hprod, out.alpha};
  bool pairs = n % 2 == 0 && (uintptr_t)iel % 8 == 0 && (uintptr_t)active % 2 == 0 && (uintptr_t)mat % 2 == 0;
  for (const void* p : wide) pairs = pairs && (uintptr_t)p % 16 == 0;
  cudaStream_t s = (cudaStream_t)stream;
  if (pairs)
    k_interp_material<2><<<grid_all(n / 2, 256), 256, 0, s>>>(box, n, active, r, t, iel, mat, nodal, m, out);
  else
    k_interp_material<1><<<grid_all(n, 256), 256, 0, s>>>(box, n, active, r, t, iel, mat, nodal, m, out);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

int mw_advect_box(mw_box box, int32_t rk, double dt, const double* dt_dev, int64_t n, double* x, double* z,
                  uint8_t* active, const double* u, const double* w, double* up, double* wp, int32_t* err,
                  void* stream) {
  if (!box_ok(box) || n < 0 || !(rk == 1 || rk == 2 || rk == 4)) return MW_ERR_BAD_ARG;
  if (n == 0) return MW_OK;
  k_advect<<<grid_all(n, 256), 256, 0, (cudaStream_t)stream>>>(box, rk, dt, dt_dev, n, x, z, active, u, w, up, wp, err);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

}  // extern "C"
