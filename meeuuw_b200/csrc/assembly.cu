// Element assembly kernels (sm_100a): Q2xQ1 Stokes and Q2 Crank-Nicolson energy.
//
// Reference: build_matrix_stokes.py:18-278 (box, plane strain) and build_matrix_energy.py:12-141.
// A CTA works on batches of EB elements; 18 (Stokes) or 9 (energy) threads per element, one element
// matrix row each.  The 3x3 Gauss basis tables and the batch's per-qpoint inputs are staged in
// shared memory; the element outputs are staged in shared memory too and leave in whole lines
// in the reference's VV order (build_matrix_stokes.py:235-276, build_matrix_energy.py:133-137).
//
// Dirichlet elimination (build_matrix_stokes.py:206-217, build_matrix_energy.py:118-130) is done
// row-locally: eliminating fixed dofs in ascending order leaves a free row i with
// f_i - sum_{fixed j ascending} K0_ij v_j and zeros in the fixed columns, and a fixed row with
// only its diagonal and rhs K0_ii v_i -- the same values the reference's sequential loop yields.
//
// Right-hand sides: each element writes its local vector to a scratch buffer; a node-centric
// gather then sums the (up to 4) element contributions in ascending element order, the order of
// the reference's scatter loop.  No atomics; results are run-to-run identical.
#include <algorithm>

#include "common.cuh"

namespace mw {

constexpr int EB_S = 16;   // elements per CTA, Stokes
constexpr int EB_T = 24;   // elements per CTA, energy (static shared memory stays under 48 KB)

// local Q2 node index from its lattice offset (dx, dz) in {0,1,2}^2
MW_HD int q2_local(int dx, int dz) {
  if (dz == 0) return dx == 0 ? 0 : (dx == 1 ? 4 : 1);
  if (dz == 1) return dx == 0 ? 7 : (dx == 1 ? 8 : 5);
  return dx == 0 ? 3 : (dx == 1 ? 6 : 2);
}

// One matrix row (element, dof) a thread, EB_S elements a pass, CTAs that stay for many passes.  A point's
// weighted coefficient is formed once per element; an entry of K then takes one rounded addition a point (the
// geometric factor 2 o o_j + t t_j of the row's own component is formed before it is weighted: adding its two
// weighted halves one after the other is one operation fewer and 8 to 15 % further from exact sums).  Rows of
// both components run the same instructions on derivatives read by component: a branch on it issued every
// multiply-add twice.  The results take the room of the derivatives and leave as bulk copies.  BLOCKS writes
// K, G, GT, M, M_eta and H, otherwise [K | G G]; both skip what they do not write.
// A pass over 256^2 elements in FP64, right-hand sides included: 337 -> 139 us, in FP32 175 -> 93; with BLOCKS
// 361 -> 188 and 187 -> 130 (a batch a CTA, derivatives and results apart, before).  Bounds: the 245 MB written
// take 37 us, the FP64 multiply-adds about 30, the loads that feed them as much; the phases of a batch
// overlap only across the CTAs of an SM.
template <typename R>
struct alignas(2 * sizeof(R)) Pair {
  R x, z;
};

template <typename R, bool BLOCKS>
struct StokesSmem {                        // R values per CTA, by offset
  static constexpr int Q = EB_S * 9;
  static constexpr int DV = 0;                                   // pairs (dN/dx, dN/dz) of the velocity
  static constexpr int DP = DV + 2 * EB_S * 81;                  // of the pressure
  static constexpr int W = DP + (BLOCKS ? 2 * EB_S * 36 : 0);    // eta JxW (FP32: eta), JxW, rho gx JxW, rho gz JxW
  static constexpr int J = W + 4 * Q;                            // the four entries of the Jacobian
  static constexpr int IN_END = J + 4 * Q;
  static constexpr int G0 = 0;                                   // rows of G before the elimination
  static constexpr int OUT = BLOCKS ? 572 : 468;                 // results per element
  static constexpr int ROOM = IN_END > EB_S * OUT ? IN_END : EB_S * OUT;
  static constexpr int NV = ROOM, NP = NV + 81, DRV = NP + 37, DRP = DRV + 162;
  static constexpr int BCV = (DRP + 72 + 3) / 4 * 4;             // doubles, then one flag word an element
  static constexpr int CTAS = BLOCKS ? 2 : 3;                    // an SM (FP64: 78 and 65 KB a CTA)
  static constexpr size_t bytes = BCV * sizeof(R) + EB_S * 18 * sizeof(double) + EB_S * sizeof(unsigned);
};

// n bytes (a multiple of 16) from shared to global memory, by one thread, both 16-byte aligned
MW_D void bulk_store(void* dst, const void* src, unsigned n) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               :: "l"(dst), "r"((unsigned)__cvta_generic_to_shared(src)), "r"(n) : "memory");
}

template <typename R, bool BLOCKS>
__global__ void __launch_bounds__(EB_S * 18, StokesSmem<R, BLOCKS>::CTAS)
k_assemble_stokes(mw_box b, mw_stokes_in in, int write, int bulk, R* __restrict__ vv_full, R* __restrict__ vv_K,
                  R* __restrict__ vv_G, R* __restrict__ vv_GT, R* __restrict__ vv_M, R* __restrict__ vv_Meta,
                  R* __restrict__ vv_H, double* __restrict__ f_el, double* __restrict__ h_el) {
  using L = StokesSmem<R, BLOCKS>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* sm = reinterpret_cast<R*>(smem_raw);
  Pair<R>* dV = reinterpret_cast<Pair<R>*>(sm + L::DV);
  Pair<R>* dP = reinterpret_cast<Pair<R>*>(sm + L::DP);
  R *wq = sm + L::W, *jc = sm + L::J, *G0 = sm + L::G0, *outs = sm;
  R *NV = sm + L::NV, *NP = sm + L::NP, *drV = sm + L::DRV, *drP = sm + L::DRP;
  double* bcv = reinterpret_cast<double*>(sm + L::BCV);
  unsigned* bcf = reinterpret_cast<unsigned*>(bcv + EB_S * 18);

  const int64_t nel = (int64_t)b.nelx * b.nelz;
  const int64_t nbatch = (nel + EB_S - 1) / EB_S;
  const int tid = threadIdx.x;
  const int nnx = 2 * b.nelx + 1;
  constexpr int NT = EB_S * 18;
  for (int i = tid; i < 81; i += NT) {
    NV[i] = (R)in.N_V[i]; drV[2 * i] = (R)in.dNdr_V[i]; drV[2 * i + 1] = (R)in.dNdt_V[i];
  }
  for (int i = tid; i < 36; i += NT) {
    NP[i] = (R)in.N_P[i]; drP[2 * i] = (R)in.dNdr_P[i]; drP[2 * i + 1] = (R)in.dNdt_P[i];
  }
  const R s = (R)(in.eta_ref / in.L_ref);                                // build_matrix_stokes.py:157
  const int el = tid / 18, ikk = tid - el * 18;
  const int i = ikk >> 1, c = ikk & 1;

  for (int64_t batch = blockIdx.x; batch < nbatch; batch += gridDim.x) {
    const int64_t e0 = batch * EB_S;
    const int ne = (int)((nel - e0) < EB_S ? (nel - e0) : EB_S);
    const bool live = el < ne;
    if (tid < EB_S) bcf[tid] = 0;
    if (tid < ne * 9) {
      const int64_t g = e0 * 9 + tid;
      const R jxw = (R)in.JxWq[g], eta = (R)in.etaq[g], rj = jxw * (R)in.rhoq[g];
      wq[tid] = sizeof(R) == 8 ? eta * jxw : eta;   // (their product alone may leave FP32's range)
      wq[L::Q + tid] = jxw;
      wq[2 * L::Q + tid] = rj * (R)in.gxq[g];
      wq[3 * L::Q + tid] = rj * (R)in.gzq[g];
      jc[tid] = (R)in.jcbi00q[g];
      jc[L::Q + tid] = (R)in.jcbi01q[g];
      jc[2 * L::Q + tid] = (R)in.jcbi10q[g];
      jc[3 * L::Q + tid] = (R)in.jcbi11q[g];
    }
    bool flag = false;
    int64_t dof = 0;
    if (live) {
      const int64_t e = e0 + el;
      dof = 2 * q2_node((int)(e % b.nelx), (int)(e / b.nelx), i, nnx) + c;     // local_to_globalV, meeuuw.py:874-882
      flag = in.bc_fix_V[dof] != 0;
    }
    __syncthreads();
    if (flag) {
      bcv[tid] = in.bc_val_V[dof];
      atomicOr(bcf + el, 1u << ikk);
    }
    // derivatives at the Gauss points: build_matrix_stokes.py:131-134
    for (int t = tid; t < ne * 81; t += NT) {
      const int q = t / 9, k = t % 81;                                   // q: point of the batch
      const R r = drV[2 * k], u = drV[2 * k + 1];
      dV[t] = Pair<R>{jc[q] * r + jc[L::Q + q] * u, jc[2 * L::Q + q] * r + jc[3 * L::Q + q] * u};
    }
    if (BLOCKS)
      for (int t = tid; t < ne * 36; t += NT) {
        const int q = t / 4, k = t % 36;
        const R r = drP[2 * k], u = drP[2 * k + 1];
        dP[t] = Pair<R>{jc[q] * r + jc[L::Q + q] * u, jc[2 * L::Q + q] * r + jc[3 * L::Q + q] * u};
      }
    __syncthreads();

    // the row's entries by node: own[j] in the row's component (column 2 j + c), oth[j] in the other one
    R own[9], oth[9], G[4], H[4], Mv = 0, f = 0;
#pragma unroll
    for (int j = 0; j < 9; ++j) own[j] = oth[j] = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) { G[k] = 0; H[k] = 0; }
    if (live) {
#pragma unroll 1
      for (int q = 0; q < 9; ++q) {
        const int eq = el * 9 + q;
        const R w = wq[eq], jxw = wq[L::Q + eq];
        // B^T C B (build_matrix_stokes.py:140), C = diag(2, 2, 1): with (o, t) the derivatives in the row's own
        // direction and the other one, 2 o o_j + t t_j in its own component, t o_j in the other
        const R* dc = reinterpret_cast<const R*>(dV + el * 81 + q * 9) + c;
        const R* dt = reinterpret_cast<const R*>(dV + el * 81 + q * 9) + (c ^ 1);
        const R o = dc[2 * i], t = dt[2 * i], wt = w * t;
#pragma unroll
        for (int j = 0; j < 9; ++j) {
          const R oj = dc[2 * j];
          const R g = R(2) * o * oj + t * dt[2 * j];
          own[j] += sizeof(R) == 8 ? g * w : g * w * jxw;
          oth[j] += sizeof(R) == 8 ? wt * oj : wt * oj * jxw;
        }
        const R n = NV[q * 9 + i];
        f += n * wq[(2 + c) * L::Q + eq];                                // :142-143
        const R ow = o * jxw;
#pragma unroll
        for (int k = 0; k < 4; ++k) G[k] -= ow * NP[q * 4 + k];          // :144-146
        if (BLOCKS) {
          const R nj = n * jxw;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const Pair<R> dk = dP[eq * 4 + k];
            H[k] += (c == 0 ? dk.x : dk.z) * nj;                         // :148-153
          }
          if (ikk < 16) Mv += NP[q * 4 + (ikk >> 2)] * NP[q * 4 + (ikk & 3)] * jxw;   // :147
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) G[k] *= s;
    }
    // ---- Dirichlet elimination (row-local form) ----
    const unsigned fx = live ? bcf[el] : 0;
    const double* fv = bcv + el * 18;
    R frow = f;
    R G1[4] = {G[0], G[1], G[2], G[3]};
    if (fx) {
      if (fx >> ikk & 1) {
        R kd = 0;
#pragma unroll
        for (int j = 0; j < 9; ++j) {
          if (j == i) kd = own[j];
          else own[j] = 0;
          oth[j] = 0;
        }
        frow = kd * (R)fv[ikk];
#pragma unroll
        for (int k = 0; k < 4; ++k) G[k] = 0;
      } else {
#pragma unroll
        for (int j = 0; j < 9; ++j) {                      // ascending dofs
          R e0 = c == 0 ? own[j] : oth[j], e1 = c == 0 ? oth[j] : own[j];
          if (fx >> (2 * j) & 1) { frow -= e0 * (R)fv[2 * j]; e0 = 0; }
          if (fx >> (2 * j + 1) & 1) { frow -= e1 * (R)fv[2 * j + 1]; e1 = 0; }
          own[j] = c == 0 ? e0 : e1;
          oth[j] = c == 0 ? e1 : e0;
        }
      }
    }
    __syncthreads();                                       // the derivatives are read: their room is reused
    if (fx >> ikk & 1) {
#pragma unroll
      for (int k = 0; k < 4; ++k) G0[el * 72 + ikk * 4 + k] = G1[k];
    }
    __syncthreads();
    if (live) {
      f_el[(e0 + el) * 18 + ikk] = (double)frow;
      if (ikk < 4) {
        R h = 0;
        for (unsigned m = fx; m; m &= m - 1) {
          const int r2 = __ffs(m) - 1;
          h -= G0[el * 72 + r2 * 4 + ikk] * (R)fv[r2];
        }
        h_el[(e0 + el) * 4 + ikk] = (double)h;
      }
    }
    __syncthreads();
    if (!write) continue;                                  // right-hand sides only
    // ---- the element results in the reference's order ----
    if (!BLOCKS) {
      if (live) {
        Pair<R>* o = reinterpret_cast<Pair<R>*>(outs + el * 468 + ikk * 26);    // :268-276
#pragma unroll
        for (int j = 0; j < 9; ++j) o[j] = c == 0 ? Pair<R>{own[j], oth[j]} : Pair<R>{oth[j], own[j]};
#pragma unroll
        for (int k = 0; k < 4; ++k) o[9 + k] = Pair<R>{G[k], G[k]};
      }
    } else if (live) {
      R* oK = outs + el * 324 + ikk * 18;
      R *oG = outs + EB_S * 324, *oGT = oG + EB_S * 72, *oH = oGT + EB_S * 72, *oM = oH + EB_S * 72;
      R* oMe = oM + EB_S * 16;
#pragma unroll
      for (int j = 0; j < 9; ++j) {                                             // :237-240
        oK[2 * j + c] = own[j];
        oK[2 * j + (c ^ 1)] = oth[j];
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        oG[el * 72 + ikk * 4 + k] = G[k];                                       // :243-246
        oGT[el * 72 + k * 18 + ikk] = G[k];                                     // :249-252
        oH[el * 72 + k * 18 + ikk] = H[k];                                      // :255-258
      }
      if (ikk < 16) {
        oM[el * 16 + ikk] = Mv;                                                 // :261-265
        oMe[el * 16 + ikk] = Mv / (R)in.eta_e[e0 + el];
      }
    }
    if (bulk) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the results, before the copies
    __syncthreads();
    auto put = [&](R* dst, const R* src, int per) {
      if (bulk) {
        if (tid == 0) bulk_store(dst + e0 * per, src, (unsigned)(ne * per * sizeof(R)));
      } else {
        for (int x = tid; x < ne * per; x += NT) dst[e0 * per + x] = src[x];
      }
    };
    if (!BLOCKS) {
      put(vv_full, outs, 468);
    } else {
      const R *oG = outs + EB_S * 324, *oGT = oG + EB_S * 72, *oH = oGT + EB_S * 72, *oM = oH + EB_S * 72;
      put(vv_K, outs, 324);
      put(vv_G, oG, 72);
      put(vv_GT, oGT, 72);
      put(vv_H, oH, 72);
      put(vv_M, oM, 16);
      put(vv_Meta, oM + EB_S * 16, 16);
    }
    if (bulk && tid == 0) {                                // the room is free once the copies have read it
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    __syncthreads();
  }
  if (bulk && tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// Sum element-local vectors onto Q2 nodes (ndof per node) in ascending element order.
__global__ void k_gather_q2(mw_box b, int ndof, const double* __restrict__ vel, double* __restrict__ out) {
  const int nnx = 2 * b.nelx + 1, nnz = 2 * b.nelz + 1;
  const int64_t nn = (int64_t)nnx * nnz;
  const int per = 9 * ndof;
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < nn; n += (int64_t)gridDim.x * blockDim.x) {
    int ix = (int)(n % nnx), iz = (int)(n / nnx);
    int exs[2], ezs[2], nx = 0, nz = 0;
    if (ix & 1) exs[nx++] = ix >> 1;
    else { if (ix / 2 - 1 >= 0) exs[nx++] = ix / 2 - 1; if (ix / 2 < b.nelx) exs[nx++] = ix / 2; }
    if (iz & 1) ezs[nz++] = iz >> 1;
    else { if (iz / 2 - 1 >= 0) ezs[nz++] = iz / 2 - 1; if (iz / 2 < b.nelz) ezs[nz++] = iz / 2; }
    for (int c = 0; c < ndof; ++c) {
      double acc = 0.0;
      for (int a = 0; a < nz; ++a)
        for (int bb = 0; bb < nx; ++bb) {
          int ex = exs[bb], ez = ezs[a];
          int k = q2_local(ix - 2 * ex, iz - 2 * ez);
          acc += vel[((int64_t)ez * b.nelx + ex) * per + k * ndof + c];
        }
      out[n * ndof + c] = acc;
    }
  }
}

// Sum element-local Q1 vectors (4 per element) onto pressure nodes in ascending element order.
__global__ void k_gather_q1(mw_box b, const double* __restrict__ hel, double* __restrict__ out) {
  const int ncx = b.nelx + 1;
  const int64_t nn = (int64_t)ncx * (b.nelz + 1);
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < nn; n += (int64_t)gridDim.x * blockDim.x) {
    int i = (int)(n % ncx), j = (int)(n / ncx);
    double acc = 0.0;
    const int ex[4] = {i - 1, i, i - 1, i};
    const int ez[4] = {j - 1, j - 1, j, j};
    const int kk[4] = {2, 3, 1, 0};
    for (int s = 0; s < 4; ++s) {
      if (ex[s] < 0 || ex[s] >= b.nelx || ez[s] < 0 || ez[s] >= b.nelz) continue;
      acc += hel[((int64_t)ez[s] * b.nelx + ex[s]) * 4 + kk[s]];
    }
    out[n] = acc;
  }
}

// ------------------------------------------------------------------------------------------
template <typename R, typename S>
__global__ void __launch_bounds__(EB_T * 9)
k_assemble_energy(mw_box b, mw_energy_in in, S* __restrict__ vv, double* __restrict__ b_el) {
  __shared__ R NT[81], dNdr[81], dNds[81];
  __shared__ R dNdx[EB_T * 81], dNdy[EB_T * 81];
  __shared__ R Tloc[EB_T * 9];
  __shared__ int bfix[EB_T * 9];
  __shared__ double bval[EB_T * 9];
  const int64_t nel = (int64_t)b.nelx * b.nelz;
  const int64_t e0 = (int64_t)blockIdx.x * EB_T;
  const int ne = (int)((nel - e0) < EB_T ? (nel - e0) : EB_T);
  const int tid = threadIdx.x;
  const int nnx = 2 * b.nelx + 1;
  for (int i = tid; i < 81; i += blockDim.x) {
    NT[i] = (R)in.N_T[i]; dNdr[i] = (R)in.dNdr_T[i]; dNds[i] = (R)in.dNds_T[i];
  }
  for (int i = tid; i < ne * 9; i += blockDim.x) {
    int el = i / 9, k = i % 9;
    int64_t e = e0 + el;
    int64_t node = q2_node((int)(e % b.nelx), (int)(e / b.nelx), k, nnx);
    Tloc[i] = (R)in.T[node];                                                // :63
    bfix[i] = in.bc_fix_T[node] ? 1 : 0;
    bval[i] = in.bc_val_T[node];
  }
  __syncthreads();
  for (int i = tid; i < ne * 9; i += blockDim.x) {
    int el = i / 9, q = i % 9;
    int64_t g = (e0 + el) * 9 + q;
    R j00 = (R)in.jcbi00q[g], j01 = (R)in.jcbi01q[g], j10 = (R)in.jcbi10q[g], j11 = (R)in.jcbi11q[g];
    for (int k = 0; k < 9; ++k) {
      dNdx[el * 81 + q * 9 + k] = j00 * dNdr[q * 9 + k] + j01 * dNds[q * 9 + k];   // :71
      dNdy[el * 81 + q * 9 + k] = j10 * dNdr[q * 9 + k] + j11 * dNds[q * 9 + k];   // :72
    }
  }
  __syncthreads();
  const int el = tid / 9, i = tid % 9;
  if (el >= ne) return;
  const int64_t e = e0 + el;
  R MM[9], Kd[9], Ka[9], bs = 0;
#pragma unroll
  for (int j = 0; j < 9; ++j) { MM[j] = 0; Kd[j] = 0; Ka[j] = 0; }
  const R rho0 = (R)in.rho0;
  for (int q = 0; q < 9; ++q) {
    const int64_t g = e * 9 + q;
    const R jxw = (R)in.JxWq[g], hc = (R)in.hcapaq[g], hk = (R)in.hcondq[g];
    const R u = (R)in.uq[g], w = (R)in.wq[g];
    const R* N = NT + q * 9;
    const R* dx = dNdx + el * 81 + q * 9;
    const R* dy = dNdy + el * 81 + q * 9;
    const R Ni = N[i];
#pragma unroll
    for (int j = 0; j < 9; ++j) {
      MM[j] += Ni * N[j] * rho0 * hc * jxw;                                     // :77
      Kd[j] += (dx[i] * dx[j] + dy[i] * dy[j]) * hk * jxw;                      // :79
      Ka[j] += Ni * (u * dx[j] + w * dy[j]) * rho0 * hc * jxw;                  // :81
    }
    bs += Ni * (R)in.hprodq[g] * jxw;                                          // :83
    if (in.formulation == 1) {                                                  // :85-110 (EBA)
      const R exx = (R)in.exxq[g], ezz = (R)in.ezzq[g], exz = (R)in.exzq[g];
      bs += Ni * 2 * (R)in.etaq[g] *
            (R(2.0 / 3.0) * exx * exx + R(2.0 / 3.0) * ezz * ezz - R(2.0 / 3.0) * exx * ezz + 2 * exz * exz) * jxw;
      bs += Ni * (R)in.alphaq[g] * (R)in.Tq[g] * (-w * rho0 * 10) * jxw;
    }
  }
  const R dt = (R)(in.dt_dev ? *in.dt_dev : in.dt);
  bs *= dt;                                                                     // :112
  R A[9];
  R rhs = bs;
#pragma unroll
  for (int j = 0; j < 9; ++j) {
    A[j] = MM[j] + (Ka[j] + Kd[j]) * dt * R(0.5);                               // :114
    rhs += (MM[j] - (Ka[j] + Kd[j]) * dt * R(0.5)) * Tloc[el * 9 + j];          // :115
  }
  const int* fx = bfix + el * 9;
  const double* fv = bval + el * 9;
  if (fx[i]) {                                                                  // :118-130
    R ad = 0;
#pragma unroll
    for (int j = 0; j < 9; ++j) if (j == i) ad = A[j];
#pragma unroll
    for (int j = 0; j < 9; ++j) A[j] = (j == i) ? ad : R(0);
    rhs = ad * (R)fv[i];
  } else {
#pragma unroll
    for (int j = 0; j < 9; ++j)
      if (fx[j]) { rhs -= A[j] * (R)fv[j]; A[j] = 0; }
  }
  S* o = vv + e * 81 + i * 9;                                                   // :133-137
#pragma unroll
  for (int j = 0; j < 9; ++j) o[j] = (S)A[j];
  b_el[e * 9 + i] = (double)rhs;
}

// Body-force element vectors f_el[2i+c] = sum_q N_V[q,i] JxW rho g_c (build_matrix_stokes.py:141-143)
// without the element matrices; fixed dofs get 0 (their rhs is K_ii * bc_val = 0 when every
// Dirichlet value is zero, :215).
__global__ void k_body_force(mw_box b, const double* __restrict__ rhoq, const double* __restrict__ gxq,
                             const double* __restrict__ gzq, const double* __restrict__ JxWq,
                             const double* __restrict__ NV, const uint8_t* __restrict__ fix, double* __restrict__ fel) {
  __shared__ double N[81];
  for (int i = threadIdx.x; i < 81; i += blockDim.x) N[i] = NV[i];
  __syncthreads();
  const int64_t n = (int64_t)b.nelx * b.nelz * 9;
  const int nnx = 2 * b.nelx + 1;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n; g += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = g / 9;
    const int i = (int)(g % 9);
    double fx = 0.0, fz = 0.0;
    for (int q = 0; q < 9; ++q) {
      const int64_t gq = e * 9 + q;
      const double t = N[q * 9 + i] * JxWq[gq] * rhoq[gq];
      fx += t * gxq[gq];
      fz += t * gzq[gq];
    }
    const int64_t node = q2_node((int)(e % b.nelx), (int)(e / b.nelx), i, nnx);
    fel[e * 18 + 2 * i] = fix[2 * node] ? 0.0 : fx;
    fel[e * 18 + 2 * i + 1] = fix[2 * node + 1] ? 0.0 : fz;
  }
}

template <typename R, bool BLOCKS>
static int launch_stokes(const mw_box& b, const mw_stokes_in& in, const mw_stokes_out& out, double* fel, double* hel,
                         cudaStream_t s) {
  const int64_t nel = (int64_t)b.nelx * b.nelz;
  auto kern = k_assemble_stokes<R, BLOCKS>;
  constexpr size_t sm = StokesSmem<R, BLOCKS>::bytes;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess)
    return MW_ERR_CUDA;
  const void* const all[7] = {out.VV_Stokes, out.VV_K, out.VV_G, out.VV_GT, out.VV_M, out.VV_M_eta, out.VV_H};
  const int write = BLOCKS ? out.VV_K != nullptr : out.VV_Stokes != nullptr;
  int bulk = 1;                            // an element's results are a multiple of 16 bytes in every array
  for (int k = BLOCKS ? 1 : 0; k < (BLOCKS ? 7 : 1); ++k)
    if ((uintptr_t)all[k] & 15) bulk = 0;
  const unsigned grid = (unsigned)std::min<int64_t>((nel + EB_S - 1) / EB_S, StokesSmem<R, BLOCKS>::CTAS * num_sms());
  kern<<<grid, EB_S * 18, sm, s>>>(b, in, write, bulk, (R*)out.VV_Stokes, (R*)out.VV_K, (R*)out.VV_G, (R*)out.VV_GT,
                                   (R*)out.VV_M, (R*)out.VV_M_eta, (R*)out.VV_H, fel, hel);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

}  // namespace mw

using namespace mw;

extern "C" {

size_t mw_assemble_stokes_workspace_bytes(mw_box box) {
  return (size_t)box.nelx * box.nelz * 22 * sizeof(double);
}

int mw_assemble_stokes(mw_box box, int32_t blocks, int32_t precision, mw_stokes_in in, mw_stokes_out out, void* work,
                       size_t work_bytes, void* stream) {
  if (box.nelx <= 0 || box.nelz <= 0 || !out.rhs_f || !out.rhs_h) return MW_ERR_BAD_ARG;
  const bool rhs_only = !out.VV_Stokes && !out.VV_K;
  if (!rhs_only && (blocks ? !(out.VV_K && out.VV_G && out.VV_GT && out.VV_M && out.VV_M_eta && out.VV_H)
                           : !out.VV_Stokes))
    return MW_ERR_BAD_ARG;
  if (work_bytes < mw_assemble_stokes_workspace_bytes(box)) return MW_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  int64_t nel = (int64_t)box.nelx * box.nelz;
  double* fel = (double*)work;
  double* hel = fel + nel * 18;
  const bool f32 = precision == MW_F32;
  int rc = blocks ? (f32 ? launch_stokes<float, true>(box, in, out, fel, hel, s)
                         : launch_stokes<double, true>(box, in, out, fel, hel, s))
                  : (f32 ? launch_stokes<float, false>(box, in, out, fel, hel, s)
                         : launch_stokes<double, false>(box, in, out, fel, hel, s));
  if (rc) return rc;
  int64_t nn = (int64_t)(2 * box.nelx + 1) * (2 * box.nelz + 1);
  k_gather_q2<<<grid_for(nn, 256), 256, 0, s>>>(box, 2, fel, out.rhs_f);
  MW_CHECK_LAUNCH();
  int64_t np = (int64_t)(box.nelx + 1) * (box.nelz + 1);
  k_gather_q1<<<grid_for(np, 256), 256, 0, s>>>(box, hel, out.rhs_h);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

int mw_stokes_rhs_body(mw_box box, const double* rhoq, const double* gxq, const double* gzq, const double* JxWq,
                       const double* N_V, const uint8_t* bc_fix_V, double* rhs_f, double* rhs_h, void* work,
                       size_t work_bytes, void* stream) {
  if (box.nelx <= 0 || box.nelz <= 0 || !rhs_f || !rhs_h) return MW_ERR_BAD_ARG;
  if (work_bytes < mw_assemble_stokes_workspace_bytes(box)) return MW_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t nel = (int64_t)box.nelx * box.nelz;
  double* fel = (double*)work;
  k_body_force<<<grid_for(nel * 9, 256), 256, 0, s>>>(box, rhoq, gxq, gzq, JxWq, N_V, bc_fix_V, fel);
  MW_CHECK_LAUNCH();
  const int64_t nn = (int64_t)(2 * box.nelx + 1) * (2 * box.nelz + 1);
  k_gather_q2<<<grid_for(nn, 256), 256, 0, s>>>(box, 2, fel, rhs_f);
  MW_CHECK_LAUNCH();
  const int64_t np = (int64_t)(box.nelx + 1) * (box.nelz + 1);
  if (cudaMemsetAsync(rhs_h, 0, sizeof(double) * np, s) != cudaSuccess) return MW_ERR_CUDA;
  return MW_OK;
}

size_t mw_assemble_energy_workspace_bytes(mw_box box) {
  return (size_t)box.nelx * box.nelz * 9 * sizeof(double);
}

int mw_assemble_energy(mw_box box, int32_t precision, mw_energy_in in, void* VV_T, double* rhs, void* work,
                       size_t work_bytes, void* stream) {
  if (box.nelx <= 0 || box.nelz <= 0 || !VV_T || !rhs) return MW_ERR_BAD_ARG;
  if (work_bytes < mw_assemble_energy_workspace_bytes(box)) return MW_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  int64_t nel = (int64_t)box.nelx * box.nelz;
  double* bel = (double*)work;
  unsigned grid = (unsigned)((nel + EB_T - 1) / EB_T);
  if (precision == MW_F32) k_assemble_energy<float, float><<<grid, EB_T * 9, 0, s>>>(box, in, (float*)VV_T, bel);
  else k_assemble_energy<double, double><<<grid, EB_T * 9, 0, s>>>(box, in, (double*)VV_T, bel);
  MW_CHECK_LAUNCH();
  int64_t nn = (int64_t)(2 * box.nelx + 1) * (2 * box.nelz + 1);
  k_gather_q2<<<grid_for(nn, 256), 256, 0, s>>>(box, 1, bel, rhs);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

}  // extern "C"
