// The matrix-free Stokes operator y = [K G; G^T 0] (u, p) on a level, and residuals of it (sm_100a).
//
// A CTA takes a tile of 16 x 16 cells and owns 14 x 14 of them: one halo cell on the left and below for
// the neighbours' sums, one on the right and above for their nodes.  Each thread loads its cell's four
// nodes, hands the shared ones to its neighbours through shared memory, computes one element product and
// exchanges the sums for shared nodes the same way; its own four nodes never leave its registers.  The
// element-tile form this replaces staged the velocity and every element's 22 results in shared memory and
// looked its indices up per node: 1065 warp instructions an element, of which 370 were the product.
//
// Measured, (u, p) -> (K u + G p, G^T u), before and now: FP32 512^2 17.5 -> 16.2 us, 128^2 5.3 -> 3.7, 8^2
// 4.9 -> 3.5; FP64 512^2 42.5 -> 34.4, 256^2 14.3 -> 12.8.  At 512^2 the packed multiply-adds alone take 5.9 us
// (they issue at half rate); the rest is the load and exchange latency that two tiles an SM leave open.
#include "cell_ops.cuh"
#include "op_apply.cuh"

namespace mw {

namespace {

// Resident CTAs: two, or three where 80 registers do without spills (FP32 without pressure).  FP64
// with two (128 registers, 156 bytes spilled with pressure) takes 31 us at 512^2 against 36 with one.
enum { OP_PLAIN = 0, OP_PCG, OP_SUM };

template <typename R, bool PRESSURE, int KIND, typename X>
__global__ void __launch_bounds__(CELLS * CELLS, sizeof(R) == 4 && !PRESSURE ? 3 : 2) k_op_apply(OpArgs<R> a,
                                                                                                 X dir) {
  if (KIND != OP_PCG) pdl_entry();
  typedef typename Vec2<R>::T R2;
  constexpr int CX = CELLS, NC = CELLS * CELLS, T = CELLS - 2;
  constexpr bool PCG = KIND == OP_PCG;
  __shared__ __align__(16) R2 sx[4 * NC];
  __shared__ __align__(16) R2 se[5 * NC];
  __shared__ R sp[PRESSURE ? 4 * NC : 1];
  const int tid = threadIdx.x, lx = tid % CX, lz = tid / CX;
  const int ex0 = blockIdx.x * T, ez0 = blockIdx.y * T;
  const int ex = ex0 + lx - 1, ez = ez0 + lz - 1;
  const LevelGeo& g = a.g;
  const bool cx0 = ex >= 0 && ex <= g.nx, cx1 = ex >= 0 && ex < g.nx;
  const bool cz0 = ez >= 0 && ez <= g.nz, cz1 = ez >= 0 && ez < g.nz;
  const bool has[4] = {cx0 && cz0, cx1 && cz0, cx0 && cz1, cx1 && cz1};
  const int64_t n0 = (int64_t)(2 * ez) * g.nnx + 2 * ex;
  const int64_t np = (int64_t)ez * (g.nx + 1) + ex;
  const R2 zero = pair(R(0), R(0));
  const bool elem = has[3] && lx < CX - 1 && lz < CELLS - 1;
  R2 x[4];
  unsigned fx = 0;
  R eq[9];
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (has[t]) {
      const uchar2 f = reinterpret_cast<const uchar2*>(a.fix)[n0 + (t >> 1) * g.nnx + (t & 1)];
      fx |= ((f.x ? 1u : 0u) | (f.y ? 2u : 0u)) << (2 * t);
    }
  if (elem) {
    const R* e = a.eta + ((int64_t)ez * g.nx + ex) * a.es;
#pragma unroll
    for (int q = 0; q < 9; ++q) eq[q] = e[q * a.qs];
  }
  const R* pold = nullptr;
  double beta = 0.0;
  int k = 0;
  if constexpr (PCG) {
    pdl_entry();                                            // (the flags and the viscosity are the set-up's)
    k = (int)*dir.it;
    if (k > 0) {
      beta = dir.rz[k & 1] / dir.rz[(k & 1) ^ 1];
      pold = (k & 1) ? dir.pbuf[0] : dir.pbuf[1];
    }
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    x[t] = zero;
    if (has[t]) {
      const int64_t n = n0 + (t >> 1) * g.nnx + (t & 1);
      if constexpr (PCG) {
        x[t] = reinterpret_cast<const R2*>(dir.z)[n];
        if (pold) {
          const R2 q = reinterpret_cast<const R2*>(pold)[n];
          x[t] = pair((R)((double)x[t].x + beta * (double)q.x), (R)((double)x[t].y + beta * (double)q.y));
        }
      } else if (a.u) {
        x[t] = reinterpret_cast<const R2*>(a.u)[n];
      }
    }
  }
  R p0 = R(0);
  if (PRESSURE && a.p && has[0]) p0 = a.p[np];
  R2 u[9], y[9];
  R yp[4] = {R(0), R(0), R(0), R(0)};
  auto masked = [&](int t) {
    return pair((fx & (1u << (2 * t))) ? R(0) : x[t].x, (fx & (2u << (2 * t))) ? R(0) : x[t].y);
  };
  u[0] = masked(0); u[4] = masked(1); u[7] = masked(2); u[8] = masked(3);
  sx[tid] = u[0]; sx[NC + tid] = u[4]; sx[2 * NC + tid] = u[7]; sx[3 * NC + tid] = u[8];
  if (PRESSURE) sp[tid] = p0;
  __syncthreads();
  if (elem) {
    u[1] = sx[tid + 1];
    u[5] = sx[2 * NC + tid + 1];
    u[3] = sx[tid + CX];
    u[6] = sx[NC + tid + CX];
    u[2] = sx[tid + CX + 1];
    const R sxe = R(2.0 / g.hx), sze = R(2.0 / g.hz), jace = R(g.hx * g.hz / 4.0);
    if constexpr (PRESSURE) {
      const R pe[4] = {p0, sp[tid + 1], sp[tid + CX + 1], sp[tid + CX]};
      k_element<true>(sxe, sze, jace, u, eq, y, R(g.s), pe, yp);
    } else {
      k_element(sxe, sze, jace, u, eq, y);
    }
  } else {
#pragma unroll
    for (int k = 0; k < 9; ++k) y[k] = zero;
  }
  se[tid] = y[1]; se[NC + tid] = y[5]; se[2 * NC + tid] = y[3]; se[3 * NC + tid] = y[6]; se[4 * NC + tid] = y[2];
  if (PRESSURE) { sp[NC + tid] = yp[1]; sp[2 * NC + tid] = yp[3]; sp[3 * NC + tid] = yp[2]; }
  __syncthreads();
  const int ownx = ex0 + T >= g.nx ? T + 1 : T, ownz = ez0 + T >= g.nz ? T + 1 : T;
  const bool own = lx >= 1 && lx <= ownx && lz >= 1 && lz <= ownz && has[0];
  if (KIND == OP_PLAIN && !own) return;
  double v = 0;
  if (own && (PCG || a.yV)) {
    // ascending element order: lower left, lower, left, own
    const R2 p2 = se[4 * NC + tid - CX - 1], p3 = se[2 * NC + tid - CX], p1 = se[tid - 1],
             p6 = se[3 * NC + tid - CX], p5 = se[NC + tid - 1];
    R2 s[4];
    s[0] = pair(((p2.x + p3.x) + p1.x) + y[0].x, ((p2.y + p3.y) + p1.y) + y[0].y);
    s[1] = pair(p6.x + y[4].x, p6.y + y[4].y);
    s[2] = pair(p5.x + y[7].x, p5.y + y[7].y);
    s[3] = y[8];
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (has[t]) {
        const int64_t n = n0 + (t >> 1) * g.nnx + (t & 1);
        const unsigned f = (fx >> (2 * t)) & 3u;
        if (f) {                                            // eliminated rows act as K_ii u_i
          const R2 dg = PCG || a.u ? reinterpret_cast<const R2*>(a.diag)[n] : zero;
          if (f & 1u) s[t].x = dg.x * x[t].x;
          if (f & 2u) s[t].y = dg.y * x[t].y;
        }
        if constexpr (PCG) {
          reinterpret_cast<R2*>((k & 1) ? dir.pbuf[1] : dir.pbuf[0])[n] = x[t];
          v += (double)x[t].x * (double)s[t].x + (double)x[t].y * (double)s[t].y;
        } else if (a.bV) {
          const R2 b = reinterpret_cast<const R2*>(a.bV)[n];
          s[t] = pair(b.x - s[t].x, b.y - s[t].y);
          if (KIND == OP_SUM) v += (double)s[t].x * (double)s[t].x + (double)s[t].y * (double)s[t].y;
        }
        reinterpret_cast<R2*>(a.yV)[n] = s[t];
      }
  }
  if (PRESSURE && own && a.yP) {                            // the elements lower left, lower, left, own
    R r = ((sp[3 * NC + tid - CX - 1] + sp[2 * NC + tid - CX]) + sp[NC + tid - 1]) + yp[0];
    if (a.bP) r = a.bP[np] - r;
    a.yP[np] = r;
    if (KIND == OP_SUM) v += (double)r * (double)r;
  }
  if constexpr (KIND != OP_PLAIN) {
    double sum;
    if (grid_sum(v, dir.part, dir.counter, blockIdx.y * gridDim.x + blockIdx.x, gridDim.x * gridDim.y, &sum)) {
      if constexpr (PCG) *dir.pap = sum;
      else residual_done(dir.sc, sum, dir.action, dir.test);
    }
  }
}

}  // namespace

int op_ensure_tables() { return ensure_cell_tables(); }

template <typename R> static dim3 tiles(const OpArgs<R>& a) {
  constexpr int T = CELLS - 2;
  return dim3((a.g.nx + T - 1) / T, (a.g.nz + T - 1) / T);
}

int cell_partials(int nx, int nz) {
  constexpr int T = CELLS - 2 * MG_MAXDEG;           // the smallest tile among the launches that sum
  return ((nx + T - 1) / T) * ((nz + T - 1) / T);
}

struct NoExtra {};

template <typename R> void op_apply(const OpArgs<R>& a, cudaStream_t s) {
  if (a.p || a.yP) pdl_launch(k_op_apply<R, true, OP_PLAIN, NoExtra>, tiles(a), CELLS * CELLS, 0, s, a, NoExtra());
  else pdl_launch(k_op_apply<R, false, OP_PLAIN, NoExtra>, tiles(a), CELLS * CELLS, 0, s, a, NoExtra());
}

template <typename R> void op_pcg_direction(const OpArgs<R>& a, const PcgDir<R>& d, cudaStream_t s) {
  pdl_launch(k_op_apply<R, false, OP_PCG, PcgDir<R>>, tiles(a), CELLS * CELLS, 0, s, a, d);
}

void op_residual(const OpArgs<double>& a, const ResidSum& r, cudaStream_t s) {
  pdl_launch(k_op_apply<double, true, OP_SUM, ResidSum>, tiles(a), CELLS * CELLS, 0, s, a, r);
}

template void op_apply<float>(const OpArgs<float>&, cudaStream_t);
template void op_apply<double>(const OpArgs<double>&, cudaStream_t);
template void op_pcg_direction<float>(const OpArgs<float>&, const PcgDir<float>&, cudaStream_t);
template void op_pcg_direction<double>(const OpArgs<double>&, const PcgDir<double>&, cudaStream_t);

}  // namespace mw
