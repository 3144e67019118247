// Multigrid set-up kernels (sm_100a): the smoother intervals' power iterations over every level at
// once, and the coarsest level's inverse.
#include "cell_ops.cuh"
#include "mg_setup.cuh"

namespace mw {

namespace {

// One power iteration of every smoothed level: v / |v|, K, D^-1 and the new norm in one launch (a
// level's blocks follow the previous level's).  Four launches a level and iteration before, one
// level after the other: 26 launches a level, each at its latency on all levels but the finest.
template <typename R>
__global__ void __launch_bounds__(CELLS * CELLS, sizeof(R) == 4 ? 3 : 2) k_power_step(
    const __grid_constant__ PowerArgs<R> A) {
  pdl_entry();
  typedef typename Vec2<R>::T R2;
  constexpr int CX = CELLS, NC = CELLS * CELLS, T = CELLS - 2;
  __shared__ __align__(16) R2 sx[4 * NC];
  __shared__ __align__(16) R2 se[5 * NC];
  int l = 0;
  while (l + 1 < A.n && (int)blockIdx.x >= A.L[l + 1].block0) ++l;
  const PowerLevel<R>& L = A.L[l];
  const LevelGeo& g = L.g;
  const int block = blockIdx.x - L.block0, nblocks = (l + 1 < A.n ? A.L[l + 1].block0 : (int)gridDim.x) - L.block0;
  const int tid = threadIdx.x, lx = tid % CX, lz = tid / CX;
  const int ex0 = (block % L.tiles_x) * T, ez0 = (block / L.tiles_x) * T;
  const int ex = ex0 + lx - 1, ez = ez0 + lz - 1;
  const bool cx0 = ex >= 0 && ex <= g.nx, cx1 = ex >= 0 && ex < g.nx;
  const bool cz0 = ez >= 0 && ez <= g.nz, cz1 = ez >= 0 && ez < g.nz;
  const bool has[4] = {cx0 && cz0, cx1 && cz0, cx0 && cz1, cx1 && cz1};
  const int64_t n0 = (int64_t)(2 * ez) * g.nnx + 2 * ex;
  const R2 zero = pair(R(0), R(0));
  const bool elem = has[3] && lx < CX - 1 && lz < CELLS - 1;
  const double inv = 1.0 / sqrt(fmax(L.lam2[A.it == 0 ? 0 : 1 + (A.it & 1)], 1e-300));
  R2 x[4];
  unsigned fx = 0;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    x[t] = zero;
    if (has[t]) {
      const int64_t n = n0 + (t >> 1) * g.nnx + (t & 1);
      const R2 v = reinterpret_cast<const R2*>(L.vin)[n];
      x[t] = pair((R)((double)v.x * inv), (R)((double)v.y * inv));
      const uchar2 f = reinterpret_cast<const uchar2*>(L.fix)[n];
      fx |= ((f.x ? 1u : 0u) | (f.y ? 2u : 0u)) << (2 * t);
    }
  }
  R eq[9];
  if (elem) {
    const R* e = L.eta + (int64_t)ez * g.nx + ex;
#pragma unroll
    for (int q = 0; q < 9; ++q) eq[q] = e[q * L.qs];
  }
  R2 u[9], y[9];
  auto masked = [&](int t) {
    return pair((fx & (1u << (2 * t))) ? R(0) : x[t].x, (fx & (2u << (2 * t))) ? R(0) : x[t].y);
  };
  u[0] = masked(0); u[4] = masked(1); u[7] = masked(2); u[8] = masked(3);
  sx[tid] = u[0]; sx[NC + tid] = u[4]; sx[2 * NC + tid] = u[7]; sx[3 * NC + tid] = u[8];
  __syncthreads();
  if (elem) {
    u[1] = sx[tid + 1];
    u[5] = sx[2 * NC + tid + 1];
    u[3] = sx[tid + CX];
    u[6] = sx[NC + tid + CX];
    u[2] = sx[tid + CX + 1];
    k_element(R(2.0 / g.hx), R(2.0 / g.hz), R(g.hx * g.hz / 4.0), u, eq, y);
  } else {
#pragma unroll
    for (int k = 0; k < 9; ++k) y[k] = zero;
  }
  se[tid] = y[1]; se[NC + tid] = y[5]; se[2 * NC + tid] = y[3]; se[3 * NC + tid] = y[6]; se[4 * NC + tid] = y[2];
  __syncthreads();
  const int ownx = ex0 + T >= g.nx ? T + 1 : T, ownz = ez0 + T >= g.nz ? T + 1 : T;
  double v = 0;
  if (lx >= 1 && lx <= ownx && lz >= 1 && lz <= ownz && has[0]) {
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
        const R2 dg = reinterpret_cast<const R2*>(L.diag)[n], di = reinterpret_cast<const R2*>(L.dinv)[n];
        if (fx & (1u << (2 * t))) s[t].x = dg.x * x[t].x;   // eliminated rows act as K_ii u_i
        if (fx & (2u << (2 * t))) s[t].y = dg.y * x[t].y;
        const R2 w = div2(s[t], dg, di);
        reinterpret_cast<R2*>(L.vout)[n] = w;
        v += (double)w.x * (double)w.x + (double)w.y * (double)w.y;
      }
  }
  double sum;
  if (grid_sum(v, L.part, L.counter, block, nblocks, &sum)) {
    L.lam2[A.last ? 0 : 1 + ((A.it + 1) & 1)] = sum;
    if (A.last) cheb_coefficients(sum, L.deg, A.ratio, A.safety, L.cheb);
  }
}

// ---------------------------------------------------------------- coarsest level
// The inverse of the SPD coarsest K by the symmetric sweep operator (each pivot turns A into
// A - c c^T / d outside its row and column, which become c / d, and the pivot -1 / d; after all of them
// A is -K^-1).  One CTA; the lower triangle lives in registers, a 6 x 6 tile a thread, and a pivot
// passes only its column through shared memory: one barrier a pivot, 36 multiply-adds a thread.  The
// in-place elimination in shared memory it replaces moved the whole matrix through shared memory for
// every pivot (0.64 ms for 162 unknowns, most of a small model's set-up).
constexpr int DT = 6, DTILES = 29;                       // up to 174 unknowns
constexpr int DPAIRS = DTILES * (DTILES + 1) / 2;
constexpr int DTHREADS = 448;                            // >= DPAIRS
constexpr int DNEL = 16;                                 // elements: (2 nx + 1)(2 nz + 1) <= 87 leaves at most 16
static_assert(DTHREADS >= DPAIRS, "a thread per tile of the triangle");

template <typename R>
__global__ void __launch_bounds__(DTHREADS, 1) k_dense_inverse(LevelGeo g, const R* __restrict__ eta,
                                                              const uint8_t* __restrict__ fix, int nd,
                                                              double* __restrict__ Ainv) {
  pdl_entry();
  __shared__ double ke[DNEL * 324];
  __shared__ double col[2][DT * DTILES];
  __shared__ double piv[2];
  const int tid = threadIdx.x;
  int I = 0;                                             // tile (I, J) of the triangle, row by row
  while ((I + 1) * (I + 2) / 2 <= tid) ++I;
  const int J = tid - I * (I + 1) / 2;
  const bool live = I * DT < nd;
  double A[DT][DT];
#pragma unroll
  for (int a = 0; a < DT; ++a)
#pragma unroll
    for (int b = 0; b < DT; ++b) A[a][b] = 0.0;
  const double sx = 2.0 / g.hx, sz = 2.0 / g.hz, jac = g.hx * g.hz / 4.0;
  const int nel = g.nx * g.nz;
  for (int i = tid; i < nel * 324; i += DTHREADS) {      // the element matrices
    const int e = i / 324, t = i % 324, ki = (t / 18) >> 1, ci = (t / 18) & 1, kj = (t % 18) >> 1, cj = (t % 18) & 1;
    double v = 0;
    for (int q = 0; q < 9; ++q) {
      const double dxi = sx * c_k.dr[q * 9 + ki], dzi = sz * c_k.dt[q * 9 + ki];
      const double dxj = sx * c_k.dr[q * 9 + kj], dzj = sz * c_k.dt[q * 9 + kj];
      double bb;
      if (ci == 0 && cj == 0) bb = 2 * dxi * dxj + dzi * dzj;
      else if (ci == 0) bb = dzi * dxj;
      else if (cj == 0) bb = dxi * dzj;
      else bb = 2 * dzi * dzj + dxi * dxj;
      v += bb * (double)eta[(int64_t)e * 9 + q] * jac * c_k.wq[q];
    }
    ke[i] = v;
  }
  __syncthreads();
  if (live) {
    int xi[DT], zi[DT], xj[DT], zj[DT];                  // lattice places of the tile's rows and columns
#pragma unroll
    for (int a = 0; a < DT; ++a) {
      const int ni = (I * DT + a) >> 1, nj = (J * DT + a) >> 1;
      xi[a] = ni % g.nnx; zi[a] = ni / g.nnx;
      xj[a] = nj % g.nnx; zj[a] = nj / g.nnx;
    }
    // an element's local dof at lattice offset (dx, dz), component c; -1 when it is not the element's
    auto local = [](int dx, int dz, int c) {
      if (dx < 0 || dx > 2 || dz < 0 || dz > 2) return -1;
      const int k = dz == 0 ? (dx == 0 ? 0 : (dx == 1 ? 4 : 1))
                            : (dz == 1 ? (dx == 0 ? 7 : (dx == 1 ? 8 : 5)) : (dx == 0 ? 3 : (dx == 1 ? 6 : 2)));
      return 2 * k + c;
    };
    for (int e = 0; e < nel; ++e) {                      // ascending order
      const int ex = 2 * (e % g.nx), ez = 2 * (e / g.nx);
      int li[DT], lj[DT];
#pragma unroll
      for (int a = 0; a < DT; ++a) {
        li[a] = I * DT + a < nd ? local(xi[a] - ex, zi[a] - ez, a & 1) : -1;
        lj[a] = J * DT + a < nd ? local(xj[a] - ex, zj[a] - ez, a & 1) : -1;
      }
#pragma unroll
      for (int a = 0; a < DT; ++a)
#pragma unroll
        for (int b = 0; b < DT; ++b)
          if (li[a] >= 0 && lj[b] >= 0) A[a][b] += ke[e * 324 + li[a] * 18 + lj[b]];
    }
  }
  // Dirichlet elimination: fixed rows and columns zero except the diagonal
  if (live) {
#pragma unroll
    for (int a = 0; a < DT; ++a)
#pragma unroll
      for (int b = 0; b < DT; ++b) {
        const int i = I * DT + a, j = J * DT + b;
        if (i < nd && j < nd && i != j && (fix[i] || fix[j])) A[a][b] = 0.0;
      }
  }
  const int ntile = (nd + DT - 1) / DT;
  for (int K = 0; K < ntile; ++K) {
#pragma unroll
    for (int kk = 0; kk < DT; ++kk) {
      const int k = K * DT + kk;
      if (k >= nd) break;
      const int buf = kk & 1;
      double* c = col[buf];
      if (live && J == K) {                              // (threads past the triangle have rows past the column)
#pragma unroll
        for (int a = 0; a < DT; ++a) c[I * DT + a] = A[a][kk];
        if (I == K) piv[buf] = 1.0 / A[kk][kk];
      } else if (live && I == K) {
#pragma unroll
        for (int b = 0; b < DT; ++b) c[J * DT + b] = A[kk][b];
      }
      __syncthreads();
      if (!live) continue;
      const double r = piv[buf];
      double ci[DT], cj[DT];
#pragma unroll
      for (int a = 0; a < DT; ++a) {
        ci[a] = c[I * DT + a];
        cj[a] = c[J * DT + a];
      }
#pragma unroll
      for (int a = 0; a < DT; ++a) {
        const double t = -(ci[a] * r);
#pragma unroll
        for (int b = 0; b < DT; ++b) A[a][b] = fma(t, cj[b], A[a][b]);
      }
      if (I == K) {
#pragma unroll
        for (int b = 0; b < DT; ++b) A[kk][b] = cj[b] * r;
      }
      if (J == K) {
#pragma unroll
        for (int a = 0; a < DT; ++a) A[a][kk] = ci[a] * r;
        if (I == K) A[kk][kk] = -r;
      }
    }
  }
  if (live) {
#pragma unroll
    for (int a = 0; a < DT; ++a)
#pragma unroll
      for (int b = 0; b < DT; ++b) {
        const int i = I * DT + a, j = J * DT + b;
        if (i < nd && j < nd) {
          Ainv[(int64_t)i * nd + j] = -A[a][b];
          if (I != J) Ainv[(int64_t)j * nd + i] = -A[a][b];
        }
      }
  }
}

}  // namespace

int setup_ensure_tables() { return ensure_cell_tables(); }

int power_tiles_x(int nx) {
  constexpr int T = CELLS - 2;
  return (nx + T - 1) / T;
}
int power_blocks(int nx, int nz) { return power_tiles_x(nx) * power_tiles_x(nz); }

template <typename R> void power_step(const PowerArgs<R>& a, int blocks, cudaStream_t s) {
  pdl_launch(k_power_step<R>, blocks, CELLS * CELLS, 0, s, a);
}

template <typename R>
bool dense_inverse(const LevelGeo& g, const R* eta, const uint8_t* fix, int nd, double* Ainv, cudaStream_t s) {
  if (nd > DT * DTILES || g.nx * g.nz > DNEL) return false;
  pdl_launch(k_dense_inverse<R>, 1, DTHREADS, 0, s, g, eta, fix, nd, Ainv);
  return true;
}

template void power_step<float>(const PowerArgs<float>&, int, cudaStream_t);
template void power_step<double>(const PowerArgs<double>&, int, cudaStream_t);
template bool dense_inverse<float>(const LevelGeo&, const float*, const uint8_t*, int, double*, cudaStream_t);
template bool dense_inverse<double>(const LevelGeo&, const double*, const uint8_t*, int, double*, cudaStream_t);

}  // namespace mw
