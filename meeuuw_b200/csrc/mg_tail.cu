// The coarse end of a V-cycle in one launch of one CTA (sm_100a).
//
// Levels whose cells (elements and the boundary's half cells) fit the threads of a CTA need no halo: a
// thread owns one cell, as in mg_level.cu, on every such level in turn.  Between levels that are not
// nested a launch each way costs 4 to 5 us a level (transfer tables, a wider halo) whatever it computes; a
// chain of odd sizes has more such levels than one of powers of two (150x97 elements: 19x13, 10x7 and 5x4
// above the coarsest 3x2).  Everything that the set-up wrote -- diagonals, viscosities, flags, transfer
// tables, as many rows of the coarsest inverse as fit -- is on its way into shared memory before the
// predecessor is waited for, all of it in flight together; only the first level's right-hand side is read
// after it.
//
// The arithmetic is that of the level launches and of the coarsest product in the same order: smoothing
// steps, node sums over the incident elements, transfer taps (from the tables, whose zero weights change
// nothing), FP64 row sums of the inverse.  The results equal a cycle of separate launches.
//
// Measured: 150x97 elements, FP32, the seven launches from 19x13 down 40 -> 31 us, a time step 11.9 ->
// 10.3 ms.  Bounded by the applies: 3000 clocks each at 280 cells (issue), 1800 at 30 (one warp's chain
// through nine Gauss points), 16 + 8 of them; transfers 2000 to 4400, the coarsest product 4000.
#include <algorithm>

#include "cell_ops.cuh"

namespace mw {

namespace {

constexpr int NT = MG_TAIL_CELLS;

struct TailTables {                                         // offsets of a direction's tables, bytes
  int pj, ri, rn, pw, rw;
};

template <typename R>
struct TailLayout {                                         // shared memory, byte offsets
  int dg[MG_TAIL_LEVELS], di[MG_TAIL_LEVELS], b[MG_TAIL_LEVELS], x[MG_TAIL_LEVELS], eta[MG_TAIL_LEVELS],
      fx[MG_TAIL_LEVELS];
  TailTables t[MG_TAIL_LEVELS][2];
  int work, xc, bd, fd, ainv, rows, total;

  int take(size_t bytes) {
    const int o = total;
    total += (int)((bytes + 15) / 16 * 16);
    return o;
  }
  // limit: bytes a CTA may have; false when the levels do not fit
  bool plan(const MgTailArgs<R>& a, int limit) {
    total = 0;
    size_t nc0 = 0, nnc = 0;
    for (int l = 0; l < a.n; ++l) {
      const LevelGeo &g = a.L[l].g, &c = l + 1 < a.n ? a.L[l + 1].g : a.gd;
      const size_t nc = (size_t)(g.nx + 1) * (g.nz + 1);
      nc0 = std::max(nc0, nc);
      nnc = std::max(nnc, (size_t)c.nnx * c.nnz);
      dg[l] = take(8 * sizeof(R) * nc);
      di[l] = take(8 * sizeof(R) * nc);
      b[l] = take(8 * sizeof(R) * nc);
      x[l] = take(8 * sizeof(R) * nc);
      eta[l] = take(sizeof(R) * nc);
      fx[l] = take(nc);
      for (int d = 0; d < 2; ++d) {
        const size_t nf = d ? g.nnz : g.nnx, mc = d ? c.nnz : c.nnx;
        t[l][d].pj = take(sizeof(int) * nf);
        t[l][d].ri = take(sizeof(int) * mc);
        t[l][d].rn = take(sizeof(int) * mc);
        t[l][d].pw = take(sizeof(double) * 3 * nf);
        t[l][d].rw = take(sizeof(double) * RTAPS * mc);
      }
    }
    work = take(std::max<size_t>(18 * sizeof(R), 8 * sizeof(double)) * nc0);   // exchange planes; FP64 residual
    xc = take(2 * sizeof(double) * nnc);                    // the coarse correction, FP64, by lattice node
    bd = take(sizeof(double) * a.nd);
    fd = take(a.nd);
    if (total > limit) return false;
    rows = std::min<int>(a.nd, (limit - total) / (int)(sizeof(double) * a.nd));
    ainv = take(sizeof(double) * a.nd * rows);
    return true;
  }
};

// N bytes (4, 8 or 16) to shared memory without waiting for them
template <int N> MW_D void copy_async(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;"
               :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "n"(N) : "memory");
}
template <typename T> MW_D void copy_all(unsigned char* dst, const T* src, int n) {
  for (int i = threadIdx.x; i < n; i += NT) copy_async<sizeof(T)>(reinterpret_cast<T*>(dst) + i, src + i);
}
MW_D void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> MW_D void copy_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(LEFT) : "memory"); }

// a level's constants on their way into shared memory, all in flight together (nodes off the lattice stay
// unset: nothing reads them); the Dirichlet bits of the thread's cell are returned
template <typename R>
MW_D unsigned stage_level(const MgTailLevel<R>& L, const LevelGeo& c, const TailLayout<R>& S, int l, unsigned char* sm) {
  typedef typename Vec2<R>::T R2;
  const LevelGeo& g = L.g;
  const int CX = g.nx + 1, NC = CX * (g.nz + 1), tid = threadIdx.x;
  R2 *dg = reinterpret_cast<R2*>(sm + S.dg[l]), *di = reinterpret_cast<R2*>(sm + S.di[l]);
  unsigned f = 0;
  if (tid < NC) {
    const int cx = tid % CX, cz = tid / CX;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if ((t & 1 && cx >= g.nx) || (t & 2 && cz >= g.nz)) continue;
      const int n = (2 * cz + (t >> 1)) * g.nnx + 2 * cx + (t & 1);
      copy_async<sizeof(R2)>(dg + t * NC + tid, reinterpret_cast<const R2*>(L.diag) + n);
      copy_async<sizeof(R2)>(di + t * NC + tid, reinterpret_cast<const R2*>(L.dinv) + n);
      const uchar2 u = reinterpret_cast<const uchar2*>(L.fix)[n];
      f |= ((u.x ? 1u : 0u) | (u.y ? 2u : 0u)) << (2 * t);
    }
    if (cx < g.nx && cz < g.nz)
      copy_async<sizeof(R)>(reinterpret_cast<R*>(sm + S.eta[l]) + tid, L.eta + cz * g.nx + cx);
  }
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    const Transfer1D& t = d ? L.tz : L.tx;
    const TailTables& o = S.t[l][d];
    const int nf = d ? g.nnz : g.nnx, mc = d ? c.nnz : c.nnx;
    copy_all(sm + o.pj, t.pj, nf);
    copy_all(sm + o.pw, t.pw, 3 * nf);
    copy_all(sm + o.ri, t.ri, mc);
    copy_all(sm + o.rn, t.rn, mc);
    copy_all(sm + o.rw, t.rw, RTAPS * mc);
  }
  return f;
}

// s = K x at the cell's nodes (the apply of k_mg_level without a halo); two block barriers
template <typename R, typename R2 = typename Vec2<R>::T>
MW_D void cell_apply(const LevelGeo& g, R ev, unsigned fx, bool inside, const R2 (&x)[4], const R2* dg, R2* work,
                     R2 (&s)[4]) {
  const int CX = g.nx + 1, NC = CX * (g.nz + 1), tid = threadIdx.x;
  const int cx = tid % CX, cz = tid / CX;
  R2 *sx = work, *se = work + 4 * NC;
  const R2 zero = pair(R(0), R(0));
  const R sxe = R(2.0 / g.hx), sze = R(2.0 / g.hz), jace = R(g.hx * g.hz / 4.0);
  R2 u[9], y[9];
  if (inside) {
    auto masked = [&](int t) {
      return pair((fx & (1u << (2 * t))) ? R(0) : x[t].x, (fx & (2u << (2 * t))) ? R(0) : x[t].y);
    };
    u[0] = masked(0); u[4] = masked(1); u[7] = masked(2); u[8] = masked(3);
    sx[tid] = u[0]; sx[NC + tid] = u[4]; sx[2 * NC + tid] = u[7]; sx[3 * NC + tid] = u[8];
  }
  __syncthreads();
  if (inside) {
    if (cx < g.nx && cz < g.nz) {
      u[1] = sx[tid + 1];
      u[5] = sx[2 * NC + tid + 1];
      u[3] = sx[tid + CX];
      u[6] = sx[NC + tid + CX];
      u[2] = sx[tid + CX + 1];
      R eq[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) eq[q] = ev;
      k_element(sxe, sze, jace, u, eq, y);
    } else {
#pragma unroll
      for (int k = 0; k < 9; ++k) y[k] = zero;
    }
    se[tid] = y[1]; se[NC + tid] = y[5]; se[2 * NC + tid] = y[3]; se[3 * NC + tid] = y[6]; se[4 * NC + tid] = y[2];
  }
  __syncthreads();
  if (!inside) return;
  // ascending element order: lower left, lower, left, own
  const bool hl = cx > 0, hb = cz > 0;
  const R2 p2 = hl && hb ? se[4 * NC + tid - CX - 1] : zero, p3 = hb ? se[2 * NC + tid - CX] : zero,
           p1 = hl ? se[tid - 1] : zero, p6 = hb ? se[3 * NC + tid - CX] : zero, p5 = hl ? se[NC + tid - 1] : zero;
  s[0] = pair(((p2.x + p3.x) + p1.x) + y[0].x, ((p2.y + p3.y) + p1.y) + y[0].y);
  s[1] = pair(p6.x + y[4].x, p6.y + y[4].y);
  s[2] = pair(p5.x + y[7].x, p5.y + y[7].y);
  s[3] = y[8];
#pragma unroll
  for (int t = 0; t < 4; ++t) {                             // eliminated rows act as K_ii u_i
    if (fx & (1u << (2 * t))) s[t].x = dg[t * NC + tid].x * x[t].x;
    if (fx & (2u << (2 * t))) s[t].y = dg[t * NC + tid].y * x[t].y;
  }
}

// The coarsest level: a row of the inverse a warp (lane j, j + 32, ... in order, then a shuffle tree, as the
// launch of its own sums it), four rows with their loads in flight together.
template <typename R>
MW_D void coarsest(const MgTailArgs<R>& A, const TailLayout<R>& S, const double* ainv, const double* bd, double* xd) {
  constexpr int ROWS = 4, STEP = 6, NW = NT / 32;
  const int lane = threadIdx.x & 31, nd = A.nd;
  for (int r0 = threadIdx.x >> 5; r0 < nd; r0 += ROWS * NW) {
    double s[ROWS] = {};
    for (int j0 = lane; j0 < nd; j0 += 32 * STEP) {
      double v[ROWS][STEP];
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const int row = r0 + i * NW;
        const double* p = row < S.rows ? ainv + row * nd : A.Ainv + (int64_t)row * nd;
#pragma unroll
        for (int k = 0; k < STEP; ++k) v[i][k] = row < nd && j0 + 32 * k < nd ? p[j0 + 32 * k] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < STEP; ++k) {
        if (j0 + 32 * k >= nd) break;
        const double b = bd[j0 + 32 * k];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) s[i] += v[i][k] * b;
      }
    }
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < ROWS; ++i) s[i] += __shfl_down_sync(0xffffffffu, s[i], o);
    if (lane == 0)
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
        if (r0 + i * NW < nd) xd[r0 + i * NW] = (double)(R)s[i];
  }
}

template <typename R, int DEG>
__global__ void __launch_bounds__(NT, 1) k_mg_tail(const __grid_constant__ MgTailArgs<R> A,
                                                   const __grid_constant__ TailLayout<R> S) {
  typedef typename Vec2<R>::T R2;
  extern __shared__ __align__(16) unsigned char tail_sm[];
  unsigned char* sm = tail_sm;
  const int tid = threadIdx.x;
  double2* xc = reinterpret_cast<double2*>(sm + S.xc);
  double* bd = reinterpret_cast<double*>(sm + S.bd);
  double* ainv = reinterpret_cast<double*>(sm + S.ainv);
  R2* work = reinterpret_cast<R2*>(sm + S.work);
  {
    unsigned f[MG_TAIL_LEVELS];
#pragma unroll
    for (int l = 0; l < MG_TAIL_LEVELS; ++l)
      f[l] = l < A.n ? stage_level(A.L[l], l + 1 < A.n ? A.L[l + 1].g : A.gd, S, l, sm) : 0u;
    copy_commit();
    copy_all(sm + S.ainv, reinterpret_cast<const double2*>(A.Ainv), A.nd * S.rows / 2);   // nd is even
    copy_commit();
    for (int i = tid; i < A.nd; i += NT) (sm + S.fd)[i] = A.fixd[i];
#pragma unroll
    for (int l = 0; l < MG_TAIL_LEVELS; ++l)
      if (l < A.n && tid < (A.L[l].g.nx + 1) * (A.L[l].g.nz + 1)) (sm + S.fx[l])[tid] = (unsigned char)f[l];
  }
  pdl_entry();

  // Down through the levels, the coarsest solve, up again.  One copy of the apply serves every step: a second
  // one costs its instruction fetches, 1100 clocks, in every launch.
#pragma unroll 1
  for (int step = 0; step < 2 * A.n; ++step) {
    const bool down = step < A.n;
    const int l = down ? step : 2 * A.n - 1 - step;
    if (step == A.n) {
      copy_wait<0>();
      __syncthreads();
      coarsest<R>(A, S, ainv, bd, reinterpret_cast<double*>(xc));
    }
    const MgTailLevel<R>& L = A.L[l];
    const LevelGeo& g = L.g;
    const LevelGeo& c = l + 1 < A.n ? A.L[l + 1].g : A.gd;
    const int CX = g.nx + 1, NC = CX * (g.nz + 1), cx = tid % CX, cz = tid / CX;
    const bool inside = tid < NC;
    const bool has[4] = {inside, inside && cx < g.nx, inside && cz < g.nz, inside && cx < g.nx && cz < g.nz};
    const R2 *dg = reinterpret_cast<const R2*>(sm + S.dg[l]), *di = reinterpret_cast<const R2*>(sm + S.di[l]);
    R2 *sb = reinterpret_cast<R2*>(sm + S.b[l]), *sx = reinterpret_cast<R2*>(sm + S.x[l]);
    const double c1s = DEG > 1 ? L.cheb[2] : 0.0;
    const R c20 = (R)L.cheb[1], c21 = DEG > 1 ? (R)L.cheb[3] : R(0);
    const TailTables &tx = S.t[l][0], &tz = S.t[l][1];
    const R2 zero = pair(R(0), R(0));
    R2 x[4], d[4], s[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) x[t] = d[t] = s[t] = zero;
    if (step == 0) {
#pragma unroll
      for (int t = 0; t < 4; ++t)
        if (has[t])
          sb[t * NC + tid] = reinterpret_cast<const R2*>(A.b)[(2 * cz + (t >> 1)) * g.nnx + 2 * cx + (t & 1)];
      copy_wait<1>();
    }
    __syncthreads();                                        // the constants; the residual or correction before
    unsigned fx = 0;
    R ev = R(0);
    if (inside) {
      fx = (sm + S.fx[l])[tid];
      ev = reinterpret_cast<const R*>(sm + S.eta[l])[tid];
    }
    if (down) {                                             // x0 = d0 = (1/theta) D^-1 b
#pragma unroll
      for (int t = 0; t < 4; ++t)
        if (has[t]) {
          const R2 b = sb[t * NC + tid];
          d[t] = x[t] = div2(pair(c20 * b.x, c20 * b.y), dg[t * NC + tid], di[t * NC + tid]);
        }
    } else {                                                // x + P x_c on the free components
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (!has[t]) continue;
        x[t] = sx[t * NC + tid];
        const int i = 2 * cx + (t & 1), k = 2 * cz + (t >> 1);
        const int J = reinterpret_cast<const int*>(sm + tx.pj)[i], K = reinterpret_cast<const int*>(sm + tz.pj)[k];
        const double *wx = reinterpret_cast<const double*>(sm + tx.pw) + 3 * i,
                     *wz = reinterpret_cast<const double*>(sm + tz.pw) + 3 * k;
        double s0 = 0, s1 = 0;
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int q = 0; q < 3; ++q) {                     // nodes past the end carry no weight
            const double w = wz[p] * wx[q];
            const double2 v = xc[min(K + p, c.nnz - 1) * c.nnx + min(J + q, c.nnx - 1)];
            s0 = fma(w, v.x, s0);
            s1 = fma(w, v.y, s1);
          }
        if (!(fx & (1u << (2 * t)))) x[t].x += (R)s0;
        if (!(fx & (2u << (2 * t)))) x[t].y += (R)s1;
      }
    }
#pragma unroll 1
    for (int j = 0; j < DEG; ++j) {
      cell_apply<R>(g, ev, fx, inside, x, dg, work, s);
      if (down && j == DEG - 1) break;
      const bool first = !down && j == 0;                   // the restart step reads no old direction
      const R c2 = first ? c20 : c21;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (!has[t]) continue;
        const R2 b = sb[t * NC + tid];
        R2 dn = div2(pair(c2 * (b.x - s[t].x), c2 * (b.y - s[t].y)), dg[t * NC + tid], di[t * NC + tid]);
        if (!first && c1s != 0.0) {
          dn.x += R(c1s) * d[t].x;
          dn.y += R(c1s) * d[t].y;
        }
        d[t] = dn;
        x[t] = pair(x[t].x + dn.x, x[t].y + dn.y);
      }
    }
    if (!down) {                                            // (xc was last read before the applies' barriers)
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (!has[t]) continue;
        const int n = (2 * cz + (t >> 1)) * g.nnx + 2 * cx + (t & 1);
        if (l == 0) reinterpret_cast<R2*>(A.x)[n] = x[t];
        else xc[n] = make_double2((double)x[t].x, (double)x[t].y);
      }
      continue;
    }
    __syncthreads();                                        // the exchange planes are read
    double2* sr = reinterpret_cast<double2*>(work);         // the residual, converted once
    if (inside) {
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        double2 r = make_double2(0.0, 0.0);
        if (has[t]) {
          const R2 b = sb[t * NC + tid];
          const R2 v = pair(b.x - s[t].x, b.y - s[t].y);
          r = make_double2((double)v.x, (double)v.y);
        }
        sr[t * NC + tid] = r;
        sx[t * NC + tid] = x[t];
      }
    }
    __syncthreads();
    const bool last = l + 1 == A.n;
    const int CC = c.nx + 1, NCC = CC * (c.nz + 1);
    for (int n = tid; n < c.nnx * c.nnz; n += NT) {
      const int J = n % c.nnx, K = n / c.nnx;
      const int fx0 = reinterpret_cast<const int*>(sm + tx.ri)[J], fz0 = reinterpret_cast<const int*>(sm + tz.ri)[K];
      const int nx = reinterpret_cast<const int*>(sm + tx.rn)[J], nz = reinterpret_cast<const int*>(sm + tz.rn)[K];
      const double *rwx = reinterpret_cast<const double*>(sm + tx.rw) + RTAPS * J,
                   *rwz = reinterpret_cast<const double*>(sm + tz.rw) + RTAPS * K;
      double wx[RTAPS], s0 = 0, s1 = 0;
#pragma unroll
      for (int q = 0; q < RTAPS; ++q) wx[q] = rwx[q];
      for (int p = 0; p < nz; ++p) {
        const double wz = rwz[p];
        const int row = ((fz0 + p) & 1) * 2 * NC + ((fz0 + p) >> 1) * CX;
#pragma unroll
        for (int q = 0; q < RTAPS; ++q)
          if (q < nx) {
            const double w = wz * wx[q];
            const double2 v = sr[row + ((fx0 + q) & 1) * NC + ((fx0 + q) >> 1)];
            s0 = fma(w, v.x, s0);
            s1 = fma(w, v.y, s1);
          }
      }
      if (last) {
        bd[2 * n] = (sm + S.fd)[2 * n] ? 0.0 : (double)(R)s0;
        bd[2 * n + 1] = (sm + S.fd)[2 * n + 1] ? 0.0 : (double)(R)s1;
      } else {
        const int t = (K & 1) * 2 + (J & 1), cell = (K >> 1) * CC + (J >> 1);
        const unsigned f = (unsigned)(sm + S.fx[l + 1])[cell] >> (2 * t);
        reinterpret_cast<R2*>(sm + S.b[l + 1])[t * NCC + cell] = pair(f & 1u ? R(0) : (R)s0, f & 2u ? R(0) : (R)s1);
      }
    }
  }
}

int tail_limit() {
  int v = 0;
  return cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, current_device()) == cudaSuccess ? v : 0;
}

template <typename R, int DEG>
bool launch_tail_deg(const MgTailArgs<R>& a, const TailLayout<R>& S, cudaStream_t s) {
  static OncePerDevice once;
  if (!raise_smem(once, k_mg_tail<R, DEG>, tail_limit())) return false;
  pdl_launch(k_mg_tail<R, DEG>, 1, NT, S.total, s, a, S);
  return true;
}

}  // namespace

template <typename R> bool mg_tail(const MgTailArgs<R>& a, int deg, cudaStream_t s) {
  TailLayout<R> S;
  if (!S.plan(a, tail_limit())) return false;
  if constexpr (mg_tail_degree<R>() > 1)
    if (deg > 1) return launch_tail_deg<R, MG_MAXDEG>(a, S, s);
  return deg <= 1 && launch_tail_deg<R, 1>(a, S, s);
}

int mg_tail_ensure_tables() { return ensure_cell_tables(); }

template bool mg_tail<float>(const MgTailArgs<float>&, int, cudaStream_t);
template bool mg_tail<double>(const MgTailArgs<double>&, int, cudaStream_t);

}  // namespace mw
