// A multigrid level's half of a V-cycle in one launch (sm_100a).
//
// The downward half smooths from a zero guess (Chebyshev-Jacobi, x0 = D^-1 b / theta, then deg - 1
// steps), forms the residual b - K x and restricts it; the upward half adds the prolonged coarse
// correction and smooths again.  A launch per operator apply and per transfer (three down, three
// up in FP32) costs a level its launch latency six times over and writes x, d and r to memory in
// between: every level of 128^2 elements and below took 25 us a cycle whatever its size.  Here a CTA
// takes a tile with enough halo for all its applies (temporal blocking) and keeps every vector of
// the tile in registers and shared memory; only b, x, the diagonal and the viscosity are read and x
// and the coarse right-hand side written.
//
// Layout: a thread owns one cell, that is one element and the four lattice nodes of its lower-left
// quadrant (corner, bottom midpoint, left midpoint, centre).  An apply exchanges, through shared
// memory planes with unit stride over the threads, the values of the five nodes an element shares
// with its right and upper neighbours, and afterwards the five sums it computed for them.  The halo
// shrinks by one cell a side and apply; a tile of 16 x 16 cells owns 16 - 2 deg - 2 a side downward and
// 16 - 2 deg upward.  Tiles of 32 x 16 cells repeat less (owning 26 x 10 and 28 x 12 of them in
// FP32) but were slower at every size (V-cycle at 512^2 180 against 169 us, at 64^2 42 against 37).
//
// Measured, FP32 V-cycle from launch to launch (the separate launches before): 512^2 293 -> 158 us,
// 256^2 184 -> 79, 128^2 139 -> 52, 64^2 107 -> 37, 8^2 31 -> 11; FP64, one smoothing step: 512^2 309 ->
// 232, 128^2 104 -> 55.
//
// The arithmetic -- element products, node sums over the incident elements in ascending order,
// smoothing steps, transfer taps -- is that of the kernels of stokes.cu in the same order, so the
// results equal a cycle of separate launches.
#include "cell_ops.cuh"

namespace mw {

namespace {

// the restriction taps along one direction for a coarse node of parity P: fine offsets and weights
template <int P> struct RTap;
template <> struct RTap<0> {
  static constexpr int n = 5;
  MW_D static constexpr int off(int i) { return i == 0 ? -3 : (i == 1 ? -1 : (i == 2 ? 0 : (i == 3 ? 1 : 3))); }
  MW_D static constexpr double w(int i) { return (i == 0 || i == 4) ? -0.125 : (i == 2 ? 1.0 : 0.375); }
};
template <> struct RTap<1> {
  static constexpr int n = 3;
  MW_D static constexpr int off(int i) { return i - 1; }
  MW_D static constexpr double w(int i) { return i == 1 ? 1.0 : 0.75; }
};

// sum of the taps of the coarse node whose cell is at index c of the planes sr[4][NC] (row length CX)
template <int PX, int PZ, int CX, int NC, typename R2>
MW_D void restrict_taps(const R2* sr, int c, double* s0, double* s1) {
  double a0 = 0, a1 = 0;
  static_for<RTap<PZ>::n>([&](auto tz) {
    constexpr int oz = RTap<PZ>::off(tz.value);
    static_for<RTap<PX>::n>([&](auto tx) {
      constexpr int ox = RTap<PX>::off(tx.value);
      constexpr double w = RTap<PZ>::w(tz.value) * RTap<PX>::w(tx.value);
      constexpr int plane = (oz & 1) * 2 + (ox & 1), dz = oz < 0 ? -((1 - oz) / 2) : oz / 2,
                    dx = ox < 0 ? -((1 - ox) / 2) : ox / 2;
      const R2 v = sr[plane * NC + c + dz * CX + dx];
      a0 = fma(w, (double)v.x, a0);
      a1 = fma(w, (double)v.y, a1);
    });
  });
  *s0 = a0;
  *s1 = a1;
}

// owned cells a side of a tile.  Downward between levels that are not nested a coarse node's taps reach
// up to four fine nodes to its right (three between nested ones), one cell more of halo.
constexpr int owned_cells(bool restricts, int applies, bool nested) {
  return CELLS - 2 * applies - (restricts ? (nested ? 2 : 3) : 0);
}

// DOWN: pre-smoothing, residual, restriction; else correction and post-smoothing.  DEG: smoothing
// steps.  PLANES: nine viscosity planes (else one value per element).  NESTED: both element counts
// halve (compile-time taps); else the transfer tables.  PART: downward with DEG = 2, the smoothing
// (PART_SMOOTH) or the residual of a.xin and its restriction (PART_RESID) alone.
enum { PART_ALL = 0, PART_SMOOTH, PART_RESID };
template <typename R, int DEG, bool DOWN, bool PLANES, bool NESTED, int PART = PART_ALL>
__global__ void __launch_bounds__(CELLS * CELLS, sizeof(R) == 4 ? 2 : 1) k_mg_level(MgArgs<R> a) {
  typedef typename Vec2<R>::T R2;
  constexpr int CX = CELLS, CZ = CELLS, NC = CX * CZ;
  constexpr int J0 = PART == PART_RESID ? DEG - 1 : 0, J1 = PART == PART_SMOOTH ? DEG - 1 : DEG;   // applies
  constexpr int AP = J1 - J0;
  constexpr bool RESTRICT = DOWN && PART != PART_SMOOTH;
  constexpr int LO = RESTRICT ? AP + 1 : AP;                // halo cells on the left and below
  constexpr int TX = owned_cells(RESTRICT, AP, NESTED), TZ = TX;
  constexpr int WX = NESTED ? CX + 3 : 26, WZ = WX;         // staged coarse nodes (upward): not nested, the 32
                                                            // fine nodes span at most 25 (nf / nc >= 3 / 2)
  static_assert(PART == PART_ALL || (DOWN && DEG > 1), "only a smoothing step and a residual are split");
  static_assert(!NESTED || TX % 2 == 0, "tiles start at even cells (transfer parity)");
  __shared__ __align__(16) R2 sx[4 * NC];                   // masked x (then the residual) by node type
  __shared__ __align__(16) R2 se[5 * NC];                   // sums for the right and upper neighbours
  __shared__ __align__(16) double2 sc[DOWN ? 1 : WX * WZ];
  constexpr int CN = RESTRICT && !NESTED ? 16 : 1;          // coarse nodes a tile restricts to, per side (at most 16)
  __shared__ double sw[2][CN][RTAPS];                       // their weights, first fine nodes and counts
  __shared__ int si[2][CN], sn[2][CN];
  const int tid = threadIdx.x, lx = tid % CX, lz = tid / CX;
  const int ex0 = blockIdx.x * TX, ez0 = blockIdx.y * TZ;
  const int ex = ex0 + lx - LO, ez = ez0 + lz - LO;
  const LevelGeo& g = a.g;
  // which of the cell's nodes lie on the lattice (the cells past the last element own the right and
  // top boundary nodes)
  const bool cx0 = ex >= 0 && ex <= g.nx, cx1 = ex >= 0 && ex < g.nx;
  const bool cz0 = ez >= 0 && ez <= g.nz, cz1 = ez >= 0 && ez < g.nz;
  const bool has[4] = {cx0 && cz0, cx1 && cz0, cx0 && cz1, cx1 && cz1};
  const int64_t n0 = (int64_t)(2 * ez) * g.nnx + 2 * ex;
  const R2 zero = pair(R(0), R(0));
  R2 b[4], dg[4], di[4], x[4], d[4];
  unsigned fx = 0;                                          // bit 2 t + c: component c of node t is fixed
  // what the set-up wrote, before the predecessor's results are waited for
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int64_t n = n0 + (t >> 1) * g.nnx + (t & 1);
    b[t] = dg[t] = di[t] = x[t] = zero;
    if (has[t]) {
      dg[t] = reinterpret_cast<const R2*>(a.diag)[n];
      di[t] = reinterpret_cast<const R2*>(a.dinv)[n];
      const uchar2 f = reinterpret_cast<const uchar2*>(a.fix)[n];
      fx |= ((f.x ? 1u : 0u) | (f.y ? 2u : 0u)) << (2 * t);
    }
  }
  R eq[9];
  if (has[3]) {
    const int64_t e = (int64_t)ez * g.nx + ex, nel = (int64_t)g.nx * g.nz;
    if (PLANES) {
#pragma unroll
      for (int q = 0; q < 9; ++q) eq[q] = a.eta[q * nel + e];
    } else {
      const R v = a.eta[e];
#pragma unroll
      for (int q = 0; q < 9; ++q) eq[q] = v;
    }
  } else {
#pragma unroll
    for (int q = 0; q < 9; ++q) eq[q] = R(0);
  }
  int j0 = 0, k0 = 0, mx = 0, mz = 0;                       // the coarse nodes on the tile's owned cells: coarse
  if constexpr (RESTRICT && !NESTED) {                      // node J lies at fine lattice position J nf / nc
    auto first = [](int c, int nf, int nc) { return (int)((2LL * c * nc + nf - 1) / nf); };
    j0 = first(ex0, g.nx, a.gc.nx);
    k0 = first(ez0, g.nz, a.gc.nz);
    mx = (ex0 + TX >= g.nx ? a.gc.nnx : first(ex0 + TX, g.nx, a.gc.nx)) - j0;
    mz = (ez0 + TZ >= g.nz ? a.gc.nnz : first(ez0 + TZ, g.nz, a.gc.nz)) - k0;
    for (int i = tid; i < 2 * CN * RTAPS; i += NC) {
      const int dir = i / (CN * RTAPS), j = i / RTAPS % CN, q = i % RTAPS;
      if (j >= (dir ? mz : mx)) continue;
      const Transfer1D& t = dir ? a.tz : a.tx;
      const int J = (dir ? k0 : j0) + j;
      sw[dir][j][q] = t.rw[RTAPS * J + q];
      if (q == 0) {
        si[dir][j] = t.ri[J];
        sn[dir][j] = t.rn[J];
      }
    }
  }
  int pj[2][2] = {{0, 0}, {0, 0}};                          // the taps of the cell's two columns and two rows
  double pw[2][2][3];
  if constexpr (!DOWN && !NESTED) {
#pragma unroll
    for (int dir = 0; dir < 2; ++dir)
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const Transfer1D& tr = dir ? a.tz : a.tx;
        const int i = min(max(2 * (dir ? ez : ex) + t, 0), (dir ? g.nnz : g.nnx) - 1);
        pj[dir][t] = tr.pj[i];
#pragma unroll
        for (int q = 0; q < 3; ++q) pw[dir][t][q] = tr.pw[3 * i + q];
      }
  }
  pdl_entry();
  const double c1s = DEG > 1 ? a.cheb[2] : 0.0;
  const R c20 = (R)a.cheb[1], c21 = DEG > 1 ? (R)a.cheb[3] : R(0);
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (has[t]) {
      const int64_t n = n0 + (t >> 1) * g.nnx + (t & 1);
      b[t] = reinterpret_cast<const R2*>(a.b)[n];
      if (!DOWN || PART == PART_RESID) x[t] = reinterpret_cast<const R2*>(a.xin)[n];
    }
  if constexpr (PART == PART_RESID) {
  } else if constexpr (DOWN) {                              // x0 = d0 = (1/theta) D^-1 b
#pragma unroll
    for (int t = 0; t < 4; ++t) d[t] = x[t] = div2(pair(c20 * b[t].x, c20 * b[t].y), dg[t], di[t]);
  } else if constexpr (!NESTED) {
    // the same with the taps of the tables
    const int i0 = max(2 * (ex0 - LO), 0), k0 = max(2 * (ez0 - LO), 0), bx = a.tx.pj[i0] & ~1, bz = a.tz.pj[k0] & ~1;
    for (int i = tid; i < WX * WZ; i += NC) {
      const int jx = bx + i % WX, jz = bz + i / WX;
      R2 v = zero;
      if (jx < a.gc.nnx && jz < a.gc.nnz) v = reinterpret_cast<const R2*>(a.xc)[(int64_t)jz * a.gc.nnx + jx];
      sc[i] = make_double2((double)v.x, (double)v.y);
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (has[t]) {
        const int c0 = (pj[1][t >> 1] - bz) * WX + pj[0][t & 1] - bx;
        double s0 = 0, s1 = 0;
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const double w = pw[1][t >> 1][p] * pw[0][t & 1][q];
            const double2 c = sc[c0 + p * WX + q];
            s0 = fma(w, c.x, s0);
            s1 = fma(w, c.y, s1);
          }
        if (!(fx & (1u << (2 * t)))) x[t].x += (R)s0;
        if (!(fx & (2u << (2 * t)))) x[t].y += (R)s1;
      }
  } else {
    // x + P x_c on the free components: the coarse nodes under the tile in shared memory, as
    // doubles (converted once), the taps of prolong_taps in its order
    const int bx = (ex0 - LO) & ~1, bz = (ez0 - LO) & ~1;
    for (int i = tid; i < WX * WZ; i += NC) {
      const int jx = bx + i % WX, jz = bz + i / WX;
      R2 v = zero;
      if (jx >= 0 && jx < a.gc.nnx && jz >= 0 && jz < a.gc.nnz)
        v = reinterpret_cast<const R2*>(a.xc)[(int64_t)jz * a.gc.nnx + jx];
      sc[i] = make_double2((double)v.x, (double)v.y);
    }
    __syncthreads();
    const double wx0 = (ex & 1) ? -0.125 : 0.375, wx2 = (ex & 1) ? 0.375 : -0.125;
    const double wz0 = (ez & 1) ? -0.125 : 0.375, wz2 = (ez & 1) ? 0.375 : -0.125;
    const double wx[3] = {wx0, 0.75, wx2}, wz[3] = {wz0, 0.75, wz2};
    const int ox = (ex & ~1) - bx, oz = (ez & ~1) - bz, mx = ex - bx, mz = ez - bz;
    double s0[4], s1[4];
    const double2 vc = sc[mz * WX + mx];
    s0[0] = vc.x; s1[0] = vc.y;
    s0[1] = s1[1] = s0[2] = s1[2] = s0[3] = s1[3] = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double2 v = sc[mz * WX + ox + i], w = sc[(oz + i) * WX + mx];
      s0[1] = fma(wx[i], v.x, s0[1]); s1[1] = fma(wx[i], v.y, s1[1]);
      s0[2] = fma(wz[i], w.x, s0[2]); s1[2] = fma(wz[i], w.y, s1[2]);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double2 c = sc[(oz + i) * WX + ox + j];
        const double p = wz[i] * wx[j];
        s0[3] = fma(p, c.x, s0[3]); s1[3] = fma(p, c.y, s1[3]);
      }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (has[t]) {
        if (!(fx & (1u << (2 * t)))) x[t].x += (R)s0[t];
        if (!(fx & (2u << (2 * t)))) x[t].y += (R)s1[t];
      }
  }
  const R sxe = R(2.0 / g.hx), sze = R(2.0 / g.hz), jace = R(g.hx * g.hz / 4.0);
  auto masked = [&](int t) {
    return pair((fx & (1u << (2 * t))) ? R(0) : x[t].x, (fx & (2u << (2 * t))) ? R(0) : x[t].y);
  };
#pragma unroll
  for (int j = J0; j < J1; ++j) {
    // ---- y = K x at the cell's nodes ----
    const int in = j - J0;                                  // cells the halo has shrunk by
    R2 u[9], y[9];
    u[0] = masked(0); u[4] = masked(1); u[7] = masked(2); u[8] = masked(3);
    sx[tid] = u[0]; sx[NC + tid] = u[4]; sx[2 * NC + tid] = u[7]; sx[3 * NC + tid] = u[8];
    __syncthreads();
    if (has[3] && lx >= in && lx <= CX - 2 - in && lz >= in && lz <= CZ - 2 - in) {
      u[1] = sx[tid + 1];
      u[5] = sx[2 * NC + tid + 1];
      u[3] = sx[tid + CX];
      u[6] = sx[NC + tid + CX];
      u[2] = sx[tid + CX + 1];
      k_element(sxe, sze, jace, u, eq, y);
    } else {
#pragma unroll
      for (int k = 0; k < 9; ++k) y[k] = zero;
    }
    se[tid] = y[1]; se[NC + tid] = y[5]; se[2 * NC + tid] = y[3]; se[3 * NC + tid] = y[6]; se[4 * NC + tid] = y[2];
    __syncthreads();
    // ascending element order: lower left, lower, left, own
    const bool hl = lx > 0, hb = lz > 0;
    const R2 p2 = hl && hb ? se[4 * NC + tid - CX - 1] : zero, p3 = hb ? se[2 * NC + tid - CX] : zero,
             p1 = hl ? se[tid - 1] : zero, p6 = hb ? se[3 * NC + tid - CX] : zero, p5 = hl ? se[NC + tid - 1] : zero;
    R2 s[4];
    s[0] = pair(((p2.x + p3.x) + p1.x) + y[0].x, ((p2.y + p3.y) + p1.y) + y[0].y);
    s[1] = pair(p6.x + y[4].x, p6.y + y[4].y);
    s[2] = pair(p5.x + y[7].x, p5.y + y[7].y);
    s[3] = y[8];
#pragma unroll
    for (int t = 0; t < 4; ++t) {                           // eliminated rows act as K_ii u_i
      if (fx & (1u << (2 * t))) s[t].x = dg[t].x * x[t].x;
      if (fx & (2u << (2 * t))) s[t].y = dg[t].y * x[t].y;
    }
    if (DOWN && j == DEG - 1) {                             // residual of the smoothed x
#pragma unroll
      for (int t = 0; t < 4; ++t) s[t] = has[t] ? pair(b[t].x - s[t].x, b[t].y - s[t].y) : zero;
      const int ownx = min(ex0 + TX >= g.nx ? TX + 1 : TX, g.nx + 1 - ex0);
      const int ownz = min(ez0 + TZ >= g.nz ? TZ + 1 : TZ, g.nz + 1 - ez0);
      const bool own = lx >= LO && lx < LO + ownx && lz >= LO && lz < LO + ownz;
      if (own && PART != PART_RESID) {
#pragma unroll
        for (int t = 0; t < 4; ++t)
          if (has[t]) {
            const int64_t n = n0 + (t >> 1) * g.nnx + (t & 1);
            reinterpret_cast<R2*>(a.x)[n] = x[t];
          }
      }
      if constexpr (!NESTED) {
#pragma unroll
        for (int t = 0; t < 4; ++t) sx[t * NC + tid] = s[t];
        __syncthreads();
        for (int i = tid; i < mx * mz; i += NC) {
          const int jx = i % mx, jz = i / mx;
          const int64_t n = (int64_t)(k0 + jz) * a.gc.nnx + j0 + jx;
          const uchar2 f = reinterpret_cast<const uchar2*>(a.fixc)[n];
          const int fx0 = si[0][jx] - 2 * (ex0 - LO), fz0 = si[1][jz] - 2 * (ez0 - LO), nx = sn[0][jx], nz = sn[1][jz];
          double wx[RTAPS];
#pragma unroll
          for (int q = 0; q < RTAPS; ++q) wx[q] = sw[0][jx][q];
          double s0 = 0, s1 = 0;
          for (int p = 0; p < nz; ++p) {
            const double wz = sw[1][jz][p];
            const int row = ((fz0 + p) & 1) * 2 * NC + ((fz0 + p) >> 1) * CX;
#pragma unroll
            for (int q = 0; q < RTAPS; ++q)
              if (q < nx) {
                const double w = wz * wx[q];
                const R2 v = sx[row + ((fx0 + q) & 1) * NC + ((fx0 + q) >> 1)];
                s0 = fma(w, (double)v.x, s0);
                s1 = fma(w, (double)v.y, s1);
              }
          }
          reinterpret_cast<R2*>(a.bc)[n] = pair(f.x ? R(0) : (R)s0, f.y ? R(0) : (R)s1);
        }
      } else {
        // coarse node (I, J) sits on the corner of fine cell (I, J); the four parities have 9, 15,
        // 15 and 25 taps, so each warp takes nodes of one parity
#pragma unroll
        for (int t = 0; t < 4; ++t) sx[t * NC + tid] = s[t];
        __syncthreads();
        const int warp = tid >> 5, px = warp & 1, pz = (warp >> 1) & 1;
        const int mx = (ownx - px + 1) / 2, mz = (ownz - pz + 1) / 2;
        for (int i = (warp >> 2) * 32 + (tid & 31); i < mx * mz; i += NC / 4) {
          const int jx = 2 * (i % mx) + px, jz = 2 * (i / mx) + pz;
          const int c = (jz + LO) * CX + jx + LO;
          const int64_t n = (int64_t)(ez0 + jz) * a.gc.nnx + ex0 + jx;
          const uchar2 f = reinterpret_cast<const uchar2*>(a.fixc)[n];
          double s0, s1;
          if (px) {
            if (pz) restrict_taps<1, 1, CX, NC>(sx, c, &s0, &s1);
            else restrict_taps<1, 0, CX, NC>(sx, c, &s0, &s1);
          } else {
            if (pz) restrict_taps<0, 1, CX, NC>(sx, c, &s0, &s1);
            else restrict_taps<0, 0, CX, NC>(sx, c, &s0, &s1);
          }
          reinterpret_cast<R2*>(a.bc)[n] = pair(f.x ? R(0) : (R)s0, f.y ? R(0) : (R)s1);
        }
      }
    } else {                                                // d = c1 d + c2 D^-1 (b - y); x += d
      const bool first = !DOWN && j == 0;                   // the restart step reads no old direction
      const R c2 = (DOWN || j > 0) ? c21 : c20;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        R2 dn = div2(pair(c2 * (b[t].x - s[t].x), c2 * (b[t].y - s[t].y)), dg[t], di[t]);
        if (!first && c1s != 0.0) {
          dn.x += R(c1s) * d[t].x;
          dn.y += R(c1s) * d[t].y;
        }
        d[t] = dn;
        x[t] = pair(x[t].x + dn.x, x[t].y + dn.y);
      }
    }
  }
  if constexpr (!RESTRICT) {
    const int ownx = ex0 + TX >= g.nx ? TX + 1 : TX, ownz = ez0 + TZ >= g.nz ? TZ + 1 : TZ;
    double v = 0;
    if (lx >= LO && lx < LO + ownx && lz >= LO && lz < LO + ownz) {
#pragma unroll
      for (int t = 0; t < 4; ++t)
        if (has[t]) {
          reinterpret_cast<R2*>(a.x)[n0 + (t >> 1) * g.nnx + (t & 1)] = x[t];
          if (!DOWN && a.bx.part) v += (double)b[t].x * (double)x[t].x + (double)b[t].y * (double)x[t].y;
        }
    }
    if (!DOWN && a.bx.part) grid_sum_parity(v, a.bx, blockIdx.y * gridDim.x + blockIdx.x, gridDim.x * gridDim.y);
  }
}

template <typename R, int DEG, bool DOWN, bool NESTED, int PART = PART_ALL>
void launch(const MgArgs<R>& a, bool planes, cudaStream_t s) {
  constexpr int T = owned_cells(DOWN && PART != PART_SMOOTH, PART == PART_ALL ? DEG : 1, NESTED);
  const dim3 grid((a.g.nx + T - 1) / T, (a.g.nz + T - 1) / T);
  if (planes) pdl_launch(k_mg_level<R, DEG, DOWN, true, NESTED, PART>, grid, CELLS * CELLS, 0, s, a);
  else pdl_launch(k_mg_level<R, DEG, DOWN, false, NESTED, PART>, grid, CELLS * CELLS, 0, s, a);
}

// Downward with two smoothing steps on large levels: the smoothing and the residual with its restriction as
// two launches.  Together they repeat 256 / 100 of the element products (a tile owns 10 x 10 cells), apart
// 256 / 196 and 256 / 144; in exchange x is read back and there is one more launch.  FP32 V-cycle with every
// level above the line split, against none: 512^2 165.5 -> 158 us, 384^2 111.5 -> 107; splitting 256^2 as
// well changes nothing there (77.5, 77.3), 128^2 and below lose (77.5 -> 78.9 with all of them).
constexpr int64_t SPLIT_ELEMENTS = 1 << 16;
template <typename R, bool NESTED>
void down2(const MgArgs<R>& a, bool planes, cudaStream_t s) {
  if ((int64_t)a.g.nx * a.g.nz <= SPLIT_ELEMENTS) {
    launch<R, MG_MAXDEG, true, NESTED>(a, planes, s);
    return;
  }
  launch<R, MG_MAXDEG, true, NESTED, PART_SMOOTH>(a, planes, s);
  MgArgs<R> r = a;
  r.xin = a.x;
  launch<R, MG_MAXDEG, true, NESTED, PART_RESID>(r, planes, s);
}

template <typename R, bool DOWN>
void pick(const MgArgs<R>& a, int deg, bool planes, cudaStream_t s) {
  const bool nested = a.g.nx == 2 * a.gc.nx && a.g.nz == 2 * a.gc.nz;
  if (deg <= 1) {
    if (nested) launch<R, 1, DOWN, true>(a, planes, s);
    else launch<R, 1, DOWN, false>(a, planes, s);
  } else {
    if constexpr (DOWN) {
      if (nested) down2<R, true>(a, planes, s);
      else down2<R, false>(a, planes, s);
    } else {
      if (nested) launch<R, MG_MAXDEG, false, true>(a, planes, s);
      else launch<R, MG_MAXDEG, false, false>(a, planes, s);
    }
  }
}

}  // namespace

int mg_ensure_tables() { return ensure_cell_tables(); }

template <typename R> void mg_down(const MgArgs<R>& a, int deg, bool planes, cudaStream_t s) {
  pick<R, true>(a, deg, planes, s);
}
template <typename R> void mg_up(const MgArgs<R>& a, int deg, bool planes, cudaStream_t s) {
  pick<R, false>(a, deg, planes, s);
}

template void mg_down<float>(const MgArgs<float>&, int, bool, cudaStream_t);
template void mg_down<double>(const MgArgs<double>&, int, bool, cudaStream_t);
template void mg_up<float>(const MgArgs<float>&, int, bool, cudaStream_t);
template void mg_up<double>(const MgArgs<double>&, int, bool, cudaStream_t);

}  // namespace mw
