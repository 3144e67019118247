// Particle-in-cell kernels for the Cartesian box (sm_100a).
//
// Reference: pic_functions.py (locate :108-137, element projection :603-650, nodal projections
// :659-1053, least squares :1061-1285, population control :1621-1812).  Interpolation and
// advection are in advect.cu.
//
// Layout: particles are SoA (x, z, r, t: f64; iel: i32; active: u8), one thread per particle where
// particles are independent, lanes or blocks per piece of the bins where they are summed; grid-stride loops.  Projections are atomic-free and deterministic: particles are binned by element (counting sort, each bin sorted by particle
// index), so every element and node sums its particles in particle-index order -- the order of
// the reference's sequential loops.  This file is compiled with -fmad=false so the basis and
// weight arithmetic rounds exactly as the reference's unfused double-precision code.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "pic_common.cuh"

namespace mw {

int num_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

bool pdl_enabled() {
  static const bool on = [] {
    const char* e = getenv("MW_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

int grid_for(int64_t n, int threads, int waves) {
  int64_t need = (n + threads - 1) / threads;
  int64_t cap = (int64_t)num_sms() * waves;
  if (need < 1) need = 1;
  return (int)(need < cap ? need : cap);
}


// ------------------------------------------------------------------------------------------
// Four quotients a particle are most of the arithmetic; from the reciprocals they take five
// multiply-adds each (4.2 M particles: 52 -> 37 us; 37 bytes a particle floor it at 24).
__global__ void k_locate(mw_box b, int64_t n, const uint8_t* __restrict__ active,
                         const double* __restrict__ x, const double* __restrict__ z,
                         double* __restrict__ r, double* __restrict__ t, int32_t* __restrict__ iel,
                         int32_t* err) {
  const int64_t nel = (int64_t)b.nelx * b.nelz;
  const double ihx = 1.0 / b.hx, ihz = 1.0 / b.hz;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint8_t act = active[i];
    const double xi = x[i], zi = z[i];
    if (!act) { r[i] = 0.0; t[i] = 0.0; iel[i] = 0; continue; }
    // the element: pic_functions.py:29-31; int() truncates toward zero, and a quotient that does not fit an int
    // is out of range (the reference would index out of bounds there)
    const double qx = quotient_exact(xi, b.hx, ihx), qz = quotient_exact(zi, b.hz, ihz);
    bool ok = qx > -2147483648.0 && qx < 2147483647.0 && qz > -2147483648.0 && qz < 2147483647.0;
    int ex = 0, ez = 0;
    int64_t e = 0;
    if (ok) {
      ex = (int)qx;
      ez = (int)qz;
      e = (int64_t)b.nelx * ez + ex;
      ok = e >= 0 && e < nel;
      if (ok && (ex < 0 || ex >= b.nelx)) {              // the reference's wrap into the next row
        ex = (int)(e % b.nelx);
        ez = (int)(e / b.nelx);
      }
    }
    if (!ok) {
      set_flag(err, MW_FLAG_ELEMENT_RANGE);
      r[i] = 0.0; t[i] = 0.0; iel[i] = -1;
      continue;
    }
    const double rr = (quotient_exact(xi - xv0(b, ex), b.hx, ihx) - 0.5) * 2;
    const double tt = (quotient_exact(zi - zv0(b, ez), b.hz, ihz) - 0.5) * 2;
    if (rr < -1.0 || rr > 1.0) set_flag(err, MW_FLAG_R_OUT_OF_BOUNDS);
    if (tt < -1.0 || tt > 1.0) set_flag(err, MW_FLAG_T_OUT_OF_BOUNDS);
    r[i] = rr; t[i] = tt; iel[i] = (int32_t)e;
  }
}


// ------------------------------------------------------------------------------------------
// Binning: counts -> exclusive scan -> scatter -> per-bin sort by particle index.
//
// Particles of an element mostly lie next to one another in memory, so the atomics go by runs: a lane
// takes four particles, and lanes whose four lie in one element join into runs of equal elements with one
// atomic each.  Any order gives the same bins (the last pass sorts them).
//
// The run of this lane's key: `head`, its first lane, and `len`.
MW_D void warp_run(int key, int* head, int* len) {
  const int lane = threadIdx.x & 31;
  const int prev = __shfl_up_sync(0xffffffffu, key, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || prev != key);
  const unsigned upto = heads & (0xffffffffu >> (31 - lane));
  *head = 31 - __clz(upto);
  const unsigned after = lane == 31 ? 0u : heads & (0xffffffffu << (lane + 1));
  *len = (after ? __ffs(after) - 1 : 32) - *head;
}

// the elements of particles 4 q .. 4 q + 3 (-1: inactive, out of range or past the end)
template <bool VEC>
MW_D void four_elements(int64_t q, int64_t n, int32_t nel, const uint8_t* __restrict__ active,
                        const int32_t* __restrict__ iel, int32_t* err, int (&e)[4]) {
  if (VEC && 4 * q + 3 < n) {
    const int4 v = reinterpret_cast<const int4*>(iel)[q];
    const uchar4 a = reinterpret_cast<const uchar4*>(active)[q];
    e[0] = a.x ? v.x : -1; e[1] = a.y ? v.y : -1; e[2] = a.z ? v.z : -1; e[3] = a.w ? v.w : -1;
    // (an active particle with a negative element is out of range too; told apart below)
    const bool bad = (a.x && (v.x < 0 || v.x >= nel)) || (a.y && (v.y < 0 || v.y >= nel)) ||
                     (a.z && (v.z < 0 || v.z >= nel)) || (a.w && (v.w < 0 || v.w >= nel));
    if (bad) set_flag(err, MW_FLAG_ELEMENT_RANGE);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t i = 4 * q + k;
      e[k] = -1;
      if (i < n && active[i]) {
        e[k] = iel[i];
        if (e[k] < 0 || e[k] >= nel) set_flag(err, MW_FLAG_ELEMENT_RANGE);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (e[k] < 0 || e[k] >= nel) e[k] = -1;
}

template <bool VEC>
__global__ void __launch_bounds__(256) k_count(int64_t n, int32_t nel, const uint8_t* __restrict__ active,
                                               const int32_t* __restrict__ iel, int32_t* __restrict__ counts,
                                               int32_t* err) {
  const int64_t nq = (n + 3) / 4, step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < nq; base += step) {
    int e[4];
    four_elements<VEC>(base + threadIdx.x, n, nel, active, iel, err, e);
    const bool one = e[0] == e[1] && e[1] == e[2] && e[2] == e[3];
    int head, len;
    warp_run(one ? e[0] : -2 - (int)(threadIdx.x & 31), &head, &len);
    if (one) {
      if (e[0] >= 0 && head == (int)(threadIdx.x & 31)) atomicAdd(counts + e[0], 4 * len);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (e[k] >= 0) atomicAdd(counts + e[k], 1);
    }
  }
}

// Sums of 1024 counts a block, and from them the exclusive prefix sum: each block adds the sums of the
// blocks before it (at most 1024) to its own scan.  offsets[n] is the total; cursor a copy of offsets.
__global__ void __launch_bounds__(1024) k_block_sums(const int32_t* __restrict__ in, int32_t* __restrict__ sums,
                                                     int64_t n) {
  __shared__ int32_t ws[32];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int32_t v = i < n ? in[i] : 0;
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = __reduce_add_sync(0xffffffffu, ws[threadIdx.x]);
    if (threadIdx.x == 0) sums[blockIdx.x] = v;
  }
}

__global__ void __launch_bounds__(1024) k_scan_offsets(const int32_t* __restrict__ in,
                                                       const int32_t* __restrict__ sums, int32_t* __restrict__ offsets,
                                                       int32_t* __restrict__ cursor, int64_t n) {
  __shared__ int32_t ws[32], wb[32];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int32_t v = i < n ? in[i] : 0;
  int32_t before = threadIdx.x < blockIdx.x ? sums[threadIdx.x] : 0;
  before = __reduce_add_sync(0xffffffffu, before);
  int32_t incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) ws[wid] = incl;
  if (lane == 0) wb[wid] = before;
  __syncthreads();
  if (wid == 0) {
    int32_t s = ws[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    ws[lane] = s;
    const int32_t total = __reduce_add_sync(0xffffffffu, wb[lane]);
    if (lane == 0) wb[0] = total;
  }
  __syncthreads();
  const int32_t off = wb[0] + (wid > 0 ? ws[wid - 1] : 0) + incl - v;
  if (i < n) {
    offsets[i] = off;
    cursor[i] = off;
    if (i == n - 1) offsets[n] = off + v;
  }
}

// Block-level exclusive scan of int32 (1024 items per block), writing block totals.
__global__ void k_scan_block(const int32_t* __restrict__ in, int32_t* __restrict__ out, int32_t* __restrict__ block_sums,
                             int64_t n) {
  __shared__ int32_t warp_sums[32];
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int32_t v = i < n ? in[i] : 0;
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_sums[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    int32_t s = lane < nw ? warp_sums[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      int32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < nw) warp_sums[lane] = s;
  }
  __syncthreads();
  int32_t base = wid > 0 ? warp_sums[wid - 1] : 0;
  if (i < n) out[i] = base + incl - v;
  if (threadIdx.x == blockDim.x - 1 && block_sums) block_sums[blockIdx.x] = base + incl;
}

__global__ void k_scan_add(int32_t* __restrict__ out, const int32_t* __restrict__ block_prefix, int64_t n) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] += block_prefix[blockIdx.x];
}

template <bool VEC>
__global__ void __launch_bounds__(256) k_scatter(int64_t n, int32_t nel, const uint8_t* __restrict__ active,
                                                 const int32_t* __restrict__ iel, int32_t* __restrict__ cursor,
                                                 int32_t* __restrict__ order) {
  const int64_t nq = (n + 3) / 4, step = (int64_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < nq; base += step) {
    const int64_t q = base + threadIdx.x;
    int e[4];
    four_elements<VEC>(q, n, nel, active, iel, nullptr, e);
    const bool one = e[0] == e[1] && e[1] == e[2] && e[2] == e[3];
    int head, len, at = 0;
    warp_run(one ? e[0] : -2 - lane, &head, &len);
    if (one && e[0] >= 0 && head == lane) at = atomicAdd(cursor + e[0], 4 * len);
    at = __shfl_sync(0xffffffffu, at, head) + 4 * (lane - head);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (e[k] < 0) continue;
      order[one ? at + k : atomicAdd(cursor + e[k], 1)] = (int32_t)(4 * q + k);
    }
  }
}

// a[0 .. m) ascending by a warp: Batcher's odd-even merge exchange (The Art of Computer Programming 5.2.2,
// Algorithm M) for any m, unless it is in order.
__device__ __noinline__ void sort_by_warp(int32_t* a, int m) {
  const int lane = threadIdx.x & 31;
  bool down = false;
  for (int j = lane + 1; j < m; j += 32) down |= a[j] < a[j - 1];
  if (!__any_sync(0xffffffffu, down)) return;
  for (int lp = 0; (1 << lp) < m; ++lp)
    for (int lk = lp; lk >= 0; --lk) {
      const int k = 1 << lk, x0 = lk == lp ? 0 : k;
      for (int q = lane;; q += 32) {
        const int x = x0 + ((q >> lk) << (lk + 1)) + (q & (k - 1)), y = x + k;
        if (y >= m) break;
        if (x >> (lp + 1) != y >> (lp + 1)) continue;
        const int u = a[x], v = a[y];
        if (u > v) {
          a[x] = v;
          a[y] = u;
        }
      }
      __syncwarp();
    }
}

// Sort each bin by particle index: 16 lanes an element, each placing its particles by the number of smaller
// indices in the bin (bins hold about 9-25 particles); bins longer than SORT_MAX one after the other by merge
// exchange.  A thread an element, sorting by insertion in global memory, read each cache line 16 times.  The
// whole binning of 4.2 M particles: 94 -> 41 us, of 33000: 39 -> 14 (nine launches and two clears before, five
// and one now); of 1.6 M in bins of 100, in order and shuffled, 417 and 218 -> 56 and 108 (insertion by one
// lane of a group: 251 and 272).
constexpr int GROUP = 16, SORT_MAX = 64;
__global__ void __launch_bounds__(256) k_sort_bins(int32_t nel, const int32_t* __restrict__ offsets,
                                                   int32_t* __restrict__ order) {
  __shared__ int32_t sm[256 / GROUP][SORT_MAX];
  const int lane = threadIdx.x % GROUP, grp = threadIdx.x / GROUP;
  for (int64_t base = blockIdx.x * (int64_t)(256 / GROUP); base < nel; base += (int64_t)gridDim.x * (256 / GROUP)) {
    const int64_t e = base + grp;
    const int b0 = e < nel ? offsets[e] : 0, m = e < nel ? offsets[e + 1] - b0 : 0;
    const bool fits = m <= SORT_MAX;
    int v0 = 0x7fffffff;
    if (fits)
      for (int j = lane; j < m; j += GROUP) {
        const int v = order[b0 + j];
        sm[grp][j] = v;
        if (j == lane) v0 = v;
      }
    // bins of up to 16 that the scatter filled in order stay as they are
    const int prev = __shfl_up_sync(0xffffffffu, v0, 1);
    const unsigned down = __ballot_sync(0xffffffffu, lane > 0 && lane < m && v0 < prev);
    const bool sorted = m <= GROUP && !((down >> (threadIdx.x & 16)) & 0xffffu);
    __syncwarp();
    if (fits && !sorted) {
      for (int j = lane; j < m; j += GROUP) {
        const int v = sm[grp][j];
        int rank = 0;
        for (int k = 0; k < m; ++k) rank += sm[grp][k] < v ? 1 : 0;
        if (rank != j) order[b0 + rank] = v;
      }
    }
    for (unsigned rest = __ballot_sync(0xffffffffu, !fits && lane == 0); rest; rest &= rest - 1) {
      const int src = __ffs(rest) - 1;
      sort_by_warp(order + __shfl_sync(0xffffffffu, b0, src), __shfl_sync(0xffffffffu, m, src));
    }
    __syncwarp();
  }
}

__global__ void k_total(const int32_t* counts, int32_t* offsets, int64_t n) {
  if (threadIdx.x == 0 && blockIdx.x == 0) offsets[n] = n > 0 ? offsets[n - 1] + counts[n - 1] : 0;
}

// ------------------------------------------------------------------------------------------
MW_D double avg_transform(int averaging, double v) {
  if (averaging == MW_AVG_GEOMETRIC) return log10(v);
  if (averaging == MW_AVG_HARMONIC) return 1.0 / v;
  return v;
}

// largest value over the warp
MW_D int warp_max(int v) { return __reduce_max_sync(0xffffffffu, v); }

// pic_functions.py:603-650 over the sorted bins.  A block takes as many elements as hold PART particles on
// average (a power of two, at most PROJ_ELEMENTS), whose particles are one piece of `order`: all of its
// threads load and transform them, PART at a time, and then a thread per element and field adds its own in
// particle order, so the sums are the sequential loop's whatever the bins' sizes.  Geometric means, in us
// (16 lanes an element; a thread an element): 512^2 elements of 4, 9, 16 particles 15, 23, 31 (33, 35, 41; 12, 17,
// 45), 256^2 of 9, 25, 64 9, 15, 31 (13, 19, 33; 10, 16, 57), 128^2 of 100 17 (17; 36).  A thread an element keeps a
// lead on meshes of 512^2 with few particles an element in memory order, and loses it in any other order.
constexpr int PART = 1024, PROJ_ELEMENTS = 64;
__global__ void __launch_bounds__(256) k_project_elements(int32_t nel, const int32_t* __restrict__ offsets,
                                                          const int32_t* __restrict__ order,
                                                          const double* __restrict__ rho,
                                                          const double* __restrict__ eta, int averaging,
                                                          double* __restrict__ rho_e, double* __restrict__ eta_e,
                                                          int32_t* err) {
  static_assert(2 * PROJ_ELEMENTS <= 256, "a thread per element and field");
  constexpr int PAD = 16;                                    // a gap every 16 values: bins of 16 on all banks
  __shared__ double sv[2][PART + PART / PAD];
  __shared__ int so[PROJ_ELEMENTS + 1];
  const int64_t total = offsets[nel];
  int shift = 6;                                             // elements of a block: 1 << shift
  while (shift > 0 && (total << shift) > (int64_t)PART * nel) --shift;
  const int pe = 1 << shift, tid = threadIdx.x, le = tid & (pe - 1), which = tid >> shift;
  for (int64_t e0 = blockIdx.x * (int64_t)pe; e0 < nel; e0 += (int64_t)gridDim.x * pe) {
    if (tid <= pe) so[tid] = offsets[min(e0 + tid, (int64_t)nel)];
    __syncthreads();
    const int b0 = so[le], b1 = so[le + 1], end = so[pe];
    double sum = 0.0;
    for (int c0 = so[0]; c0 < end; c0 += PART) {
      for (int j = c0 + tid; j < min(c0 + PART, end); j += 256) {
        const int p = order[j], i = j - c0;
        sv[0][i + i / PAD] = rho[p];
        sv[1][i + i / PAD] = avg_transform(averaging, eta[p]);
      }
      __syncthreads();
      if (which < 2)
        for (int i = max(b0, c0) - c0; i < min(b1, c0 + PART) - c0; ++i) sum = sum + sv[which][i + i / PAD];
      __syncthreads();
    }
    const int64_t e = e0 + le;
    if (e < nel && which < 2) {
      const double c = (double)(b1 - b0);
      if (which == 0) {
        if (b1 == b0) set_flag(err, MW_FLAG_EMPTY_ELEMENT);
        rho_e[e] = sum / c;
      } else if (averaging == MW_AVG_GEOMETRIC) {
        eta_e[e] = pow(10.0, sum / c);
      } else if (averaging == MW_AVG_HARMONIC) {
        eta_e[e] = c / sum;
      } else {
        eta_e[e] = sum / c;
      }
    }
    __syncthreads();                                         // the offsets are read
  }
}

// Corner-node projection (pic_functions.py:659-1053): node (2i, 2j) sums the particles of its
// (up to) four incident elements, merged in particle-index order.
struct ProjFields {
  const double* phi[MW_MAX_FIELDS];
  double* out[MW_MAX_FIELDS];
  int averaging[MW_MAX_FIELDS];
  int n;
};

MW_D void corner_weight(int flavour, int k, double r, double t, bool* use, double* w) {
  if (flavour == 1) { *use = true; *w = 1.0; return; }
  if (flavour == 2) {
    *use = true;
    if (k == 0) *w = 0.25 * (1 - r) * (1 - t);
    else if (k == 1) *w = 0.25 * (1 + r) * (1 - t);
    else if (k == 2) *w = 0.25 * (1 + r) * (1 + t);
    else *w = 0.25 * (1 - r) * (1 + t);
    return;
  }
  bool u;
  if (k == 0) u = (r <= 0 && t <= 0);
  else if (k == 1) u = (r >= 0 && t <= 0);
  else if (k == 2) u = (r >= 0 && t >= 0);
  else u = (r <= 0 && t >= 0);
  *use = u;
  if (flavour == 3) { *w = 1.0; return; }
  if (k == 0) *w = -r * -t;
  else if (k == 1) *w = (1 - r) * -t;
  else if (k == 2) *w = (1 - r) * (1 - t);
  else *w = -r * (1 - t);
}

__global__ void k_project_corners(mw_box b, int flavour, const int32_t* __restrict__ offsets,
                                  const int32_t* __restrict__ order, const double* __restrict__ r,
                                  const double* __restrict__ t, ProjFields pf) {
  const int ncx = b.nelx + 1, ncz = b.nelz + 1;
  const int nnx = 2 * b.nelx + 1;
  const int64_t ncorner = (int64_t)ncx * ncz;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < ncorner; c += (int64_t)gridDim.x * blockDim.x) {
    int i = (int)(c % ncx), j = (int)(c / ncx);
    // incident elements and this node's local corner index in each
    int pos[4], end[4], kk[4];
    int ne = 0;
    const int ex[4] = {i, i - 1, i - 1, i};
    const int ez[4] = {j, j, j - 1, j - 1};
    for (int k = 0; k < 4; ++k) {
      if (ex[k] < 0 || ex[k] >= b.nelx || ez[k] < 0 || ez[k] >= b.nelz) continue;
      int e = ez[k] * b.nelx + ex[k];
      pos[ne] = offsets[e]; end[ne] = offsets[e + 1]; kk[ne] = k; ++ne;
    }
    double acc[MW_MAX_FIELDS];
    double cnt = 0.0;
    for (int f = 0; f < pf.n; ++f) acc[f] = 0.0;
    while (true) {
      int best = -1, bp = 0x7fffffff;
      for (int s = 0; s < ne; ++s)
        if (pos[s] < end[s]) { int p = order[pos[s]]; if (p < bp) { bp = p; best = s; } }
      if (best < 0) break;
      ++pos[best];
      bool use; double w;
      corner_weight(flavour, kk[best], r[bp], t[bp], &use, &w);
      if (!use) continue;
      if (flavour == 1 || flavour == 3) cnt = cnt + 1.0;
      else cnt = cnt + 1 * w;
      for (int f = 0; f < pf.n; ++f) {
        double v = avg_transform(pf.averaging[f], pf.phi[f][bp]);
        acc[f] = (flavour == 1 || flavour == 3) ? acc[f] + v : acc[f] + v * w;
      }
    }
    int64_t node = (int64_t)(2 * j) * nnx + 2 * i;
    for (int f = 0; f < pf.n; ++f) {
      double v;
      if (pf.averaging[f] == MW_AVG_GEOMETRIC) v = pow(10.0, acc[f] / cnt);
      else if (pf.averaging[f] == MW_AVG_HARMONIC) v = cnt / acc[f];
      else v = acc[f] / cnt;
      pf.out[f][node] = v;
    }
  }
}

// Faster form of the same projection: each element sums its particles (in particle-index order)
// per corner into partials (nel x 4 x (nfield+1) doubles), then each corner node adds the partials
// of its incident elements in ascending element order and applies the averaging.  The sums agree
// with the reference's particle-ordered sums to rounding (different association).
// NF: capacity for the fields (pf.n <= NF).  16 lanes an element: each loads one particle of 16 (its
// weights on the four corners, its transformed fields), then each keeps one (corner, field) sum and
// walks the 16 in particle order.  A thread an element with all of its sums ran at 12 % of the warps,
// one gather after the other.  Two fields of 262144 elements, nodes filled in: 131 -> 88 us.
template <int NF>
__global__ void __launch_bounds__(256) k_project_elem_partials(mw_box b, int flavour,
                                                               const int32_t* __restrict__ offsets,
                                                               const int32_t* __restrict__ order,
                                                               const double* __restrict__ r,
                                                               const double* __restrict__ t, ProjFields pf,
                                                               double* __restrict__ part) {
  constexpr int NR = (4 * (NF + 1) + GROUP - 1) / GROUP;     // sums a lane keeps
  // a particle's weights and values side by side (the lanes of a group read one particle's at a time),
  // groups padded apart so that the two of a warp use different banks
  constexpr int SW = GROUP * 4 + 4, SV = GROUP * NF + 4;
  __shared__ double sw[256 / GROUP][SW], sv[256 / GROUP][SV];
  __shared__ uint8_t suse[256];
  const int64_t nel = (int64_t)b.nelx * b.nelz;
  const int nf1 = pf.n + 1, nsum = 4 * nf1;
  const int lane = threadIdx.x % GROUP, grp = threadIdx.x / GROUP, g0 = threadIdx.x - lane;
  const bool plain = flavour == 1 || flavour == 3, all = flavour <= 2;
  for (int64_t base = blockIdx.x * (int64_t)(256 / GROUP); base < nel; base += (int64_t)gridDim.x * (256 / GROUP)) {
    const int64_t e = base + threadIdx.x / GROUP;
    const int b0 = e < nel ? offsets[e] : 0, m = e < nel ? offsets[e + 1] - b0 : 0;
    const int rounds = (warp_max(m) + GROUP - 1) / GROUP;
    double acc[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) acc[i] = 0.0;
    for (int c = 0; c < rounds; ++c) {
      const int j = c * GROUP + lane;
      if (j < m) {
        const int p = order[b0 + j];
        const double rp = r[p], tp = t[p];
        int mask = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          bool use; double w;
          corner_weight(flavour, k, rp, tp, &use, &w);
          sw[grp][lane * 4 + k] = w;
          if (use) mask |= 1 << k;
        }
        suse[threadIdx.x] = (uint8_t)mask;
#pragma unroll
        for (int f = 0; f < NF; ++f)
          if (f < pf.n) sv[grp][lane * NF + f] = avg_transform(pf.averaging[f], pf.phi[f][p]);
      }
      __syncwarp();
      const int k1 = min(GROUP, m - c * GROUP);
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const int q = i * GROUP + lane;
        if (q < nsum) {
          const int k = q / nf1, f = q - k * nf1;
          const double* wk = sw[grp] + k;
          const double* vf = sv[grp] + (f < pf.n ? f : 0);
          const bool count = f == pf.n;
          for (int s = 0; s < k1; ++s) {
            if (!all && !((suse[g0 + s] >> k) & 1)) continue;
            const double v = count ? 1.0 : vf[s * NF];
            acc[i] = plain ? acc[i] + v : acc[i] + v * wk[s * 4];
          }
        }
      }
      __syncwarp();
    }
    if (e < nel) {
      double* o = part + e * nsum;
#pragma unroll
      for (int i = 0; i < NR; ++i)
        if (i * GROUP + lane < nsum) o[i * GROUP + lane] = acc[i];
    }
  }
}

// The corner values (partials of the incident elements in ascending order, the averaging) of a tile and
// from them its edge and centre nodes (pic_functions.py:801-809), in one launch: the tile recomputes the
// corners on its right and top for itself.
constexpr int PFX = 32, PFZ = 8;
template <int NF>
__global__ void __launch_bounds__(PFX * PFZ) k_project_finish(mw_box b, ProjFields pf,
                                                              const double* __restrict__ part) {
  __shared__ double sc[NF][(PFX + 1) * (PFZ + 1)];
  const int ntx = (b.nelx + PFX - 1) / PFX;                  // (tiles in x alone: a mesh may be taller than the grid's y)
  const int i0 = (int)(blockIdx.x % ntx) * PFX, j0 = (int)(blockIdx.x / ntx) * PFZ;
  const int nf1 = pf.n + 1;
  const int64_t nnx = 2 * b.nelx + 1;
  for (int c = threadIdx.x; c < (PFX + 1) * (PFZ + 1); c += PFX * PFZ) {
    const int i = i0 + c % (PFX + 1), j = j0 + c / (PFX + 1);
    if (i > b.nelx || j > b.nelz) continue;
    double acc[NF + 1];
#pragma unroll
    for (int f = 0; f <= NF; ++f) acc[f] = 0.0;
    // ascending element order: (j-1,i-1) corner 2, (j-1,i) corner 3, (j,i-1) corner 1, (j,i) corner 0
    for (int s2 = 0; s2 < 4; ++s2) {
      const int ex = (s2 & 1) ? i : i - 1, ez = (s2 & 2) ? j : j - 1;
      if (ex < 0 || ex >= b.nelx || ez < 0 || ez >= b.nelz) continue;
      const int k = s2 == 0 ? 2 : (s2 == 1 ? 3 : (s2 == 2 ? 1 : 0));
      const double* o = part + ((int64_t)ez * b.nelx + ex) * 4 * nf1 + k * nf1;
#pragma unroll
      for (int f = 0; f < NF; ++f)
        if (f < pf.n) acc[f] += o[f];
      acc[NF] += o[pf.n];
    }
    const double cnt = acc[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f)
      if (f < pf.n) {
        double v;
        if (pf.averaging[f] == MW_AVG_GEOMETRIC) v = pow(10.0, acc[f] / cnt);
        else if (pf.averaging[f] == MW_AVG_HARMONIC) v = cnt / acc[f];
        else v = acc[f] / cnt;
        sc[f][c] = v;
      }
  }
  __syncthreads();
  const int li = threadIdx.x % PFX, lj = threadIdx.x / PFX;
  // the corners past the last full tile column and row belong to the last tile
  const int wi = i0 + PFX >= b.nelx ? b.nelx + 1 - i0 : PFX, wj = j0 + PFZ >= b.nelz ? b.nelz + 1 - j0 : PFZ;
  for (int jj = lj; jj < wj; jj += PFZ)
    for (int ii = li; ii < wi; ii += PFX) {
      const int i = i0 + ii, j = j0 + jj, c = jj * (PFX + 1) + ii;
      const bool rx = i < b.nelx, rz = j < b.nelz;
      const int64_t n = (int64_t)(2 * j) * nnx + 2 * i;
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        if (f >= pf.n) continue;
        double* o = pf.out[f] + n;
        const double* q = sc[f] + c;
        o[0] = q[0];
        if (rx) o[1] = 0.50 * (q[0] + q[1]);
        if (rz) o[nnx] = 0.50 * (q[0] + q[PFX + 1]);
        if (rx && rz) o[nnx + 1] = 0.25 * (((q[0] + q[1]) + q[PFX + 2]) + q[PFX + 1]);
      }
    }
}

// Edge and centre nodes from the corners: pic_functions.py:801-809.
__global__ void k_fill_q2(mw_box b, ProjFields pf) {
  const int nnx = 2 * b.nelx + 1, nnz = 2 * b.nelz + 1;
  const int64_t nn = (int64_t)nnx * nnz;
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < nn; n += (int64_t)gridDim.x * blockDim.x) {
    int ix = (int)(n % nnx), iz = (int)(n / nnx);
    bool ox = ix & 1, oz = iz & 1;
    if (!ox && !oz) continue;
    for (int f = 0; f < pf.n; ++f) {
      double* o = pf.out[f];
      double v;
      if (ox && !oz) v = 0.50 * (o[n - 1] + o[n + 1]);
      else if (!ox && oz) v = 0.50 * (o[n - nnx] + o[n + nnx]);
      else v = 0.25 * (((o[n - nnx - 1] + o[n - nnx + 1]) + o[n + nnx + 1]) + o[n + nnx - 1]);
      o[n] = v;
    }
  }
}

// ------------------------------------------------------------------------------------------
// phiq[e, q] = sum_k N[q, k] phi[node_k(e)]: project_nodal_field_onto_qpoints.py:12-62.
__global__ void k_nodal_to_q(mw_box b, int space, const double* __restrict__ Ntab, const double* __restrict__ phi,
                             double* __restrict__ phiq) {
  __shared__ double Ns[81];
  int m = (space == MW_SPACE_Q2) ? 9 : 4;
  for (int i = threadIdx.x; i < 9 * m; i += blockDim.x) Ns[i] = Ntab[i];
  __syncthreads();
  const int64_t nq = (int64_t)b.nelx * b.nelz * 9;
  const int nnx = 2 * b.nelx + 1;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < nq; g += (int64_t)gridDim.x * blockDim.x) {
    int64_t e = g / 9;
    int q = (int)(g % 9);
    int ex = (int)(e % b.nelx), ez = (int)(e / b.nelx);
    double acc;
    if (space == MW_SPACE_Q2) {
      acc = Ns[q * 9] * phi[q2_node(ex, ez, 0, nnx)];
      for (int k = 1; k < 9; ++k) acc = acc + Ns[q * 9 + k] * phi[q2_node(ex, ez, k, nnx)];
    } else if (space == MW_SPACE_Q1_ON_V) {
      acc = Ns[q * 4] * phi[q2_node(ex, ez, 0, nnx)];
      for (int k = 1; k < 4; ++k) acc = acc + Ns[q * 4 + k] * phi[q2_node(ex, ez, k, nnx)];
    } else {
      acc = Ns[q * 4] * phi[q1_node(ex, ez, 0, b.nelx)];
      for (int k = 1; k < 4; ++k) acc = acc + Ns[q * 4 + k] * phi[q1_node(ex, ez, k, b.nelx)];
    }
    phiq[g] = acc;
  }
}

// ------------------------------------------------------------------------------------------
// Least-squares particle fits (pic_functions.py:1098-1285) and their slope limiter
// (pic_functions.py:1068-1089).  One thread per element sums the normal equations over the
// element's bin in particle-index order -- each accumulator in the reference's order, products
// formed as the reference writes them ((sx*sx)*sz, sx*(sz*sz), (v*sx)*sz) -- then solves them by
// Gaussian elimination with partial pivoting (the reference calls LAPACK's solve).
struct LsFields {
  const double* phi[MW_MAX_FIELDS];
  double* coef[MW_MAX_FIELDS];
  double* fmin[MW_MAX_FIELDS];
  double* fmax[MW_MAX_FIELDS];
  int n;
};

// Python's min(a, b): a unless b < a
MW_D double py_min(double a, double b) { return b < a ? b : a; }
MW_D double py_sign(double v) { return v < 0 ? -1.0 : 1.0; }

// limiter(c_0, c_1, c_2, S, L, h), pic_functions.py:1068-1089
MW_D void ls_limiter(double c0, double& c1, double& c2, double S, double L, double h) {
  const double k_u = py_min(c0 - S, L - c0);
  double k_l = (fabs(c1) + fabs(c2)) * h / 2;
  if (k_l > k_u) {
    const double c_max = k_u * 2 / h;
    c1 = py_sign(c1) * py_min(fabs(c1), c_max);
    c2 = py_sign(c2) * py_min(fabs(c2), c_max);
  }
  k_l = (fabs(c1) + fabs(c2)) * h / 2;
  if (k_l > k_u) {
    const double c_change = (k_l - k_u) / h;
    c1 = py_sign(c1) * (fabs(c1) - c_change);
    c2 = py_sign(c2) * (fabs(c2) - c_change);
  }
}

// Solve A x = b in place (b -> x) for the NC x NC system: Gaussian elimination, partial pivoting
// (first largest magnitude in the column).  Returns false on a zero pivot.
template <int NC>
MW_D bool small_solve(double (&A)[NC][NC], double (&b)[NC]) {
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    int piv = k;
    double best = fabs(A[k][k]);
#pragma unroll
    for (int i = k + 1; i < NC; ++i)
      if (fabs(A[i][k]) > best) { best = fabs(A[i][k]); piv = i; }
    if (best == 0.0) return false;
    if (piv != k) {
#pragma unroll
      for (int j = 0; j < NC; ++j) { double tmp = A[k][j]; A[k][j] = A[piv][j]; A[piv][j] = tmp; }
      double tmp = b[k]; b[k] = b[piv]; b[piv] = tmp;
    }
#pragma unroll
    for (int i = k + 1; i < NC; ++i) {
      const double l = A[i][k] / A[k][k];
#pragma unroll
      for (int j = k + 1; j < NC; ++j) A[i][j] = A[i][j] - l * A[k][j];
      b[i] = b[i] - l * b[k];
    }
  }
#pragma unroll
  for (int k = NC - 1; k >= 0; --k) {
    double s = b[k];
#pragma unroll
    for (int j = k + 1; j < NC; ++j) s = s - A[k][j] * b[j];
    b[k] = s / A[k][k];
  }
  return true;
}

// element centre x_V[icon_V[8, iel]] = i hx / 2 with i = 2 ex + 1 (build_velocity_mesh.py:116-117)
MW_D double x_centre(const mw_box& b, int ex) { return ((double)(2 * ex + 1) * b.hx) / 2; }
MW_D double z_centre(const mw_box& b, int ez) { return ((double)(2 * ez + 1) * b.hz) / 2; }

template <int NC>
__global__ void k_ls_fit(mw_box b, const int32_t* __restrict__ offsets, const int32_t* __restrict__ order,
                         const double* __restrict__ x, const double* __restrict__ z, LsFields f, double limit_h,
                         int32_t* err) {
  const int64_t nel = (int64_t)b.nelx * b.nelz;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nel; e += (int64_t)gridDim.x * blockDim.x) {
    const int ex = (int)(e % b.nelx), ez = (int)(e / b.nelx);
    const double xe = x_centre(b, ex), ze = z_centre(b, ez);
    const int b0 = offsets[e], b1 = offsets[e + 1];
    if (b1 == b0) { set_flag(err, MW_FLAG_EMPTY_ELEMENT); continue; }
    double A[NC][NC];
#pragma unroll
    for (int i = 0; i < NC; ++i)
#pragma unroll
      for (int j = 0; j < NC; ++j) A[i][j] = 0.0;
    A[0][0] = (double)(b1 - b0);
    for (int j = b0; j < b1; ++j) {                       // pic_functions.py:1134-1146 / :1226-1246
      const int p = order[j];
      const double sx = x[p] - xe, sz = z[p] - ze;
      A[0][1] += sx;
      A[0][2] += sz;
      if (NC == 4) A[0][3] += sx * sz;
      A[1][1] += sx * sx;
      A[1][2] += sx * sz;
      if (NC == 4) A[1][3] += (sx * sx) * sz;
      A[2][2] += sz * sz;
      if (NC == 4) {
        A[2][3] += sx * (sz * sz);
        A[3][3] += (sx * sx) * (sz * sz);
      }
    }
#pragma unroll
    for (int i = 1; i < NC; ++i)
#pragma unroll
      for (int j = 0; j < i; ++j) A[i][j] = A[j][i];
    for (int fi = 0; fi < f.n; ++fi) {
      const double* phi = f.phi[fi];
      double rhs[NC];
#pragma unroll
      for (int i = 0; i < NC; ++i) rhs[i] = 0.0;
      double vmin = 0.0, vmax = 0.0;
      for (int j = b0; j < b1; ++j) {
        const int p = order[j];
        const double sx = x[p] - xe, sz = z[p] - ze, v = phi[p];
        rhs[0] += v;
        rhs[1] += v * sx;
        rhs[2] += v * sz;
        if (NC == 4) rhs[3] += (v * sx) * sz;
        if (j == b0 || v < vmin) vmin = v;                 // np.min / np.max (:1164-1167)
        if (j == b0 || v > vmax) vmax = v;
      }
      double M[NC][NC];
#pragma unroll
      for (int i = 0; i < NC; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) M[i][j] = A[i][j];
      if (!small_solve<NC>(M, rhs)) set_flag(err, MW_FLAG_NONFINITE);
      if (NC == 3 && limit_h > 0.0) ls_limiter(rhs[0], rhs[1], rhs[2], vmin, vmax, limit_h);   // meeuuw.py:1241-1248
#pragma unroll
      for (int i = 0; i < NC; ++i) f.coef[fi][e * NC + i] = rhs[i];
      if (f.fmin[fi]) f.fmin[fi][e] = vmin;
      if (f.fmax[fi]) f.fmax[fi][e] = vmax;
    }
  }
}

// a + b (xq - x_e) + c (zq - z_e) [+ d (xq - x_e)(zq - z_e)] at every qpoint (meeuuw.py:1517-1532)
template <int NC>
__global__ void k_ls_q(mw_box b, const double* __restrict__ coef, const double* __restrict__ xq,
                       const double* __restrict__ zq, double* __restrict__ phiq) {
  const int64_t nq = (int64_t)b.nelx * b.nelz * 9;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < nq; g += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = g / 9;
    const int ex = (int)(e % b.nelx), ez = (int)(e / b.nelx);
    const double* c = coef + e * NC;
    const double dx = xq[g] - x_centre(b, ex), dz = zq[g] - z_centre(b, ez);
    double v = c[0] + c[1] * dx + c[2] * dz;
    if (NC == 4) v = v + c[3] * dx * dz;
    phiq[g] = v;
  }
}

// ------------------------------------------------------------------------------------------
// Population control (pic_functions.py:1621-1812).
//
// numpy's pairwise summation of a float64 array (np.add.reduce, so np.mean / np.average): < 8
// values sequentially from 0; up to 128 in eight interleaved partial sums combined as a tree,
// then the remainder; longer arrays split at an 8-aligned half.  v(k) is the k-th value.
template <typename V>
MW_D double np_pairwise(const V& v, int k0, int n) {
  if (n < 8) {
    double res = 0.0;
    for (int i = 0; i < n; ++i) res += v(k0 + i);
    return res;
  }
  if (n <= 128) {
    double r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = v(k0 + j);
    int i = 8;
    for (; i < n - (n % 8); i += 8)
#pragma unroll
      for (int j = 0; j < 8; ++j) r[j] += v(k0 + i + j);
    double res = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
    for (; i < n; ++i) res += v(k0 + i);
    return res;
  }
  int n2 = n / 2;
  n2 -= n2 % 8;
  return np_pairwise(v, k0, n2) + np_pairwise(v, k0 + n2, n - n2);
}

// counter-based uniform [0, 1) numbers (SplitMix64 finaliser, 53-bit mantissa)
MW_D double splitmix_u01(uint64_t seed, uint64_t k) {
  uint64_t zz = seed + (k + 1) * 0x9E3779B97F4A7C15ull;
  zz = (zz ^ (zz >> 30)) * 0xBF58476D1CE4E5B9ull;
  zz = (zz ^ (zz >> 27)) * 0x94D049BB133111EBull;
  zz ^= zz >> 31;
  return (double)(zz >> 11) * (1.0 / 9007199254740992.0);
}

__global__ void k_pc_need(int32_t nel, int32_t nmin, const int32_t* __restrict__ counts, int32_t* __restrict__ need) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nel; e += (int64_t)gridDim.x * blockDim.x) {
    const int32_t d = nmin - counts[e];
    need[e] = d > 0 ? d : 0;                                      // :1655-1657
  }
}

__global__ void k_pc_flag(int64_t n, const uint8_t* __restrict__ active, int32_t* __restrict__ flag) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    flag[i] = active[i] ? 0 : 1;
}

__global__ void k_pc_list(int64_t n, const int32_t* __restrict__ flag, const int32_t* __restrict__ off,
                          int32_t* __restrict__ avail) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (flag[i]) avail[off[i]] = (int32_t)i;                     // :1680-1688, index order
}

// totals: need_off[nel] (particles needed), avail_off[n] (inactive particles)
__global__ void k_pc_check(const int32_t* __restrict__ need_total, const int32_t* __restrict__ avail_total,
                           int64_t max_new, int32_t* __restrict__ added, int32_t* err) {
  if (threadIdx.x || blockIdx.x) return;
  const int32_t need = *need_total, avail = *avail_total;
  int32_t a = need;
  if (need > avail) { set_flag(err, MW_FLAG_POP_UNAVAILABLE); a = 0; }      // :1722-1733
  else if ((int64_t)need > max_new) { set_flag(err, MW_FLAG_POP_DRAWS); a = 0; }
  *added = a;
}

struct PcFields {
  double* f[MW_MAX_FIELDS];
  int n;
};

// One thread per added particle j: its element (need_off[e] <= j < need_off[e + 1]), its particle
// (avail[j]), its position from two uniform numbers, the nearest particle's material and the
// element particles' means of the `avg` fields (eta, u, w on the box path; :1739-1799).  The
// element's particles are its step-start bin filtered by the current active flags, read before any
// flag changes (k_pc_commit sets them); added particles are inactive, so no thread reads a value
// another one writes.
__global__ void k_pc_fill(mw_box b, const int32_t* __restrict__ need_off, const int32_t* __restrict__ offsets,
                          const int32_t* __restrict__ order, const int32_t* __restrict__ avail,
                          const int32_t* __restrict__ added, const uint8_t* __restrict__ active, int32_t* iel,
                          double* r, double* t, double* x, double* z, int8_t* mat, int32_t* source, PcFields avg,
                          const double* __restrict__ draws, uint64_t seed, int64_t max_new, int32_t* err) {
  const int32_t total = *added;
  const int64_t nel = (int64_t)b.nelx * b.nelz;
  const int nnx = 2 * b.nelx + 1;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < max_new && j < total;
       j += (int64_t)gridDim.x * blockDim.x) {
    int64_t lo = 0, hi = nel - 1;                                // last e with need_off[e] <= j
    while (lo < hi) {
      const int64_t mid = (lo + hi + 1) / 2;
      if (need_off[mid] <= j) lo = mid; else hi = mid - 1;
    }
    const int64_t e = lo;
    const int ex = (int)(e % b.nelx), ez = (int)(e / b.nelx);
    const int b0 = offsets[e], b1 = offsets[e + 1];
    int m = 0;
    for (int k = b0; k < b1; ++k) m += active[order[k]] ? 1 : 0;
    if (m == 0) { set_flag(err, MW_FLAG_POP_MASK_EMPTY); continue; }      // :1747-1748
    const int pid = avail[j];
    const double lo_ = -0.95, hi_ = 0.95;                       // random.uniform(-0.95, 0.95)
    const double u0 = draws ? draws[2 * j] : splitmix_u01(seed, 2 * (uint64_t)j);
    const double u1 = draws ? draws[2 * j + 1] : splitmix_u01(seed, 2 * (uint64_t)j + 1);
    const double rr = lo_ + (hi_ - lo_) * u0, tt = lo_ + (hi_ - lo_) * u1;
    double N[9];
    q2_basis<double>(rr, tt, N);
    double xn = 0.0, zn = 0.0;
    for (int k = 0; k < 9; ++k) {                                 // np.dot(N, x_V[icon_V[:, iel]])
      const int64_t nd = q2_node(ex, ez, k, nnx);
      const int ix = (int)(nd % nnx), iz = (int)(nd / nnx);
      xn = xn + N[k] * (((double)ix * b.hx) / 2);
      zn = zn + N[k] * (((double)iz * b.hz) / 2);
    }
    // nearest particle (the first in index order on ties, as np.argmin)
    double best = 0.0;
    int bi = -1;
    for (int k = b0; k < b1; ++k) {
      const int q = order[k];
      if (!active[q]) continue;
      const double dx = x[q] - xn, dz = z[q] - zn;
      const double d = dx * dx + dz * dz;
      if (bi < 0 || d < best) { best = d; bi = q; }
    }
    auto nth = [&](int kk) -> int {                              // the kk-th particle of the mask
      int c = 0;
      for (int k = b0; k < b1; ++k) {
        const int q = order[k];
        if (!active[q]) continue;
        if (c == kk) return q;
        ++c;
      }
      return order[b0];
    };
    for (int fi = 0; fi < avg.n; ++fi) {                          // np.average(field[mask])
      double* fld = avg.f[fi];
      const double sm = np_pairwise([&](int kk) { return fld[nth(kk)]; }, 0, m);
      fld[pid] = sm / m;
    }
    iel[pid] = (int32_t)e;
    r[pid] = rr;
    t[pid] = tt;
    x[pid] = xn;
    z[pid] = zn;
    if (mat) mat[pid] = mat[bi];
    if (source) source[pid] = bi;
  }
}

__global__ void k_pc_commit(const int32_t* __restrict__ avail, const int32_t* __restrict__ added, int64_t max_new,
                            uint8_t* __restrict__ active) {
  const int32_t total = *added;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < max_new && j < total;
       j += (int64_t)gridDim.x * blockDim.x)
    active[avail[j]] = 1;
}

// Exclusive scan of any length (block scans, recursively over the block totals).
static int scan_any(const int32_t* in, int32_t* out, int64_t n, int32_t* scratch, size_t scratch_ints,
                    cudaStream_t s) {
  const int T = 1024;
  const int64_t nb = (n + T - 1) / T;
  if (nb <= 1) {
    k_scan_block<<<1, T, 0, s>>>(in, out, nullptr, n);
    MW_CHECK_LAUNCH();
    return MW_OK;
  }
  if ((size_t)(2 * nb) > scratch_ints) return MW_ERR_WORKSPACE;
  int32_t* bsum = scratch;
  int32_t* bpre = scratch + nb;
  k_scan_block<<<(unsigned)nb, T, 0, s>>>(in, out, bsum, n);
  MW_CHECK_LAUNCH();
  int rc = scan_any(bsum, bpre, nb, scratch + 2 * nb, scratch_ints - 2 * nb, s);
  if (rc) return rc;
  k_scan_add<<<(unsigned)nb, T, 0, s>>>(out, bpre, n);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

static size_t scan_any_ints(int64_t n) {
  size_t s = 0;
  for (int64_t m = (n + 1023) / 1024; m > 1; m = (m + 1023) / 1024) s += 2 * m;
  return s + 64;
}

}  // namespace mw

using namespace mw;

// blocks of 16 element groups (GROUP lanes each)
static unsigned groups_grid(int64_t nel) {
  const int64_t need = (nel + 256 / GROUP - 1) / (256 / GROUP);
  return (unsigned)(need < 65536 ? need : 65536);
}

static bool box_ok(const mw_box& b) { return b.nelx > 0 && b.nelz > 0 && b.hx > 0 && b.hz > 0; }

extern "C" {

int mw_locate_box(mw_box box, int64_t n, const uint8_t* active, const double* x, const double* z, double* r,
                  double* t, int32_t* iel, int32_t* err, void* stream) {
  if (!box_ok(box) || n < 0) return MW_ERR_BAD_ARG;
  if (n == 0) return MW_OK;
  k_locate<<<grid_all(n, 256), 256, 0, (cudaStream_t)stream>>>(box, n, active, x, z, r, t, iel, err);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

size_t mw_bin_workspace_bytes(int32_t nel) {
  int64_t nb = ((int64_t)nel + 1 + 1023) / 1024;
  return (size_t)((int64_t)nel + 2 * nb + 16) * sizeof(int32_t);
}

int mw_bin_particles(int32_t nel, int64_t n, const uint8_t* active, const int32_t* iel, int32_t* counts,
                     int32_t* offsets, int32_t* order, void* work, size_t work_bytes, int32_t* err, void* stream) {
  if (nel <= 0 || n < 0 || (int64_t)nel > 1024LL * 1024LL) return MW_ERR_BAD_ARG;
  if (work_bytes < mw_bin_workspace_bytes(nel)) return MW_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  int32_t* cursor = (int32_t*)work;
  int32_t* sums = cursor + nel;
  const bool vec = (uintptr_t)iel % 16 == 0 && (uintptr_t)active % 4 == 0;   // four particles a load
  if (cudaMemsetAsync(counts, 0, sizeof(int32_t) * nel, s) != cudaSuccess) return MW_ERR_CUDA;
  if (n > 0) {
    if (vec) k_count<true><<<grid_all((n + 3) / 4, 256), 256, 0, s>>>(n, nel, active, iel, counts, err);
    else k_count<false><<<grid_all((n + 3) / 4, 256), 256, 0, s>>>(n, nel, active, iel, counts, err);
    MW_CHECK_LAUNCH();
  }
  const unsigned nb = (unsigned)((nel + 1023) / 1024);
  if (nb > 1) {
    k_block_sums<<<nb, 1024, 0, s>>>(counts, sums, nel);
    MW_CHECK_LAUNCH();
  }
  k_scan_offsets<<<nb, 1024, 0, s>>>(counts, sums, offsets, cursor, nel);
  MW_CHECK_LAUNCH();
  if (n > 0) {
    if (vec) k_scatter<true><<<grid_all((n + 3) / 4, 256), 256, 0, s>>>(n, nel, active, iel, cursor, order);
    else k_scatter<false><<<grid_all((n + 3) / 4, 256), 256, 0, s>>>(n, nel, active, iel, cursor, order);
    MW_CHECK_LAUNCH();
    k_sort_bins<<<groups_grid(nel), 256, 0, s>>>(nel, offsets, order);
    MW_CHECK_LAUNCH();
  }
  return MW_OK;
}

int mw_project_elements(int32_t nel, const int32_t* offsets, const int32_t* order, const double* rho,
                        const double* eta, int32_t averaging, double* rho_e, double* eta_e, int32_t* err,
                        void* stream) {
  if (nel <= 0 || averaging < 0 || averaging > 2) return MW_ERR_BAD_ARG;
  const unsigned grid = (unsigned)std::min<int64_t>(nel, 8 * num_sms());
  k_project_elements<<<grid, 256, 0, (cudaStream_t)stream>>>(nel, offsets, order, rho, eta, averaging, rho_e, eta_e,
                                                             err);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

size_t mw_project_nodes_workspace_bytes(mw_box box, int32_t nfield) {
  return (size_t)box.nelx * box.nelz * 4 * (nfield + 1) * sizeof(double);
}

int mw_project_nodes(mw_box box, int32_t flavour, int32_t nfield, const int32_t* averaging, const int32_t* offsets,
                     const int32_t* order, const double* r, const double* t, const double* const* phi,
                     double* const* phi_nodal, void* work, size_t work_bytes, void* stream) {
  if (!box_ok(box) || flavour < 1 || flavour > 4 || nfield < 1 || nfield > MW_MAX_FIELDS) return MW_ERR_BAD_ARG;
  ProjFields pf;
  pf.n = nfield;
  for (int f = 0; f < nfield; ++f) {
    if (averaging[f] < 0 || averaging[f] > 2) return MW_ERR_BAD_ARG;
    pf.phi[f] = phi[f]; pf.out[f] = phi_nodal[f]; pf.averaging[f] = averaging[f];
  }
  cudaStream_t s = (cudaStream_t)stream;
  int64_t nc = (int64_t)(box.nelx + 1) * (box.nelz + 1);
  if (work && work_bytes >= mw_project_nodes_workspace_bytes(box, nfield)) {
    const int64_t nel = (int64_t)box.nelx * box.nelz;
    const unsigned tiles = (unsigned)((box.nelx + PFX - 1) / PFX) * (unsigned)((box.nelz + PFZ - 1) / PFZ);
    const double* part = (const double*)work;
    auto go = [&](auto cap) {
      constexpr int NF = cap.value;
      k_project_elem_partials<NF><<<groups_grid(nel), 256, 0, s>>>(box, flavour, offsets, order, r, t, pf,
                                                                   (double*)work);
      if (cudaGetLastError() != cudaSuccess) return MW_ERR_CUDA;
      k_project_finish<NF><<<tiles, PFX * PFZ, 0, s>>>(box, pf, part);
      return cudaGetLastError() == cudaSuccess ? MW_OK : MW_ERR_CUDA;
    };
    if (nfield <= 2) return go(std::integral_constant<int, 2>{});
    if (nfield <= 4) return go(std::integral_constant<int, 4>{});
    return go(std::integral_constant<int, MW_MAX_FIELDS>{});
  } else {
    // no workspace: per-node merge of the incident elements' particles in particle-index order
    k_project_corners<<<grid_for(nc, 128), 128, 0, s>>>(box, flavour, offsets, order, r, t, pf);
  }
  MW_CHECK_LAUNCH();
  int64_t nn = (int64_t)(2 * box.nelx + 1) * (2 * box.nelz + 1);
  k_fill_q2<<<grid_for(nn, 256), 256, 0, s>>>(box, pf);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

int mw_nodal_to_qpoints(mw_box box, int32_t space, const double* N, const double* phi, double* phiq, void* stream) {
  if (!box_ok(box) || space < 0 || space > 2) return MW_ERR_BAD_ARG;
  int64_t nq = (int64_t)box.nelx * box.nelz * 9;
  k_nodal_to_q<<<grid_for(nq, 256), 256, 0, (cudaStream_t)stream>>>(box, space, N, phi, phiq);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

int mw_ls_fit(mw_box box, int32_t ncoef, const int32_t* offsets, const int32_t* order, const double* x,
              const double* z, mw_ls_fields fields, double limit_h, int32_t* err, void* stream) {
  if (!box_ok(box) || !(ncoef == 3 || ncoef == 4) || fields.n < 1 || fields.n > MW_MAX_FIELDS || !offsets ||
      !order || !x || !z)
    return MW_ERR_BAD_ARG;
  if (ncoef == 4 && limit_h > 0.0) return MW_ERR_BAD_ARG;       // the reference limits P1 fits only
  LsFields f;
  f.n = fields.n;
  for (int i = 0; i < fields.n; ++i) {
    if (!fields.phi[i] || !fields.coef[i]) return MW_ERR_BAD_ARG;
    f.phi[i] = fields.phi[i]; f.coef[i] = fields.coef[i]; f.fmin[i] = fields.fmin[i]; f.fmax[i] = fields.fmax[i];
  }
  const int64_t nel = (int64_t)box.nelx * box.nelz;
  cudaStream_t s = (cudaStream_t)stream;
  if (ncoef == 3) k_ls_fit<3><<<grid_for(nel, 128), 128, 0, s>>>(box, offsets, order, x, z, f, limit_h, err);
  else k_ls_fit<4><<<grid_for(nel, 128), 128, 0, s>>>(box, offsets, order, x, z, f, 0.0, err);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

int mw_ls_to_qpoints(mw_box box, int32_t ncoef, const double* coef, const double* xq, const double* zq,
                     double* phiq, void* stream) {
  if (!box_ok(box) || !(ncoef == 3 || ncoef == 4) || !coef || !xq || !zq || !phiq) return MW_ERR_BAD_ARG;
  const int64_t nq = (int64_t)box.nelx * box.nelz * 9;
  cudaStream_t s = (cudaStream_t)stream;
  if (ncoef == 3) k_ls_q<3><<<grid_for(nq, 256), 256, 0, s>>>(box, coef, xq, zq, phiq);
  else k_ls_q<4><<<grid_for(nq, 256), 256, 0, s>>>(box, coef, xq, zq, phiq);
  MW_CHECK_LAUNCH();
  return MW_OK;
}

size_t mw_population_workspace_bytes(int32_t nel, int64_t nparticle) {
  const size_t ints = (size_t)2 * (nel + 1) + (size_t)3 * (nparticle + 1) + scan_any_ints(nel + 1) +
                      scan_any_ints(nparticle + 1) + 64;
  return ints * sizeof(int32_t);
}

int mw_population_control(mw_box box, int32_t nparticle_min, int64_t nparticle, const int32_t* counts,
                          const int32_t* offsets, const int32_t* order, uint8_t* active, int32_t* iel, double* r,
                          double* t, double* x, double* z, int8_t* mat, int32_t* source, mw_pc_fields avg,
                          const double* draws, int64_t max_new, uint64_t seed, int32_t* added, void* work,
                          size_t work_bytes, int32_t* err, void* stream) {
  if (!box_ok(box) || nparticle < 1 || nparticle > INT32_MAX - 1 || !counts || !offsets || !order || !active ||
      !iel || !r || !t || !x || !z || !added || !work || avg.n < 0 || avg.n > MW_MAX_FIELDS)
    return MW_ERR_BAD_ARG;
  PcFields pf;
  pf.n = avg.n;
  for (int i = 0; i < avg.n; ++i) {
    if (!avg.f[i]) return MW_ERR_BAD_ARG;
    pf.f[i] = avg.f[i];
  }
  const int32_t nel = box.nelx * box.nelz;
  if (work_bytes < mw_population_workspace_bytes(nel, nparticle)) return MW_ERR_WORKSPACE;
  if (!draws) max_new = nparticle;                 // the device draws as many numbers as it needs
  if (max_new < 0) return MW_ERR_BAD_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  int32_t* need = (int32_t*)work;
  int32_t* need_off = need + (nel + 1);
  int32_t* flag = need_off + (nel + 1);
  int32_t* avail_off = flag + (nparticle + 1);
  int32_t* avail = avail_off + (nparticle + 1);
  int32_t* scratch = avail + (nparticle + 1);
  const size_t scratch_ints = work_bytes / sizeof(int32_t) - (size_t)(scratch - need);
  k_pc_need<<<grid_for(nel, 256), 256, 0, s>>>(nel, nparticle_min, counts, need);
  MW_CHECK_LAUNCH();
  int rc = scan_any(need, need_off, nel, scratch, scratch_ints, s);
  if (rc) return rc;
  k_total<<<1, 32, 0, s>>>(need, need_off, nel);
  MW_CHECK_LAUNCH();
  k_pc_flag<<<grid_for(nparticle, 256), 256, 0, s>>>(nparticle, active, flag);
  MW_CHECK_LAUNCH();
  rc = scan_any(flag, avail_off, nparticle, scratch, scratch_ints, s);
  if (rc) return rc;
  k_total<<<1, 32, 0, s>>>(flag, avail_off, nparticle);
  MW_CHECK_LAUNCH();
  k_pc_list<<<grid_for(nparticle, 256), 256, 0, s>>>(nparticle, flag, avail_off, avail);
  MW_CHECK_LAUNCH();
  k_pc_check<<<1, 32, 0, s>>>(need_off + nel, avail_off + nparticle, max_new, added, err);
  MW_CHECK_LAUNCH();
  if (max_new > 0) {
    k_pc_fill<<<grid_for(max_new, 128), 128, 0, s>>>(box, need_off, offsets, order, avail, added, active, iel, r, t,
                                                     x, z, mat, source, pf, draws, seed, max_new, err);
    MW_CHECK_LAUNCH();
    k_pc_commit<<<grid_for(max_new, 256), 256, 0, s>>>(avail, added, max_new, active);
    MW_CHECK_LAUNCH();
  }
  return MW_OK;
}

}  // extern "C"
