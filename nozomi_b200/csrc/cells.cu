// Uniform-grid cell lists on the GPU: the work of DiffSim3d.set_segments
// (simulation_toolkit/simulation_engine/diffsim3d.py:107-174), which the
// reference does on the host with a numpy loop over cells x spheres (twice) and
// an argsort per cell.
//
// Membership is the reference's predicate, in float64 and in its operation
// order (diffsim3d.py:128-141): sphere s belongs to cell (n, m, p) when all six
// boundary distances of its bounding box are below jump_tol.  The predicate is
// separable per axis and, per axis, monotone in the cell index, so each sphere
// enumerates only the box of cells it can belong to.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_fp16.h>
#include "kernels.cuh"

namespace nz {

// in_segment's two terms on one axis for cell index n (diffsim3d.py:128-133).
__device__ __forceinline__ double seg_lo(double n, double dL, double r, double x, double L) {
  return __dsub_rn(__dsub_rn(__dsub_rn(__dmul_rn(n, dL), r), x), L / 2);
}
__device__ __forceinline__ double seg_hi(double n, double dL, double r, double x, double L) {
  return __dsub_rn(x, __dsub_rn(__dadd_rn(__dmul_rn(n + 1, dL), r), L / 2));
}

struct CellGeom {
  double Lx, Ly, Lz;
  int nx, ny, nz;
  double tol;
};

// Valid cell range [lo, hi] on one axis (empty when lo > hi, and for a lane
// that is not live), by each G lanes of a warp, a candidate cell a lane.
template <int G>
__device__ __forceinline__ void axis_range(bool live, double x, double r, double L, int nseg, double tol, int lane,
                                           int& lo, int& hi) {
  const double dL = L / nseg;
  const int a = max(int(floor((x - r + L / 2 - tol) / dL)) - 2, 0);
  const int b = live ? min(int(ceil((tol + r + x + L / 2) / dL)) + 2, nseg - 1) : -1;
  lo = 1;
  hi = 0;
  for (int base = a; __any_sync(0xffffffffu, base <= b); base += G) {
    const int n = base + lane % G;
    const unsigned ok = __ballot_sync(0xffffffffu, n <= b && seg_lo(double(n), dL, r, x, L) < tol &&
                                                       seg_hi(double(n), dL, r, x, L) < tol) >>
                            (lane & ~(G - 1)) &
                        (0xffffffffu >> (32 - G));
    if (ok) {
      if (lo > hi) lo = base + __ffs(ok) - 1;
      hi = base + 31 - __clz(ok);
    }
  }
}

// Rounded membership, for the fused walk's near lists: a sphere is listed in
// a cell of its box-test window (in_segment < margin) only when the
// Euclidean distance from its centre to the cell's box is at most
// r + margin + 1e-4 um.  A walker in the cell (or within d of it) can touch
// or lie inside only spheres whose centre is within r + tol + reach + d of
// the box, and the fused walk takes the near list only while
// (d + reach) * 1.02 + tol + 2 nm <= margin, so these lists hold every
// sphere the walk can meet; the corners of the box test's window, about a
// third of its entries for cells small beside the spheres, are left out.
__device__ __forceinline__ bool within_round(double x, double y, double z, double r, const CellGeom& g, int n, int m,
                                             int p) {
  const double dLx = g.Lx / g.nx, dLy = g.Ly / g.ny, dLz = g.Lz / g.nz;
  const double x0 = n * dLx - g.Lx / 2, y0 = m * dLy - g.Ly / 2, z0 = p * dLz - g.Lz / 2;
  const double ex = fmax(fmax(x0 - x, 0.0), x - (x0 + dLx));
  const double ey = fmax(fmax(y0 - y, 0.0), y - (y0 + dLy));
  const double ez = fmax(fmax(z0 - z, 0.0), z - (z0 + dLz));
  const double R = r + g.tol + 1e-4;
  return ex * ex + ey * ey + ez * ez <= R * R;
}

// The cells of every sphere, counted (items null) or filled in: G lanes a
// sphere, over the cells of its box, so that their atomics fall on
// neighbouring counters.  Bound by the atomics, and for many spheres in few
// cells each by the double-precision ranges, which every lane of a sphere
// forms (a warp a sphere took 0.60 ms to count 1.1e6 spheres of 23 cells, two
// lanes 0.11).
template <bool ROUND, int G>
__global__ void __launch_bounds__(256) cells_members_kernel(const double* __restrict__ sph, int S, CellGeom g,
                                                            const int* __restrict__ offsets, int* __restrict__ cursor,
                                                            int* __restrict__ items) {
  const size_t at = (blockIdx.x * size_t(blockDim.x) + threadIdx.x) / G;
  const bool live = at < size_t(S);
  const int s = live ? int(at) : 0, lane = threadIdx.x & 31;
  const double x = sph[s], y = sph[size_t(S) + s], z = sph[2 * size_t(S) + s], r = sph[3 * size_t(S) + s];
  int x0, x1, y0, y1, z0, z1;
  axis_range<G>(live, x, r, g.Lx, g.nx, g.tol, lane, x0, x1);
  axis_range<G>(live, y, r, g.Ly, g.ny, g.tol, lane, y0, y1);
  axis_range<G>(live, z, r, g.Lz, g.nz, g.tol, lane, z0, z1);
  if (x0 > x1 || y0 > y1 || z0 > z1) return;
  auto add = [&](int n, int m, int p) {
    if (ROUND && !within_round(x, y, z, r, g, n, m, p)) return;
    const size_t c = (size_t(p) * g.ny + m) * g.nx + n;
    const int slot = atomicAdd(cursor + c, 1);
    if (items) items[offsets[c] + slot] = s;
  };
  const unsigned Y = unsigned(y1 - y0 + 1), Z = unsigned(z1 - z0 + 1);
  const unsigned first = lane % G;
  if (ROUND && G <= 2) {  // a lane takes every G-th row: the distances in y and z are formed once a row
    unsigned m = first % Y, p = first / Y;
    while (p < Z) {
      for (int n = x0; n <= x1; ++n) add(n, y0 + int(m), z0 + int(p));
      m += G;
      while (m >= Y) {
        m -= Y;
        ++p;
      }
    }
    return;
  }
  // every G-th cell of the box: the lane's first, and the step of G, as digits
  const unsigned X = unsigned(x1 - x0 + 1);
  unsigned n = first % X, m = first / X % Y, p = first / X / Y;
  const unsigned dn = G % X, dm = G / X % Y, dp = G / X / Y;
  while (p < Z) {
    add(x0 + int(n), y0 + int(m), z0 + int(p));
    n += dn;
    m += dm;
    p += dp;
    if (n >= X) {
      n -= X;
      ++m;
    }
    if (m >= Y) {
      m -= Y;
      ++p;
    }
  }
}

template <bool ROUND>
int cells_members(const double* sph, int S, const CellGeom& g, const int* offsets, int* cursor, int* items,
                  cudaStream_t st) {
  auto launch = [&](auto kernel, int lanes) {
    kernel<<<unsigned((size_t(S) * lanes + 255) / 256), 256, 0, st>>>(sph, S, g, offsets, cursor, items);
  };
  // lanes a sphere: many while spheres alone do not fill the GPU.  Counted, one
  // thread a sphere / 2 / 8 / 32 lanes: 6,000 spheres of 450 cells 0.091 /
  // 0.040 / 0.021 / 0.019 ms, 80,000 of 247 0.159 / 0.103 / 0.056 / 0.079,
  // 3e5 of 8 0.076 / 0.050 / 0.058 / 0.177, 1e6 of 4 0.110 / 0.080 / 0.152 / 0.542.
  if (S <= 16384) launch(cells_members_kernel<ROUND, 32>, 32);
  else if (S <= 524288) launch(cells_members_kernel<ROUND, 8>, 8);
  else launch(cells_members_kernel<ROUND, 2>, 2);
  return check_launch("cells_members_kernel");
}

// Ascending order within each cell's list, keys in [0, S).  A warp per list of
// up to kWarpSort entries: nothing to do when they ascend already, else a
// bitonic sort in registers, entry 32 k + lane in v[k].  A CTA notes the
// lists of two and more entries among its `chunk` cells (nearly all cells of a
// fine grid in a nearly empty box have none: a warp launched for each of 8e6
// cells took 0.53 ms) and its warps take them in turn.
// Bound by its compare-exchanges (21 rounds for 33-64 entries).  One thread
// per cell and a heapsort in memory took 2.1 ms for two lists of 420,000
// cells (57 entries a cell in one of them), this
// 0.3 ms with the check of their index lists.
constexpr int kWarpSort = 128;

template <int R>
__device__ __forceinline__ void bitonic_sort(int (&v)[R], int lane) {
#pragma unroll
  for (int size = 2; size <= 32 * R; size *= 2) {
#pragma unroll
    for (int stride = size / 2; stride > 0; stride /= 2) {
      if (stride >= 32) {
#pragma unroll
        for (int k = 0; k < R; ++k) {
          const int o = k ^ (stride / 32);
          if (o > k) {
            const bool up = ((32 * k) & size) == 0;
            const int a = min(v[k], v[o]), b = max(v[k], v[o]);
            v[k] = up ? a : b;
            v[o] = up ? b : a;
          }
        }
      } else {
#pragma unroll
        for (int k = 0; k < R; ++k) {
          const int o = __shfl_xor_sync(0xffffffffu, v[k], stride);
          const bool up = ((32 * k + lane) & size) == 0;
          v[k] = up == ((lane & stride) == 0) ? min(v[k], o) : max(v[k], o);
        }
      }
    }
  }
}

template <int R, typename T>
__device__ __forceinline__ void sort_list(T* a, int n, int lane) {
  int v[R];
  bool sorted = true;
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int i = 32 * k + lane;
    v[k] = i < n ? int(a[i]) : 0x7fffffff;
    const int next = i + 1 < n ? int(a[i + 1]) : 0x7fffffff;
    sorted &= v[k] <= next;
  }
  if (__all_sync(0xffffffffu, sorted)) return;
  bitonic_sort<R>(v, lane);
#pragma unroll
  for (int k = 0; k < R; ++k)
    if (32 * k + lane < n) a[32 * k + lane] = T(v[k]);
}

template <typename T>
__global__ void __launch_bounds__(256) lists_sort_kernel(const int* __restrict__ start, const int* __restrict__ count,
                                                         int ncell, int chunk, T* __restrict__ list) {
  __shared__ int s_cells[256], s_n;
  const int t = threadIdx.x, lane = t & 31;
  if (t == 0) s_n = 0;
  __syncthreads();
  const long long mine = 1ll * blockIdx.x * chunk + t;
  if (t < chunk && mine < ncell && count[mine] >= 2 && count[mine] <= kWarpSort)
    s_cells[atomicAdd(&s_n, 1)] = int(mine);
  __syncthreads();
  for (int q = t >> 5; q < s_n; q += 8) {
    const int c = s_cells[q], n = count[c];
    T* a = list + start[c];
    if (n <= 32) sort_list<1>(a, n, lane);
    else if (n <= 64) sort_list<2>(a, n, lane);
    else sort_list<4>(a, n, lane);
  }
}

// Longer lists (coarse grids): a CTA per list marks its entries in a bitmap
// of the S keys in shared memory and reads them back in order, unless they
// ascend already.  CTAs look over `chunk` cells at a time, few enough that a
// coarse grid's lists reach every SM.  Lists with repeats are heapsorted by
// one thread.  With more keys than the bitmap holds, a CTA sorts a list of up
// to kSharedSort entries in shared memory by a bitonic network, and beyond
// that each thread heapsorts a list.  1.1e6 spheres with lists of 564: the
// heapsorts, a thread each, took 2.9 ms from entries almost in order and 4.2
// from the order that cells_members_kernel leaves; the network 0.38 ms.
template <typename T>
__device__ void heapsort(T* a, int n) {
  auto sift = [&](int root, int end) {
    while (2 * root + 1 < end) {
      int child = 2 * root + 1;
      if (child + 1 < end && a[child] < a[child + 1]) child++;
      if (!(a[root] < a[child])) return;
      const T t = a[root];
      a[root] = a[child];
      a[child] = t;
      root = child;
    }
  };
  for (int i = n / 2 - 1; i >= 0; --i) sift(i, n);
  for (int end = n - 1; end > 0; --end) {
    const T t = a[0];
    a[0] = a[end];
    a[end] = t;
    sift(0, end);
  }
}

constexpr int kBitmapKeys = 1 << 20;  // 128 KiB of shared memory
constexpr int kSharedSort = 1 << 13;  // 32 KiB: seven CTAs an SM

template <typename T>
__global__ void __launch_bounds__(256) long_lists_sort_kernel(const int* __restrict__ start,
                                                              const int* __restrict__ count, int ncell, int chunk,
                                                              int S, T* __restrict__ list) {
  extern __shared__ unsigned s_bits[];  // (S + 31) / 32 words, or kSharedSort keys
  __shared__ int s_cells[256];
  __shared__ int s_n, s_repeats, s_before[8];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int words = (S + 31) / 32;
  for (long long base = 1ll * blockIdx.x * chunk; base < ncell; base += 1ll * gridDim.x * chunk) {
    const bool is_long = t < chunk && base + t < ncell && count[base + t] > kWarpSort;
    __syncthreads();
    if (t == 0) s_n = 0;
    __syncthreads();
    if (is_long) s_cells[atomicAdd(&s_n, 1)] = int(base) + t;
    __syncthreads();
    const int found = s_n;
    for (int q = 0; q < found; ++q) {
      const int c = s_cells[q], n = count[c];
      T* a = list + start[c];
      bool sorted = true;
      for (int i = t + 1; i < n; i += 256) sorted &= a[i - 1] <= a[i];
      if (__syncthreads_and(sorted)) continue;
      if (S > kBitmapKeys) {
        if (n > kSharedSort) continue;
        int* const v = reinterpret_cast<int*>(s_bits);
        int size2 = 2 * kWarpSort;
        while (size2 < n) size2 *= 2;
        for (int i = t; i < size2; i += 256) v[i] = i < n ? int(a[i]) : 0x7fffffff;
        for (int size = 2; size <= size2; size *= 2)
          for (int stride = size / 2; stride > 0; stride /= 2) {
            __syncthreads();
            for (int i = t; i < size2 / 2; i += 256) {
              const int k = 2 * i - (i & (stride - 1)), o = k + stride;
              const int x = v[k], y = v[o];
              if ((x > y) == ((k & size) == 0)) {
                v[k] = y;
                v[o] = x;
              }
            }
          }
        __syncthreads();
        for (int i = t; i < n; i += 256) a[i] = T(v[i]);
        __syncthreads();
        continue;
      }
      for (int w = t; w < words; w += 256) s_bits[w] = 0u;
      if (t == 0) s_repeats = 0;
      __syncthreads();
      for (int i = t; i < n; i += 256) {
        const unsigned k = unsigned(a[i]);
        if (k >= unsigned(S) || (atomicOr(&s_bits[k >> 5], 1u << (k & 31)) >> (k & 31)) & 1u) s_repeats = 1;
      }
      __syncthreads();
      if (s_repeats) {
        if (t == 0) heapsort(a, n);
        __syncthreads();
        continue;
      }
      // a run of words per thread: its entries' first place, then the entries
      const int per = (words + 255) / 256, w0 = min(words, t * per), w1 = min(words, w0 + per);
      int mine = 0;
      for (int w = w0; w < w1; ++w) mine += __popc(s_bits[w]);
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) s_before[warp] = incl;
      __syncthreads();
      int at = incl - mine;
      for (int w = 0; w < warp; ++w) at += s_before[w];
      for (int w = w0; w < w1; ++w)
        for (unsigned b = s_bits[w]; b; b &= b - 1) a[at++] = T(32 * w + __ffs(b) - 1);
      __syncthreads();
    }
    if (S > kBitmapKeys && is_long && count[base + t] > kSharedSort) {
      T* a = list + start[base + t];
      const int n = count[base + t];
      int i = 1;
      while (i < n && a[i - 1] <= a[i]) ++i;
      if (i < n) heapsort(a, n);
    }
  }
}

// Both kernels over a set of lists with keys below S.
template <typename T>
int sort_lists(const int* start, const int* count, int ncell, int S, T* list, cudaStream_t st) {
  // cells of a CTA: a list a warp for few cells, four waves of CTAs (8 an SM) for more
  const int chunk = std::min(256, std::max(8, ncell / (4 * 8 * 148)));
  lists_sort_kernel<T><<<unsigned((ncell + chunk - 1ll) / chunk), 256, 0, st>>>(start, count, ncell, chunk, list);
  int rc = check_launch("lists_sort_kernel");
  if (rc) return rc;
  const size_t bytes = S <= kBitmapKeys ? size_t((S + 31) / 32) * sizeof(unsigned) : kSharedSort * sizeof(int);
  // at every size: the 48 KiB allowed without it are for static and dynamic bytes together
  if (cudaFuncSetAttribute(long_lists_sort_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kBitmapKeys / 8) != cudaSuccess)
    return check_launch("long_lists_sort_kernel attribute");
  const int most = 148 * 4, per = std::min(256, (ncell - 1) / most + 1);
  const int ctas = std::min(most, (ncell - 1) / per + 1);
  long_lists_sort_kernel<T><<<unsigned(ctas), 256, bytes, st>>>(start, count, ncell, per, S, list);
  return check_launch("long_lists_sort_kernel");
}

// Orderable 64-bit key of a double (ascending keys = ascending values).
__device__ __forceinline__ unsigned long long okey(double v) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// The padded table.  in_segment of a sphere and a cell is the largest of six
// distances, two per axis; a CTA takes up to kSegCells cells of one row
// (same m, p), so the y and z distances of a sphere are formed once for all
// of them.  The K spheres of least (in_segment, index) of each cell:
//   1. a histogram of the distances over kSegBuckets equal steps finds the
//      step of the K-th.  A sphere's distances from the row and from the
//      row's first cell are formed in double precision (a sphere far larger
//      than the box, a flat wall, is the difference of two large numbers),
//      rounded, and moved from cell to cell in single precision: within the
//      steps the roundings are a thousandth of one (1.5e-3 of the box), so
//      spheres two steps below the K-th are in, two steps above out;
//   2. the spheres of the three steps between, a few tens, are collected and
//      ranked by their exact double-precision keys.  Beyond kSegCandidates
//      (cells of hundreds of spheres, equal distances) a radix select over
//      the collected keys takes over, or over the passes' spheres when shared
//      memory does not hold the keys: 1e5 spheres in 3^3 cells, 8,412 a cell,
//      take 1.21 ms, 2.86 with the keys formed anew for each digit;
//   3. two passes in index order count and write the chosen ones, a run of
//      spheres per warp, ties to the lower index.
// A sixteenth of the spheres, looked at first, gives a step that almost
// surely lies beyond the K-th; a sphere whose y or z distance is past it is
// passed over from then on, which is most of them (without success the
// histogram is taken again over all steps); those left, a few hundred, are
// noted and the later passes look at them alone.  Bound by the one full pass
// over the spheres, from L2.  20^3 cells of 28,890 spheres took 7.6 ms with a CTA a cell and
// ten double-precision passes over all spheres (8-bit radix select, then the
// output), 0.37 ms so.
constexpr int kSegCells = 8, kSegBuckets = 1024, kSegCandidates = 256, kSegSample = 16;
constexpr int kSegKeys = kSegCells * kSegBuckets / 2;  // keys that fit where the histograms were
constexpr int kSegKept = 4096;          // spheres noted for the later passes
constexpr int kSegBitmap = 262144;      // spheres up to which they are noted

struct SegCell {
  int step;                // step of the K-th smallest
  int rank, count;         // how many of the steps around it are taken, of how many
  unsigned long long key;  // key of the K-th; rank: how many spheres equal to it are taken
};

__device__ __forceinline__ double axis_distance(double lo, double hi, double r, double x, double half) {
  // seg_lo and seg_hi with n dL and (n + 1) dL formed once per cell
  return fmax(__dsub_rn(__dsub_rn(__dsub_rn(lo, r), x), half), __dsub_rn(x, __dsub_rn(__dadd_rn(hi, r), half)));
}

__global__ void __launch_bounds__(256, 3) segments_fill_kernel(const double* __restrict__ sph, int S, CellGeom g, int K,
                                                            int per, int* __restrict__ segments) {
  __shared__ union {
    int hist[kSegCells][kSegBuckets];
    unsigned long long keys[kSegKeys];
  } sm;
  __shared__ int s_digit[256];
  __shared__ SegCell s_cell[kSegCells];
  __shared__ int s_n[kSegCells];
  __shared__ int s_less[8][kSegCells], s_tie[8][kSegCells];
  __shared__ int s_limit;
  __shared__ int s_warp[8];
  extern __shared__ int s_kept[];  // kSegKept spheres within the limit, in order; a bit per sphere
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int chunks = (g.nx + per - 1) / per;
  const int n0 = int(blockIdx.x % chunks) * per, nc = min(per, g.nx - n0);
  const int row = int(blockIdx.x / chunks), m = row % g.ny, p = row / g.ny;
  int* const out = segments + (size_t(row) * g.nx + n0) * K;
  if (K >= S) {  // every sphere is in every list
    for (int c = 0; c < nc; ++c)
      for (int i = t; i < S; i += blockDim.x) out[size_t(c) * K + i] = i;
    return;
  }
  const double dLx = g.Lx / g.nx, dLy = g.Ly / g.ny, dLz = g.Lz / g.nz;
  // for the steps: half a cell, the centres of the row and of its first cell
  const float hx = float(0.5 * dLx), hy = float(0.5 * dLy), hz = float(0.5 * dLz), fx = float(dLx);
  const double oy = (m + 0.5) * dLy - g.Ly / 2, oz = (p + 0.5) * dLz - g.Lz / 2, ox = (n0 + 0.5) * dLx - g.Lx / 2;
  const float span = float(fmax(g.Lx, fmax(g.Ly, g.Lz)));
  const float scale = float(kSegBuckets) / (1.5f * span);
  auto step_of = [&](float v) {  // (v + span / 2) * scale; ascending in v, NaN last as its key
    return __float2int_rd(fmaxf(0.0f, fminf(float(kSegBuckets - 1), __fmaf_rn(v, scale, kSegBuckets / 3.0f))));
  };
  auto yz_step = [&](int i, float& yz) {
    const double r = sph[3 * size_t(S) + i];
    yz = fmaxf(float(fabs(sph[size_t(S) + i] - oy) - r) - hy, float(fabs(sph[2 * size_t(S) + i] - oz) - r) - hz);
    return step_of(yz);
  };
  auto x_ends = [&](int i, float& xl, float& xh) {  // both sides' distances from the first cell's centre
    const double x = sph[i] - ox, r = sph[3 * size_t(S) + i];
    xl = float(x - r);
    xh = float(-x - r);
  };
  auto step_in = [&](int c, float yz, float xl, float xh) {
    const float at = c * fx;
    return step_of(fmaxf(yz, fmaxf(xl - at, xh + at) - hx));
  };
  auto key_of = [&](int i, int c) {  // exact: the reference's in_segment, operation by operation
    const double r = sph[3 * size_t(S) + i];
    double v = axis_distance(__dmul_rn(double(n0 + c), dLx), __dmul_rn(double(n0 + c) + 1, dLx), r, sph[i], g.Lx / 2);
    v = fmax(v, axis_distance(__dmul_rn(double(m), dLy), __dmul_rn(double(m) + 1, dLy), r, sph[size_t(S) + i],
                              g.Ly / 2));
    v = fmax(v, axis_distance(__dmul_rn(double(p), dLz), __dmul_rn(double(p) + 1, dLz), r, sph[2 * size_t(S) + i],
                              g.Lz / 2));
    return okey(v);
  };
  // the step at which a histogram's running count reaches `target`, or
  // `steps`, by a warp; `run`: the count before it
  auto reach = [&](const int* hist, int steps, int target, int& run) {
    run = 0;
    for (int base = 0; base < steps; base += 32) {
      int incl = hist[base + lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      const unsigned reached = __ballot_sync(0xffffffffu, run + incl >= target);
      if (reached) {
        const int b = __ffs(reached) - 1;
        run += __shfl_sync(0xffffffffu, incl - hist[base + lane], b);
        return base + b;
      }
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    return steps;
  };
  const unsigned lower = (1u << lane) - 1u;
  int len = S;  // the passes' spheres: all, or the first len entries of s_kept
  bool noted = false;
  auto sphere = [&](int k) { return noted ? s_kept[k] : k; };
  // histograms of every stride-th of the passes' spheres, steps up to `limit`
  auto histogram = [&](int stride, int limit) {
    __syncthreads();
    for (int i = t; i < nc * kSegBuckets; i += blockDim.x) (&sm.hist[0][0])[i] = 0;
    __syncthreads();
    for (int k = t * stride; k < len; k += blockDim.x * stride) {
      const int i = sphere(k);
      float yz, xl, xh;
      if (yz_step(i, yz) > limit) continue;
      x_ends(i, xl, xh);
      for (int c = 0; c < nc; ++c) {
        const int b = step_in(c, yz, xl, xh);
        if (b <= limit) atomicAdd(&sm.hist[c][b], 1);
      }
    }
    __syncthreads();
  };
  // notes the spheres whose y and z distances are within the limit, in order
  auto note = [&](int limit) {
    unsigned* const bits = reinterpret_cast<unsigned*>(s_kept + kSegKept);
    const int words = (S + 31) / 32;
#pragma unroll 4
    for (int w = warp; w < words; w += 8) {
      const int i = 32 * w + lane;
      float yz;
      const unsigned mask = __ballot_sync(0xffffffffu, i < S && yz_step(min(i, S - 1), yz) <= limit);
      if (lane == 0) bits[w] = mask;
    }
    __syncthreads();
    const int each = (words + 255) / 256, w0 = min(words, t * each), w1 = min(words, w0 + each);
    int mine = 0;
    for (int w = w0; w < w1; ++w) mine += __popc(bits[w]);
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int at = incl - mine, all = 0;
    for (int w = 0; w < 8; ++w) {
      if (w < warp) at += s_warp[w];
      all += s_warp[w];
    }
    if (all > kSegKept) return;
    for (int w = w0; w < w1; ++w)
      for (unsigned b = bits[w]; b; b &= b - 1) s_kept[at++] = 32 * w + __ffs(b) - 1;
    noted = true;
    len = all;
    __syncthreads();
  };

  // 1. the step of each cell's K-th
  int limit = kSegBuckets - 1;
  if (S >= 128 * kSegSample) {
    histogram(kSegSample, limit);
    if (t == 0) s_limit = 0;
    __syncthreads();
    if (warp < nc) {
      int before;
      const int b = reach(sm.hist[warp], kSegBuckets, 2 * (K / kSegSample) + 8, before);
      if (lane == 0) atomicMax(&s_limit, b);
    }
    __syncthreads();
    limit = min(limit, s_limit + 2);
    if (S <= kSegBitmap) note(limit);
  }
  for (;;) {
    histogram(1, limit);
    if (t == 0) s_limit = 0;
    __syncthreads();
    if (warp < nc) {
      int below;
      const int b = reach(sm.hist[warp], kSegBuckets, K, below);
      if (b > 0) below -= sm.hist[warp][b - 1];  // up to two steps below the K-th's
      if (lane == 0) {
        SegCell& q = s_cell[warp];
        q.step = b;
        q.count = 0;
        for (int k = max(0, b - 1); k <= min(kSegBuckets - 1, b + 1); ++k) q.count += sm.hist[warp][k];
        q.rank = K - below;
        s_n[warp] = 0;
        atomicMax(&s_limit, b + 1);
      }
    }
    __syncthreads();
    if (s_limit <= limit || limit == kSegBuckets - 1) break;  // the steps around every K-th were counted
    limit = kSegBuckets - 1;
    noted = false;
    len = S;
  }
  limit = min(limit, s_limit);

  // 2. the exact key of the K-th
  const int room = kSegKeys / per;  // keys of a cell
  for (int k = t; k < len; k += blockDim.x) {
    const int i = sphere(k);
    float yz, xl, xh;
    if (yz_step(i, yz) > limit) continue;
    x_ends(i, xl, xh);
    for (int c = 0; c < nc; ++c) {
      const int step = s_cell[c].step;
      if (s_cell[c].count > room || abs(step_in(c, yz, xl, xh) - step) > 1) continue;
      sm.keys[c * room + atomicAdd(&s_n[c], 1)] = key_of(i, c);
    }
  }
  __syncthreads();
  if (warp < nc && s_n[warp] <= kSegCandidates) {  // each candidate: how many are less, how many equal
    const int n = s_n[warp], rank = s_cell[warp].rank;
    const unsigned long long* const keys = sm.keys + warp * room;
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
      const unsigned long long k = keys[i];
      int less = 0, same = 0;
      for (int j = 0; j < n; ++j) {
        less += keys[j] < k;
        same += keys[j] == k;
      }
      if (less < rank && rank <= less + same) {  // every candidate equal to the K-th writes the same
        s_cell[warp].key = k;
        s_n[warp] = rank - less;
      }
    }
    __syncwarp();
    if (lane == 0 && n > 0) s_cell[warp].rank = s_n[warp];
  }
  __syncthreads();
  for (int c = 0; c < nc; ++c) {  // many spheres around the K-th: radix select by 8 bits over them
    const SegCell q = s_cell[c];
    if (q.count <= kSegCandidates) continue;
    const bool held = q.count <= room;  // their keys were collected
    unsigned long long prefix = 0ull, mask = 0ull;
    int rank = q.rank;
    for (int digit = 7; digit >= 0; --digit) {
      __syncthreads();
      s_digit[t] = 0;
      __syncthreads();
      auto add = [&](unsigned long long k) {
        if ((k & mask) == prefix) atomicAdd(&s_digit[(k >> (8 * digit)) & 255ull], 1);
      };
      if (held)
        for (int j = t; j < q.count; j += blockDim.x) add(sm.keys[c * room + j]);
      for (int j = t; !held && j < len; j += blockDim.x) {
        const int i = sphere(j);
        float yz, xl, xh;
        if (yz_step(i, yz) > limit) continue;
        x_ends(i, xl, xh);
        if (abs(step_in(c, yz, xl, xh) - q.step) <= 1) add(key_of(i, c));
      }
      __syncthreads();
      int before;
      const int b = reach(s_digit, 256, rank, before);
      rank -= before;
      prefix |= static_cast<unsigned long long>(b) << (8 * digit);
      mask |= 255ull << (8 * digit);
    }
    __syncthreads();
    if (t == 0) {
      s_cell[c].key = prefix;
      s_cell[c].rank = rank;
    }
    __syncthreads();
  }

  // 3. a run of the passes' spheres per warp: count, then write in order
  const int run = (len + 255) / 256 * 32;
  const int k0 = min(len, warp * run), k1 = min(len, k0 + run);
  auto classify = [&](int i, int c, float yz, float xl, float xh, bool& less, bool& tie) {
    const int d = step_in(c, yz, xl, xh) - s_cell[c].step;
    less = d < -1;
    tie = false;
    if (d >= -1 && d <= 1) {
      const unsigned long long k = key_of(i, c);
      less = k < s_cell[c].key;
      tie = k == s_cell[c].key;
    }
  };
  int less_n[kSegCells], tie_n[kSegCells];
#pragma unroll
  for (int c = 0; c < kSegCells; ++c) less_n[c] = tie_n[c] = 0;
  for (int base = k0; base < k1; base += 32) {
    const int i = base + lane < k1 ? sphere(base + lane) : -1;
    float yz, xl, xh;
    const bool live = i >= 0 && yz_step(i, yz) <= limit;
    if (!__any_sync(0xffffffffu, live)) continue;
    if (live) x_ends(i, xl, xh);
#pragma unroll
    for (int c = 0; c < kSegCells; ++c) {
      if (c >= nc) break;
      bool less = false, tie = false;
      if (live) classify(i, c, yz, xl, xh, less, tie);
      less_n[c] += __popc(__ballot_sync(0xffffffffu, less));
      tie_n[c] += __popc(__ballot_sync(0xffffffffu, tie));
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int c = 0; c < kSegCells; ++c) {
      s_less[warp][c] = less_n[c];
      s_tie[warp][c] = tie_n[c];
    }
  }
  __syncthreads();
  int at[kSegCells], ties[kSegCells];
#pragma unroll
  for (int c = 0; c < kSegCells; ++c) {
    at[c] = ties[c] = 0;
    if (c >= nc) continue;
    for (int w = 0; w < warp; ++w) {
      at[c] += s_less[w][c];
      ties[c] += s_tie[w][c];
    }
    at[c] += min(ties[c], s_cell[c].rank);
  }
  for (int base = k0; base < k1; base += 32) {
    const int i = base + lane < k1 ? sphere(base + lane) : -1;
    float yz, xl, xh;
    const bool live = i >= 0 && yz_step(i, yz) <= limit;
    if (!__any_sync(0xffffffffu, live)) continue;
    if (live) x_ends(i, xl, xh);
#pragma unroll
    for (int c = 0; c < kSegCells; ++c) {
      if (c >= nc) break;
      bool less = false, tie = false;
      if (live) classify(i, c, yz, xl, xh, less, tie);
      const unsigned tb = __ballot_sync(0xffffffffu, tie);
      const bool take = less || (tie && ties[c] + __popc(tb & lower) < s_cell[c].rank);
      ties[c] += __popc(tb);
      const unsigned kb = __ballot_sync(0xffffffffu, take);
      const int pos = at[c] + __popc(kb & lower);
      if (take && pos < K) out[size_t(c) * K + pos] = i;
      at[c] += __popc(kb);
    }
  }
}

// Fused-walk list entries, three passes: (1) each entry gets its structure id
// and, parked in .x, its sphere index; (2) each cell's entries are sorted by
// (structure id, sphere index) with a heapsort in place; (3) each entry gets
// its sphere record.  Sorted by structure id, a walker labelled L may stop at
// the first entry of a higher structure.
__global__ void gather_ids_kernel(const float* __restrict__ spheres, int S, const int* __restrict__ items, int n,
                                  float4* __restrict__ sph4, int* __restrict__ sid) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int s = items[k];
  sid[k] = int(spheres[4 * S + s]);
  sph4[k].x = __int_as_float(s);
}

__global__ void gather_sort_kernel(const int* __restrict__ start, const int* __restrict__ count, int ncell,
                                   float4* __restrict__ sph4, int* __restrict__ sid) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  const int base = start[c], n = count[c];
  auto key = [&](int i) {
    return (static_cast<unsigned long long>(static_cast<unsigned>(sid[base + i])) << 32) |
           static_cast<unsigned>(__float_as_int(sph4[base + i].x));
  };
  auto swap = [&](int i, int j) {
    const int t = sid[base + i];
    sid[base + i] = sid[base + j];
    sid[base + j] = t;
    const float u = sph4[base + i].x;
    sph4[base + i].x = sph4[base + j].x;
    sph4[base + j].x = u;
  };
  auto sift = [&](int root, int end) {
    while (2 * root + 1 < end) {
      int child = 2 * root + 1;
      if (child + 1 < end && key(child) < key(child + 1)) child++;
      if (key(root) < key(child)) {
        swap(root, child);
        root = child;
      } else {
        return;
      }
    }
  };
  for (int i = n / 2 - 1; i >= 0; --i) sift(i, n);
  for (int end = n - 1; end > 0; --end) {
    swap(0, end);
    sift(0, end);
  }
}

__global__ void gather_records_kernel(const float* __restrict__ spheres, int S, int n, float4* __restrict__ sph4) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int s = __float_as_int(sph4[k].x);
  sph4[k] = make_float4(spheres[s], spheres[S + s], spheres[2 * S + s], spheres[3 * S + s]);
}

// Index lists: each entry becomes its sphere's record index, then each
// cell's entries are sorted ascending (sort_lists).  Sphere order within the
// reference layout is usually already by structure, so the sort mostly finds
// its input in order.
template <typename T>
__global__ void index_fill_kernel(const int* __restrict__ items, int n, const int* __restrict__ perm,
                                  T* __restrict__ idx) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int s = items[k];
  idx[k] = T(perm ? perm[s] : s);
}

// Packed near entries (nz_cells_pack): the near filter of the fused walk in
// half precision, two spheres an instruction (near_bits_packed in
// walk_fused.cu).  An entry stores its sphere's centre relative to the cell's
// centre and the radius R of the ball the filter tests,
//   R = r (1 + 5e-5) + tol + 2 nm + E,  rounded up,
// with E a bound on the error of the filter's distance.  With u = 2^-11 (one
// rounding), rho = r + tol, M the near margin (distance of the walker from
// the cell plus reach <= M wherever the near lists are taken), h half the
// cell's diagonal and m = h + 2 M + rho >= the lengths of the walker's and
// the sphere's positions and of their difference d, for a sphere whose true
// distance from the segment is within its ball:
//   rounding of the two positions and of d              3 u m
//   of the segment's direction and length               2 u M
//   of d^2, d.e, s (s + 2 d.e) and their sum, at |d| <= rho + M,
//   as a distance                              u (2 rho + 7 M + 5.5 M^2 / rho)
//   of R + 2 % reach and its square                     2 u rho
// E is their sum and 15 % more (10 nm for r = 1 um, 0.5 um cells and margin).
// Spheres that half precision holds badly (R above 100 um, centres beyond
// 200 um) get R = inf: always near.  M is at most 100 um (kPackMargin), so a
// sphere in reach is within 200 um and d^2 below the largest half (255.9^2).
constexpr float kPackMargin = 100.0f;

__device__ __forceinline__ void pack_entry(float4 c, float ox, float oy, float oz, float h, float M, __half* v) {
  const float x = c.x - ox, y = c.y - oy, z = c.z - oz;  // single precision: its rounding is in the 15 %
  const float u = 1.0f / 2048, rho = c.w + kTol, m = h + 2 * M + rho;
  const float E = 1.15f * u * (3 * m + 9 * M + 4 * rho + 5.5f * M * M / rho);
  const float R = (c.w * 1.00005f + (kTol + 2e-3f) + E) * 1.000001f;
  const bool fits = R <= 100.0f && fabsf(x) <= 200.0f && fabsf(y) <= 200.0f && fabsf(z) <= 200.0f;
  v[0] = __float2half_rn(fits ? x : 0.0f);
  v[1] = __float2half_rn(fits ? y : 0.0f);
  v[2] = __float2half_rn(fits ? z : 0.0f);
  v[3] = fits ? __float2half_ru(R) : __ushort_as_half(0x7c00);
}

// Eight lanes a cell, a pair each, so that entries are read and pairs written
// by lines.
template <typename T>
__global__ void __launch_bounds__(256) cells_pack_kernel(const float4* __restrict__ rec4, const T* __restrict__ idx,
                                                         const int* __restrict__ start,
                                                         const int* __restrict__ count, Grid g, float h, float M,
                                                         uint4* __restrict__ pack) {
  const int nx = int(g.nLx), ny = int(g.nLy), ncell = nx * ny * int(g.nLz);
  const int c = int((blockIdx.x * size_t(blockDim.x) + threadIdx.x) >> 3), lane = threadIdx.x & 7;
  if (c >= ncell) return;
  const int n = count[c], s = start[c];
  // the cell's centre as the walk forms it (step_cell)
  const float ox = __fmaf_rn(float(c % nx), g.dLx, 0.5f * (g.dLx - g.Lx));
  const float oy = __fmaf_rn(float((c / nx) % ny), g.dLy, 0.5f * (g.dLy - g.Ly));
  const float oz = __fmaf_rn(float(c / (nx * ny)), g.dLz, 0.5f * (g.dLz - g.Lz));
  uint4* out = pack + ((s + c + 1) >> 1);
  for (int i = 2 * lane; i < n; i += 16) {
    __half a[4], b[4];
    pack_entry(__ldg(rec4 + int(idx[s + i])), ox, oy, oz, h, M, a);
    pack_entry(__ldg(rec4 + int(idx[s + min(i + 1, n - 1)])), ox, oy, oz, h, M, b);
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = uint32_t(__half_as_ushort(a[k])) | (uint32_t(__half_as_ushort(b[k])) << 16);
    out[i >> 1] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// Safe balls of the records (nz_cells_pack): a ball around a sphere's centre
// such that a walker of the sphere's structure whose segment stays in it
// takes its whole jump.  It lies 2 nm + 0.005 % of r inside the sphere (the
// fraction of the sphere itself is then at least the jump, by far more than
// the rounding of the reference's arithmetic) and as far, and 1 % of r more,
// outside the (r + tol) ball of every sphere of a lower structure (none of
// them contains the walker or stops it).  The walk uses them in iterations
// that stay within the near margin of the walker's cell, so a point where a
// lower sphere meets this one lies within that margin of the box, and the
// near list of the cell that the point falls in or is clamped to holds the
// lower sphere: the lists of the cells that this sphere meets hold them all.
// A warp per record; the squared radius is stored, -1 for none.  80,000
// records on 0.67 um cells take 0.37 ms, 0.56 ms over the full lists of every
// cell of the sphere's box.
template <typename T>
__global__ void __launch_bounds__(256) cells_safe_kernel(const float4* __restrict__ rec4,
                                                         const int* __restrict__ rec_sid, int S,
                                                         const T* __restrict__ idx, const int* __restrict__ start,
                                                         const int* __restrict__ count, Grid g,
                                                         float* __restrict__ safe) {
  const int k = int((blockIdx.x * size_t(blockDim.x) + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (k >= S) return;
  const float4 c = __ldg(rec4 + k);
  const int sid = __ldg(rec_sid + k);
  float best = c.w * 0.99995f - 2e-3f;
  const float reach = c.w * 1.001f + 0.01f;
  const int nx = int(g.nLx), ny = int(g.nLy);
  auto cell = [](float x, float L, float d, float n) {
    return int(fminf(n - 1, fmaxf(0.f, floorf((x + L / 2) / d))));
  };
  const int x0 = cell(c.x - reach, g.Lx, g.dLx, g.nLx), x1 = cell(c.x + reach, g.Lx, g.dLx, g.nLx);
  const int y0 = cell(c.y - reach, g.Ly, g.dLy, g.nLy), y1 = cell(c.y + reach, g.Ly, g.dLy, g.nLy);
  const int z0 = cell(c.z - reach, g.Lz, g.dLz, g.nLz), z1 = cell(c.z + reach, g.Lz, g.dLz, g.nLz);
  // distance of the centre from cell n of an axis; a boundary cell stands for
  // all beyond it
  auto gap = [](float x, int n, float L, float d, int last) {
    const float lo = n == 0 ? -1e30f : n * d - L / 2, hi = n == last ? 1e30f : (n + 1) * d - L / 2;
    return fmaxf(0.f, fmaxf(lo - x, x - hi));
  };
  for (int p = z0; p <= z1; ++p)
    for (int m = y0; m <= y1; ++m) {
      const float ez = gap(c.z, p, g.Lz, g.dLz, int(g.nLz) - 1), ey = gap(c.y, m, g.Ly, g.dLy, ny - 1);
      for (int n = x0; n <= x1; ++n) {
        const float ex = gap(c.x, n, g.Lx, g.dLx, nx - 1);
        if (ex * ex + ey * ey + ez * ez > reach * reach) continue;
        const int q = (p * ny + m) * nx + n;
        const int s = start[q], e = s + count[q];
        for (int i = s + lane; i < e; i += 32) {
          const int o = int(idx[i]);
          if (o >= k || __ldg(rec_sid + o) >= sid) continue;  // records are in order of structures
          const float4 d = __ldg(rec4 + o);
          const float fx = d.x - c.x, fy = d.y - c.y, fz = d.z - c.z;
          const float apart = sqrtf(fx * fx + fy * fy + fz * fz) * 0.99999f - d.w * 1.00005f;
          best = fminf(best, apart - 2e-3f - kTol - 0.01f * c.w);
        }
      }
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = fminf(best, __shfl_xor_sync(0xffffffffu, best, o));
  if (lane == 0) safe[k] = best > 0.0f ? best * best : -1.0f;
}

// Exclusive scan of in[lo, hi) into out[lo, hi) by one CTA (1024 threads, 8
// items per thread per pass), starting from carry; returns the range's total
// (in every thread).
__device__ __forceinline__ int block_scan_range(const int* __restrict__ in, int* __restrict__ out, int lo, int hi,
                                                int carry) {
  constexpr int kItems = 8;
  __shared__ int s_warp[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int base = lo; base < hi; base += 1024 * kItems) {
    int v[kItems];
    int sum = 0;
    const int first = base + threadIdx.x * kItems;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      v[j] = (first + j < hi) ? in[first + j] : 0;
      sum += v[j];
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    if (wid == 0) {
      int t = s_warp[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += y;
      }
      s_warp[lane] = t;
    }
    __syncthreads();
    int run = carry + (wid > 0 ? s_warp[wid - 1] : 0) + x - sum;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      if (first + j < hi) out[first + j] = run;
      run += v[j];
    }
    carry += s_warp[31];
    __syncthreads();
  }
  return carry;
}

// Single-CTA exclusive scan of n ints.
__global__ void __launch_bounds__(1024) scan_kernel(const int* __restrict__ in, int* __restrict__ out, int n,
                                                    int* __restrict__ total) {
  const int t = block_scan_range(in, out, 0, n, 0);
  if (threadIdx.x == 0 && total) *total = t;
}

// Multi-CTA form for long arrays: each CTA sums one tile, one CTA scans the
// tile sums, each CTA then scans its tile from its offset.
__global__ void __launch_bounds__(1024) tile_sum_kernel(const int* __restrict__ in, int n, int* __restrict__ sums) {
  __shared__ int s_red[32];
  const int lo = blockIdx.x * kScanTile, hi = min(n, lo + kScanTile);
  int v = 0;
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) v += in[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = s_red[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) sums[blockIdx.x] = v;
  }
}

__global__ void __launch_bounds__(1024) tile_scan_kernel(const int* __restrict__ in, int* __restrict__ out, int n,
                                                         const int* __restrict__ offsets) {
  const int lo = blockIdx.x * kScanTile, hi = min(n, lo + kScanTile);
  block_scan_range(in, out, lo, hi, offsets[blockIdx.x]);
}

// Multi-CTA scan without scratch (nz_exclusive_scan_i32): each CTA scans its
// tile from 0; one CTA scans the tiles' totals (a tile's last prefix plus its
// last value) and leaves each tile's offset in the tile's first element,
// whose own prefix is 0; each CTA adds its offset to the rest of its tile.
__global__ void __launch_bounds__(1024) tile_local_scan_kernel(const int* __restrict__ in, int* __restrict__ out,
                                                               int n) {
  const int lo = blockIdx.x * kScanTile, hi = min(n, lo + kScanTile);
  block_scan_range(in, out, lo, hi, 0);
}

__global__ void __launch_bounds__(1024) tile_offsets_kernel(const int* __restrict__ in, int* out, int n,
                                                            int* __restrict__ total) {
  __shared__ int s_warp[32];
  const int tiles = (n + kScanTile - 1) / kScanTile;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int carry = 0;
  for (int base = 0; base < tiles; base += 1024) {
    const int i = base + threadIdx.x;
    const int last = min(n, (i + 1) * kScanTile) - 1;
    const int v = i < tiles ? out[last] + in[last] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    int before = carry, all = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < wid) before += s_warp[w];
      all += s_warp[w];
    }
    // a tile of one element: its offset replaces the prefix just read
    if (i < tiles) out[size_t(i) * kScanTile] = before + x - v;
    carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void __launch_bounds__(1024) tile_add_kernel(int* __restrict__ out, int n) {
  const int lo = blockIdx.x * kScanTile, hi = min(n, lo + kScanTile);
  const int offset = out[lo];
  for (int i = lo + 1 + threadIdx.x; i < hi; i += blockDim.x) out[i] += offset;
}

int scan_tiles(int n) { return (n + kScanTile - 1) / kScanTile; }

int exclusive_scan(const int* in, int* out, int n, int* tile_sums, int* tile_offsets, cudaStream_t st) {
  if (n <= kScanSingle || !tile_sums || !tile_offsets) {
    scan_kernel<<<1, 1024, 0, st>>>(in, out, n, nullptr);
    return check_launch("scan_kernel");
  }
  const int tiles = scan_tiles(n);
  tile_sum_kernel<<<tiles, 1024, 0, st>>>(in, n, tile_sums);
  int rc = check_launch("tile_sum_kernel");
  if (rc) return rc;
  scan_kernel<<<1, 1024, 0, st>>>(tile_sums, tile_offsets, tiles, nullptr);
  rc = check_launch("scan_kernel");
  if (rc) return rc;
  tile_scan_kernel<<<tiles, 1024, 0, st>>>(in, out, n, tile_offsets);
  return check_launch("tile_scan_kernel");
}

}  // namespace nz

using namespace nz;

extern "C" int nz_cells_count(const double* spheres64, int S, double Lx, double Ly, double Lz, int nx, int ny, int nz_,
                              double jump_tol, int* counts, void* stream) {
  if (S < 0 || nx <= 0 || ny <= 0 || nz_ <= 0 || !counts || (S > 0 && !spheres64))
    return set_error(NZ_ERR_ARG, "nz_cells_count: bad arguments (S=%d grid=%dx%dx%d)", S, nx, ny, nz_);
  const size_t ncell = size_t(nx) * ny * nz_;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(counts, 0, ncell * sizeof(int), st) != cudaSuccess) return check_launch("nz_cells_count memset");
  if (S == 0) return NZ_OK;
  CellGeom g{Lx, Ly, Lz, nx, ny, nz_, jump_tol};
  return cells_members<false>(spheres64, S, g, nullptr, counts, nullptr, st);
}

extern "C" int nz_cells_count_round(const double* spheres64, int S, double Lx, double Ly, double Lz, int nx, int ny,
                                    int nz_, double margin, int* counts, void* stream) {
  if (S < 0 || nx <= 0 || ny <= 0 || nz_ <= 0 || !counts || (S > 0 && !spheres64) || !(margin >= 0.0))
    return set_error(NZ_ERR_ARG, "nz_cells_count_round: bad arguments (S=%d grid=%dx%dx%d)", S, nx, ny, nz_);
  const size_t ncell = size_t(nx) * ny * nz_;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(counts, 0, ncell * sizeof(int), st) != cudaSuccess)
    return check_launch("nz_cells_count_round memset");
  if (S == 0) return NZ_OK;
  CellGeom g{Lx, Ly, Lz, nx, ny, nz_, margin};
  return cells_members<true>(spheres64, S, g, nullptr, counts, nullptr, st);
}

extern "C" int nz_cells_fill_round(const double* spheres64, int S, double Lx, double Ly, double Lz, int nx, int ny,
                                   int nz_, double margin, const int* offsets, const int* counts, int* cursor,
                                   int* items, void* stream) {
  if (S < 0 || nx <= 0 || ny <= 0 || nz_ <= 0 || !offsets || !counts || !cursor || (S > 0 && !spheres64) ||
      !(margin >= 0.0))
    return set_error(NZ_ERR_ARG, "nz_cells_fill_round: bad arguments (S=%d grid=%dx%dx%d)", S, nx, ny, nz_);
  const size_t ncell = size_t(nx) * ny * nz_;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(cursor, 0, ncell * sizeof(int), st) != cudaSuccess)
    return check_launch("nz_cells_fill_round memset");
  if (S == 0) return NZ_OK;
  CellGeom g{Lx, Ly, Lz, nx, ny, nz_, margin};
  int rc = cells_members<true>(spheres64, S, g, offsets, cursor, items, st);
  if (rc != NZ_OK) return rc;
  return sort_lists(offsets, counts, int(ncell), S, items, st);
}

extern "C" int nz_exclusive_scan_i32(const int* in, int* out, int n, int* total, void* stream) {
  if (n < 0 || n > (1 << 26) || (n > 0 && (!in || !out)))
    return set_error(NZ_ERR_ARG, "nz_exclusive_scan_i32: bad arguments (n=%d)", n);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // one CTA for short arrays (and in place or overlapping, where values that
  // the tiles still need would be gone): 20,000 counts take it 21 us, the
  // tiles' three launches 23; 65,536 52 and 23
  const uintptr_t i0 = reinterpret_cast<uintptr_t>(in), o0 = reinterpret_cast<uintptr_t>(out);
  const bool overlap = i0 < o0 + size_t(n) * sizeof(int) && o0 < i0 + size_t(n) * sizeof(int);
  if (n <= 5 * kScanTile / 2 || overlap) {
    scan_kernel<<<1, 1024, 0, st>>>(in, out, n, total);
    return check_launch("scan_kernel");
  }
  const int tiles = scan_tiles(n);
  tile_local_scan_kernel<<<tiles, 1024, 0, st>>>(in, out, n);
  int rc = check_launch("tile_local_scan_kernel");
  if (rc) return rc;
  tile_offsets_kernel<<<1, 1024, 0, st>>>(in, out, n, total);
  rc = check_launch("tile_offsets_kernel");
  if (rc) return rc;
  tile_add_kernel<<<tiles, 1024, 0, st>>>(out, n);
  return check_launch("tile_add_kernel");
}

extern "C" int nz_cells_fill(const double* spheres64, int S, double Lx, double Ly, double Lz, int nx, int ny, int nz_,
                             double jump_tol, const int* offsets, const int* counts, int* cursor, int* items,
                             void* stream) {
  if (S < 0 || nx <= 0 || ny <= 0 || nz_ <= 0 || !offsets || !counts || !cursor || (S > 0 && !spheres64))
    return set_error(NZ_ERR_ARG, "nz_cells_fill: bad arguments (S=%d grid=%dx%dx%d)", S, nx, ny, nz_);
  const size_t ncell = size_t(nx) * ny * nz_;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(cursor, 0, ncell * sizeof(int), st) != cudaSuccess) return check_launch("nz_cells_fill memset");
  if (S == 0) return NZ_OK;
  CellGeom g{Lx, Ly, Lz, nx, ny, nz_, jump_tol};
  int rc = cells_members<false>(spheres64, S, g, offsets, cursor, items, st);
  if (rc != NZ_OK) return rc;
  return sort_lists(offsets, counts, int(ncell), S, items, st);
}

extern "C" int nz_segments_fill(const double* spheres64, int S, double Lx, double Ly, double Lz, int nx, int ny,
                                int nz_, int K, int* segments, void* stream) {
  if (S <= 0 || nx <= 0 || ny <= 0 || nz_ <= 0 || K <= 0 || K > S || !spheres64 || !segments)
    return set_error(NZ_ERR_ARG, "nz_segments_fill: bad arguments (S=%d K=%d)", S, K);
  const size_t ncell = size_t(nx) * ny * nz_;
  if (ncell > 0x7fffffffu) return set_error(NZ_ERR_ARG, "nz_segments_fill: too many cells");
  CellGeom g{Lx, Ly, Lz, nx, ny, nz_, 0.0};
  // cells of a row a CTA: as many as leave the GPU full
  int per = kSegCells;
  while (per > 1 && 1ll * ny * nz_ * ((nx + per - 1) / per) < 2 * 148) per /= 2;
  const unsigned ctas = unsigned(size_t(ny) * nz_ * ((nx + per - 1) / per));
  const size_t bytes = kSegKept * sizeof(int) + (S <= kSegBitmap ? size_t((S + 31) / 32) * sizeof(unsigned) : 0);
  if (cudaFuncSetAttribute(segments_fill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kSegKept * int(sizeof(int)) + kSegBitmap / 8) != cudaSuccess)
    return check_launch("segments_fill_kernel attribute");
  segments_fill_kernel<<<ctas, 256, bytes, static_cast<cudaStream_t>(stream)>>>(spheres64, S, g, K, per, segments);
  return check_launch("segments_fill_kernel");
}

extern "C" int nz_cells_gather(const float* spheres, int S, const int* items, int n_items, const int* cell_start,
                               const int* cell_count, int ncell, float* sph4, int* sid, void* stream) {
  if (S < 0 || n_items < 0 || ncell < 0 ||
      (n_items > 0 && (!spheres || !items || !sph4 || !sid || !cell_start || !cell_count)))
    return set_error(NZ_ERR_ARG, "nz_cells_gather: bad arguments");
  if (reinterpret_cast<uintptr_t>(sph4) % 16 != 0) return set_error(NZ_ERR_ARG, "nz_cells_gather: sph4 not 16-byte aligned");
  if (n_items == 0) return NZ_OK;
  if (ncell == 0) return set_error(NZ_ERR_ARG, "nz_cells_gather: %d items but no cells", n_items);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float4* s4 = reinterpret_cast<float4*>(sph4);
  gather_ids_kernel<<<(n_items + 255) / 256, 256, 0, st>>>(spheres, S, items, n_items, s4, sid);
  int rc = check_launch("gather_ids_kernel");
  if (rc) return rc;
  gather_sort_kernel<<<(ncell + 127) / 128, 128, 0, st>>>(cell_start, cell_count, ncell, s4, sid);
  rc = check_launch("gather_sort_kernel");
  if (rc) return rc;
  gather_records_kernel<<<(n_items + 255) / 256, 256, 0, st>>>(spheres, S, n_items, s4);
  return check_launch("gather_records_kernel");
}

extern "C" int nz_cells_index(const int* items, int n_items, const int* perm, int S, const int* cell_start,
                              const int* cell_count, int ncell, void* idx, int idx_bytes, void* stream) {
  if (n_items < 0 || ncell < 0 || S < 0 || (idx_bytes != 2 && idx_bytes != 4) ||
      (n_items > 0 && (!items || !idx || !cell_start || !cell_count || ncell == 0)))
    return set_error(NZ_ERR_ARG, "nz_cells_index: bad arguments (items=%d cells=%d idx_bytes=%d)", n_items, ncell,
                     idx_bytes);
  if (idx_bytes == 2 && S > 65536)
    return set_error(NZ_ERR_ARG, "nz_cells_index: %d spheres do not fit 16-bit indices", S);
  if (n_items == 0) return NZ_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (idx_bytes == 2) {
    auto* p = static_cast<uint16_t*>(idx);
    index_fill_kernel<uint16_t><<<(n_items + 255) / 256, 256, 0, st>>>(items, n_items, perm, p);
    int rc = check_launch("index_fill_kernel");
    if (rc) return rc;
    return sort_lists(cell_start, cell_count, ncell, S, p, st);
  } else {
    auto* p = static_cast<int*>(idx);
    index_fill_kernel<int><<<(n_items + 255) / 256, 256, 0, st>>>(items, n_items, perm, p);
    int rc = check_launch("index_fill_kernel");
    if (rc) return rc;
    return sort_lists(cell_start, cell_count, ncell, S, p, st);
  }
}

extern "C" size_t nz_cells_pack_bytes(int n_items, int ncell, int S) {
  if (n_items < 0 || ncell < 0 || S < 0) return 0;
  return (pack_radii(S) + pack_pairs(n_items, ncell)) * 16;
}

extern "C" int nz_cells_pack(const float* rec4, const int* rec_sid, int S, const void* idx, int idx_bytes,
                             const int* start, const int* count, int n_items, const nz_grid* grid, float margin,
                             void* pack, void* stream) {
  int rc = check_grid(grid, "nz_cells_pack");
  if (rc) return rc;
  if (S < 0 || n_items < 0 || (idx_bytes != 2 && idx_bytes != 4) || !(margin > 0.0f) || !pack ||
      (reinterpret_cast<uintptr_t>(pack) & 15) || !start || !count || (S > 0 && (!rec4 || !rec_sid)) ||
      (n_items > 0 && !idx) ||
      (reinterpret_cast<uintptr_t>(rec4) & 15))
    return set_error(NZ_ERR_ARG, "nz_cells_pack: bad arguments (S=%d items=%d idx_bytes=%d)", S, n_items, idx_bytes);
  if (!(grid->dLx <= 1e4f && grid->dLy <= 1e4f && grid->dLz <= 1e4f))
    return set_error(NZ_ERR_ARG, "nz_cells_pack: cell edges above 1e4 um");
  if (!(margin <= kPackMargin)) return set_error(NZ_ERR_ARG, "nz_cells_pack: margin above 100 um");
  const long long ncell = 1ll * grid->nx * grid->ny * grid->nz;
  if (ncell + n_items > 0x7fffffffll) return set_error(NZ_ERR_ARG, "nz_cells_pack: too many cells and entries");
  const Grid g{grid->Lx, grid->Ly, grid->Lz, grid->dLx, grid->dLy, grid->dLz, float(grid->nx), float(grid->ny),
               float(grid->nz)};
  const float h = float(0.5 * sqrt(double(g.dLx) * g.dLx + double(g.dLy) * g.dLy + double(g.dLz) * g.dLz));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned blocks = unsigned((8 * ncell + 255) / 256);
  const float4* r = reinterpret_cast<const float4*>(rec4);
  float* safe = static_cast<float*>(pack);
  uint4* out = static_cast<uint4*>(pack) + pack_radii(S);
  const unsigned sblocks = unsigned((size_t(S) * 32 + 255) / 256);
  if (idx_bytes == 2)
    cells_pack_kernel<<<blocks, 256, 0, st>>>(r, static_cast<const uint16_t*>(idx), start, count, g, h, margin, out);
  else
    cells_pack_kernel<<<blocks, 256, 0, st>>>(r, static_cast<const int*>(idx), start, count, g, h, margin, out);
  rc = check_launch("cells_pack_kernel");
  if (rc || S == 0) return rc;
  if (idx_bytes == 2)
    cells_safe_kernel<<<sblocks, 256, 0, st>>>(r, rec_sid, S, static_cast<const uint16_t*>(idx), start, count, g, safe);
  else
    cells_safe_kernel<<<sblocks, 256, 0, st>>>(r, rec_sid, S, static_cast<const int*>(idx), start, count, g, safe);
  return check_launch("cells_safe_kernel");
}
