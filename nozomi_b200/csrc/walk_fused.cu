// Fused walk: many time steps per launch, walker state in registers.
//
// The collision rule is the reference's, unchanged
// (simulation_toolkit/simulation_engine/sim3d_kernel.cu:758-874): label, first
// draw, collision pass over the cell's spheres, advance, scatter or continue.
// What changes is how the work is organised:
//
//  * one thread per walker runs a whole range of steps; each lane moves to its
//    next step as soon as its current one ends, so lanes of a warp do not wait
//    for each other's extra collision iterations at every step;
//  * the reference's two passes over the cell list (label, then collisions)
//    are one pass under the label carried from the previous iteration; the
//    pass proves that label (some containing sphere of that structure, none of
//    a lower one) or the iteration is redone with the recomputed label, so the
//    result is the reference's;
//  * the near lists (the same cell grid with a smaller margin) serve every
//    iteration whose reach fits their margin, the full lists the rest;
//  * list entries are record indices (or, in record lists, carry their
//    sphere's record and structure id inline);
//  * packed near lists (nz_cells_pack) are walked by warps (walk_warp).  A
//    walker whose segment stays in the safe ball of the sphere that held it
//    last takes its whole jump and scans nothing: three of four iterations of
//    walkers inside axons.  The others scan their list in two passes: the
//    first marks the near spheres, those whose (r + tol) ball comes within
//    2 nm and 2 % of the reach of the segment ahead, from the packed entries
//    in half precision, two spheres an instruction; any other sphere neither
//    contains the walker nor can lower the jump fraction.  The second runs
//    the reference's inside test and the fractions for the marked ones only.
//    Full lists are scanned by the whole warp together;
//  * all other lists are walked by each lane on its own (walk_one), the near
//    spheres marked by their distance from the walker against the reach;
//  * each iteration has one draw site (the scatter draw of this step or the
//    first draw of the next), and the inside and outside fractions share one
//    instruction stream (step_either; with one division, step_one, in
//    walk_warp);
//  * phase is accrued as the 3-vector Phi = sum_n G_n p_n with Kahan
//    compensation, the wrap correction on the wrapped axis only; every
//    direction's phase is u_d . Phi (the reference's per-direction sums
//    regrouped; identical in exact arithmetic);
//  * draws are counter-based (Philox at walker, step, draw), so a walker's
//    trajectory does not depend on which thread, CTA or launch runs it.
#include <algorithm>
#include <cstdint>
#include <cuda_fp16.h>
#include <mutex>
#include "kernels.cuh"

namespace nz {

struct ScanOut {
  float fin, fout;
  bool any_in;
};

// Dynamic shared memory: the records of a job (staged batched walk only),
// then, in walk_warp's phase modes, each thread's walker's Phi with its compensation
// (a float4 per thread: Phi, compensation x; then a float2 per thread:
// compensation y, z), in its other modes its origin and id (a float4 per
// thread; the origin in the moment modes only).  They are touched once a step
// or draw and would hold registers through the collision pass.
extern __shared__ __align__(16) float4 s_stage[];
template <int MODE>
constexpr size_t phi_bytes(int threads) {
  return size_t(threads) * ((MODE & NZ_MODE_PHI) ? 24 : 16);
}

// Record `key` of the substrate's record array (SH: the staged copy).  In
// the bounds-checked build an index outside [0, S) sets oob and reads
// nothing: the entry becomes a NaN record that is neither near nor
// containing, with a key that stops nothing.
template <bool SH>
__device__ __forceinline__ float4 record(const float4* __restrict__ rec, int S, int& key, int& oob) {
  if (kCheckBounds && (key < 0 || key >= S)) {
    oob = 1;
    key = -1;
    return make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
  }
  if constexpr (SH) return s_stage[key];  // SH: the job's records were copied there
  return __ldg(rec + key);
}

// One list entry: its sphere's record and a key.  Record lists (LK 0): the
// record inline, the key the structure id.  Index lists (LK 2 or 4): the key
// the record index, the record read from the substrate's record array.  The
// entries of a cell ascend by key.  In either form the entries of structure
// L have keys in [lo, hi) (label_bounds): key < hi is "structure <= L" and
// key < lo "structure < L"; for a walker in the box every key is below lo
// (box: record lists then need none).
template <int LK, bool SH>
__device__ __forceinline__ void entry(const void* __restrict__ list, const float4* __restrict__ rec,
                                      const int* __restrict__ sid, int k, int S, int& oob, int& key, float4& c,
                                      bool box = false) {
  if constexpr (LK == 0) {
    key = box ? -1 : __ldg(sid + k);
    c = __ldg(rec + k);
  } else {
    if constexpr (LK == 2) key = int(__ldg(static_cast<const unsigned short*>(list) + k));
    else key = __ldg(static_cast<const int*>(list) + k);
    c = record<SH>(rec, S, key, oob);
  }
}

// This iteration's reach |j| * jump_remaining, from the hardware reciprocal
// square root: within a few ulp of sqrtf, far inside the 2 % + 2 nm of slack
// of the only two uses (the near test and the first-pass filter), which
// decide what is scanned, never a result.
__device__ __forceinline__ float reach_of(float a, float jr) { return a * rsqrtf(fmaxf(a, 1e-30f)) * jr; }

// Jumps below this squared length (1e-4 um; none at all where D is 0) are too
// short for the filters' arithmetic, which mark every entry then.  beyond
// passes over the spheres that the segment cannot come near, with the filter
// of scan_cell: with no jump at all the quadratic has no roots, and the
// fraction of an outside sphere would be 0 at any distance.
constexpr float kTinyJump2 = 1e-8f;
__device__ __forceinline__ bool beyond(float dx, float dy, float dz, float r, float a, float jr) {
  if (a >= kTinyJump2) return false;
  const float ro = r + (kTol + reach_of(a, jr) * 1.02f + 2e-3f);
  return !(__fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz)) <= ro * ro);
}

// The reference's collision pass over one cell's list for one walker of
// known label (sim3d_kernel.cu:800-830), lane by lane: only for the rare
// iteration whose label had to be corrected.
template <int LK, bool T64, bool SH>
__device__ __noinline__ void scan_lane(const void* __restrict__ list, const float4* __restrict__ rec,
                                       int start, int count, int lo, int hi, float x, float y, float z, float a,
                                       float jx, float jy, float jz, float jr, int S, int& oob, ScanOut& o) {
  o.fin = 0.0f;
  o.fout = kBig;
  o.any_in = false;
  for (int i = 0; i < count; ++i) {
    int key;
    float4 c;
    entry<LK, SH>(list, rec, nullptr, start + i, S, oob, key, c);
    if (key >= hi) break;
    const float dx = x - c.x, dy = y - c.y, dz = z - c.z;
    if (beyond(dx, dy, dz, c.w, a, jr)) continue;
    const bool inside = dx * dx + dy * dy + dz * dz - c.w * c.w < 0;
    if (inside || key < lo) {
      const float f = step_either_t<T64>(inside, dx, dy, dz, c.w, a, jx, jy, jz);
      if (inside) {
        o.any_in = true;
        if (o.fin < f) o.fin = f;
      } else if (f < o.fout) {
        o.fout = f;
      }
    }
  }
}

// The near filter's view of one walker's iteration.
struct Reach {
  float mx, my, mz, m2;  // twice the displacement left in this step; the displacement's squared length
  float k;               // -1/2 over that square
  float slack;
};

// Whether a sphere's (r + tol) ball, grown by 2 nm, 0.005 % of r and 2 % of
// the reach (or by `slack`), meets the segment that the walker would walk in
// this iteration.  A sphere farther from the whole segment neither contains
// the walker nor can stop it: its root lies beyond the segment's end, or the
// ray misses it, by far more than the rounding of the reference's
// arithmetic.  A filter, not the reference's arithmetic: fused multiply-adds
// are fine here.
__device__ __forceinline__ bool is_near(const Reach& g, float x, float y, float z, float4 c) {
  const float dx = x - c.x, dy = y - c.y, dz = z - c.z;
  const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
  const float dm = __fmaf_rn(dx, g.mx, __fmaf_rn(dy, g.my, dz * g.mz));
  const float t = __saturatef(dm * g.k);  // the segment's nearest point to the centre
  const float ro = __fmaf_rn(c.w, 1.00005f, g.slack);
  return __fmaf_rn(t, __fmaf_rn(t, g.m2, dm), d2) <= ro * ro;
}

// Near masks cover 32 list entries: entry i at bit (i >> 1) | (i & 1) << 4.
__device__ __forceinline__ int bit_entry(int bit) { return 2 * (bit & 15) + (bit >> 4); }

// Near mask of up to 16 pairs of packed near entries (nz_cells_pack), two
// entries an instruction in half precision: px.. the position relative to
// the cell's centre, ex.. the segment's direction, len its length, grow 2 %
// of it.  The entries' radii hold the rounding of these distances.
// Structures are not told apart here; entries past n are cut by the caller.
__device__ __forceinline__ uint32_t near_bits_packed(const uint4* __restrict__ pk, int pairs, __half2 px, __half2 py,
                                                     __half2 pz, __half2 ex, __half2 ey, __half2 ez, __half2 len,
                                                     __half2 grow) {
  uint32_t bits = 0u;
  const __half2 zero = __float2half2_rn(0.0f), two = __float2half2_rn(2.0f);
  auto test = [&](uint4 v) {
    const __half2 dx = __hsub2(px, *reinterpret_cast<const __half2*>(&v.x));
    const __half2 dy = __hsub2(py, *reinterpret_cast<const __half2*>(&v.y));
    const __half2 dz = __hsub2(pz, *reinterpret_cast<const __half2*>(&v.z));
    const __half2 d2 = __hfma2(dx, dx, __hfma2(dy, dy, __hmul2(dz, dz)));
    const __half2 de = __hfma2(dx, ex, __hfma2(dy, ey, __hmul2(dz, ez)));
    const __half2 t = __hmin2(__hmax2(__hneg2(de), zero), len);  // the segment's nearest point to the centre
    const __half2 near2 = __hfma2(t, __hfma2(de, two, t), d2);
    const __half2 ro = __hadd2(*reinterpret_cast<const __half2*>(&v.w), grow);
    return __hle2_mask(near2, __hmul2(ro, ro));
  };
  for (int i = 0; i < pairs; i += 2) {  // may read one pair past the list: nz_cells_pack_bytes leaves room
    const uint4 a = __ldg(pk + i), b = __ldg(pk + i + 1);
    bits |= test(a) & (0x00010001u << i);
    bits |= test(b) & (0x00020002u << i);
  }
  return bits;
}

// The marked entries that a jump below kTinyJump2 can come near, out of line.
template <int LK, bool SH>
__device__ __noinline__ uint32_t close_bits(uint32_t bits, const void* __restrict__ list,
                                            const float4* __restrict__ rec, int first, float x, float y, float z,
                                            float a, float jr, int S, int& oob) {
  uint32_t keep = 0u;
  while (bits) {
    const int bit = __ffs(bits) - 1;
    bits &= bits - 1u;
    int key;
    float4 c;
    entry<LK, SH>(list, rec, nullptr, first + bit_entry(bit), S, oob, key, c);
    if (!beyond(x - c.x, y - c.y, z - c.z, c.w, a, jr)) keep |= 1u << bit;
  }
  return keep;
}

// Fractions of the marked entries of one walker (bits, as near_bits marks
// them, of the entries from list position `first` on): the reference's inside
// test, then the fraction of a containing sphere or of a lower structure's
// sphere.  within: the containing sphere with the largest fraction.  lower:
// a sphere of a lower structure contains the walker.
template <int LK, bool T64, bool SH>
__device__ __forceinline__ void fractions(uint32_t bits, const void* __restrict__ list,
                                          const float4* __restrict__ rec, int first, int lo, int hi, float x, float y,
                                          float z, float a, float jx, float jy, float jz, int S, int& oob, ScanOut& o,
                                          bool& lower, int& within) {
  while (bits) {
    const int i = bit_entry(__ffs(bits) - 1);
    bits &= bits - 1u;
    int key;
    float4 c;
    entry<LK, SH>(list, rec, nullptr, first + i, S, oob, key, c);
    if (key >= hi) continue;
    const bool below = key < lo;
    const float dx = x - c.x, dy = y - c.y, dz = z - c.z;
    const float d2 = dx * dx + dy * dy + dz * dz;
    const bool inside = d2 - c.w * c.w < 0;
    if (inside || below) {
      lower |= inside && below;
      const float f = T64 ? step_either_t<T64>(inside, dx, dy, dz, c.w, a, jx, jy, jz)
                          : step_one(inside, dx, dy, dz, d2, c.w, a, jx, jy, jz);
      if (inside) {
        if (!o.any_in || o.fin < f) within = key;
        o.any_in = true;
        if (o.fin < f) o.fin = f;
      } else if (f < o.fout) {
        o.fout = f;
      }
    }
  }
}

// Lists without packed entries, each lane by itself: one pass over a cell's
// list under assumed label L.  Returns false when the
// walker's label is not L (then nothing in `o` is used).  Ends at the first
// entry of a structure above L (the reference skips those spheres, :805-806).
// BOX: walkers in the box read no structure ids.
template <int LK, bool T64, bool SH, bool BOX>
__device__ __forceinline__ bool scan_cell(const void* __restrict__ list, const float4* __restrict__ rec,
                                          const int* __restrict__ sid, int start, int count, int nstructures,
                                          int lo, int hi, float x, float y, float z, int L, float a, float jx,
                                          float jy, float jz, float reach, int S, int& oob, ScanOut& o) {
  o.fin = 0.0f;
  o.fout = kBig;
  o.any_in = false;
  bool found = false, lower = false, stop = false;
  const float slack = kTol + reach * 1.02f + 2e-3f;
  const bool box = BOX && L >= nstructures;
  constexpr int kUnroll = 4;
  for (int base = 0; base < count && !stop; base += 32) {
    const int m = min(32, count - base);
    // first pass: which entries are near, i.e. within (r + slack), a slack of
    // at least 2.1 nm that dwarfs the rounding of d2 and r*r, so that a far
    // sphere neither contains the walker nor lies within this iteration's
    // reach; predicated, one entry per load
    // kUnroll entries are loaded together, so that their loads (two
    // dependent ones each in index form) are in flight at once; entries past
    // the first of a higher structure are invalid too (keys ascend), so a
    // batch never marks one near
    uint32_t near_mask = 0u;
    for (int i0 = 0; i0 < m && !stop; i0 += kUnroll) {
      int key[kUnroll];
      float4 c[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        if (i0 + u < m) {
          entry<LK, SH>(list, rec, sid, start + base + i0 + u, S, oob, key[u], c[u], box);
        } else {  // past the chunk: a NaN record, never near, stops nothing
          key[u] = -1;
          c[u] = make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const bool valid = key[u] < hi;
        stop |= !valid;
        const float dx = x - c[u].x, dy = y - c[u].y, dz = z - c[u].z;
        // a filter, not the reference's arithmetic: fused multiply-adds are
        // fine here (their rounding is far inside the slack)
        const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
        const float t = c[u].w + slack;
        near_mask |= (valid && d2 <= t * t) ? (1u << (i0 + u)) : 0u;
      }
    }
    // second pass, near entries only: the reference's inside test, then the
    // fraction of a containing sphere or of a lower structure's sphere
    while (near_mask) {
      const int i = __ffs(near_mask) - 1;
      near_mask &= near_mask - 1;
      int key;
      float4 c;
      entry<LK, SH>(list, rec, sid, start + base + i, S, oob, key, c, box);
      const bool below = key < lo;
      const float dx = x - c.x, dy = y - c.y, dz = z - c.z;
      const float d2 = dx * dx + dy * dy + dz * dz;
      const bool inside = d2 - c.w * c.w < 0;
      lower |= inside && below;
      found |= inside && !below;
      if (inside || below) {
        const float f = step_either_t<T64>(inside, dx, dy, dz, c.w, a, jx, jy, jz);
        if (inside) {
          o.any_in = true;
          if (o.fin < f) o.fin = f;
        } else if (f < o.fout) {
          o.fout = f;
        }
      }
    }
  }
  return !(lower || (L < nstructures && !found));
}

// The reference's label pass (sim3d_kernel.cu:766-785): lowest structure id
// among the spheres containing the walker, nstructures if none.  In index
// form the entries ascend by structure, so the first containing one decides.
template <int LK, bool SH>
__device__ __noinline__ int label_of(const void* __restrict__ list, const float4* __restrict__ rec,
                                        const int* __restrict__ sid, const int* __restrict__ rec_sid, int start,
                                        int count, int nstructures, float x, float y, float z, int S, int& oob) {
  int L = nstructures;
  for (int i = 0; i < count; ++i) {
    if constexpr (LK == 0) {
      const int s = __ldg(sid + start + i);
      if (s < L) {
        const float4 c = __ldg(rec + start + i);
        if (inside_test(x - c.x, y - c.y, z - c.z, c.w) < 0) L = s;
      }
    } else {
      int key;
      float4 c;
      entry<LK, SH>(list, rec, sid, start + i, S, oob, key, c);
      if (inside_test(x - c.x, y - c.y, z - c.z, c.w) < 0) return __ldg(rec_sid + key);
    }
  }
  return L;
}

// Keys [lo, hi) of structure L: its records in index form (lo = hi = S for
// the box), its id in record form.
template <int LK>
__device__ __forceinline__ void label_bounds(const JobDev& J, int L, int& lo, int& hi) {
  if constexpr (LK == 0) {
    lo = L;
    hi = L + 1;
  } else if (L >= J.nstructures) {
    lo = hi = J.S;
  } else {
    lo = __ldg(J.sid_start + L);
    hi = __ldg(J.sid_start + L + 1);
  }
}

// Cell of the walker at the start of a step and the cell's centre: the
// clamped floor of x times the reciprocal cell edge plus half the cells.  For a walker
// within a rounding error of a cell face this can be the neighbour of the
// reference's division-based cell (cell_of); the walk's result is the same
// with either: the near test measures the walker's distance to the cell taken
// here, and the full lists reach jump_tol beyond their cell, so both lists
// hold every sphere the iteration can touch or be inside.
__device__ __forceinline__ int step_cell(const JobDev& J, float x, float y, float z, float& mx, float& my,
                                         float& mz) {
  const Grid& g = J.g;
  const float cz = fminf(g.nLz - 1, fmaxf(0.f, floorf(__fmaf_rn(z, J.idLz, 0.5f * g.nLz))));
  const float cy = fminf(g.nLy - 1, fmaxf(0.f, floorf(__fmaf_rn(y, J.idLy, 0.5f * g.nLy))));
  const float cx = fminf(g.nLx - 1, fmaxf(0.f, floorf(__fmaf_rn(x, J.idLx, 0.5f * g.nLx))));
  mx = __fmaf_rn(cx, g.dLx, 0.5f * (g.dLx - g.Lx));
  my = __fmaf_rn(cy, g.dLy, 0.5f * (g.dLy - g.Ly));
  mz = __fmaf_rn(cz, g.dLz, 0.5f * (g.dLz - g.Lz));
  return cell_index(J.nx, J.ny, cx, cy, cz);
}

// Start and count of cell `cell`'s list (the near list when near).  In the
// bounds-checked build a cell outside the grid, or a range outside the list,
// gives an empty list and sets oob.
__device__ __forceinline__ void cell_list(const JobDev& J, bool near, int cell, int& start, int& count, int& oob) {
  if (kCheckBounds && (cell < 0 || cell >= J.ncell)) {
    oob = 1;
    start = count = 0;
    return;
  }
  start = __ldg((near ? J.near_start : J.cell_start) + cell);
  count = __ldg((near ? J.near_count : J.cell_count) + cell);
  if (kCheckBounds) {
    const int n = near ? J.near_items : J.n_items;
    if (start < 0 || count < 0 || (n > 0 && start + count > n)) {
      oob = 1;
      start = count = 0;
    }
  }
}

// Draw `draw` of step s scaled by ds.
__device__ __forceinline__ void jump_of(const JobDev& J, uint32_t wid, int s, int draw, float ds, float& jx, float& jy,
                                        float& jz) {
  float n0, n1, n2;
  philox_normal3(J.key0, J.key1, J.stream, wid, uint32_t(s), uint32_t(draw), n0, n1, n2);
  jx = ds * n0;
  jy = ds * n1;
  jz = ds * n2;
}

// Steps [s0, s1) of the walkers of one warp, walker w in each live lane; all
// 32 lanes run the loop together until the last one is done (they share the
// scan of full lists).  Bound by issue slots and the latency of the list
// loads, with 80 registers a thread (6 warps a scheduler; 96 registers
// without the last spills are slower, 64 with more of them too): 8e8
// walker-steps on a packed substrate took 49.5 ms with every entry's record
// filtered in single precision against the reach, and up to five fractions
// for a warp's worst lane; 38.8 ms so.  Tried: all lanes' entries, or their
// marked ones, pooled over the warp in shared memory (56.3, 48.5 ms).
// Registers hold position, label and the step's jump, shared memory Phi and its
// compensation; the origin (spins0) and the flag word stay in memory and are
// updated in place on the rare wrap / iteration-cap events (with moments, which
// read the origin every step, it is in shared memory too).
template <int MODE, int LK, bool SH>
__device__ __forceinline__ void walk_warp(const JobDev& J, bool live, int w, int s0, int s1,
                                          double* s_mom, float4* s_phi) {
  static_assert(LK != 0, "index lists only");
  constexpr bool kMom = (MODE & NZ_MODE_MOMENTS) != 0;
  constexpr bool kDisp = (MODE & kModeDisp) != 0;
  constexpr bool kOrig = kMom || kDisp;  // origin in shared memory
  constexpr bool kPhi = (MODE & NZ_MODE_PHI) != 0;
  constexpr bool kT64 = (MODE & NZ_MODE_TANGENT64) != 0;
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  float x = 0.f, y = 0.f, z = 0.f;
  int label = 0;
  uint32_t wid = 0;
  float sig = 1.f;
  static_assert(!(kOrig && (MODE & NZ_MODE_PHI)), "one of phase sums and origin");
  float4& phi_sum = s_phi[threadIdx.x];  // phase modes only
  float4& origin = s_phi[threadIdx.x];   // other modes: origin (moment modes) and id
  float2& phi_comp = reinterpret_cast<float2*>(s_phi + blockDim.x)[threadIdx.x];
  int s = live ? s0 : s1;
  int niter = 0, cell = 0;
  // start and count of the step cell's primary list (the near list where
  // there is one), loaded as soon as the cell is known so that the load
  // overlaps the draw
  int pstart = 0, pcount = 0;
  float mx = 0.f, my = 0.f, mz = 0.f;  // centre of the step's cell
  float jr = 1.0f, jx = 0.0f, jy = 0.0f, jz = 0.0f;
  // ds depends on the label only; it is recomputed when the label at the
  // start of a step differs from the one it was computed for
  int ds_label = 0;
  float ds = 0.f;
  int oob = 0;  // bounds-checked build: an index was out of range
  int lo = 0, hi = 0;  // keys of structure `label`
  int within = -1;     // record of a sphere that contained the walker (-1: none known)
  const float dt = J.dt;
  if (live) {
    const float4 P = J.pos[w];
    x = P.x; y = P.y; z = P.z;
    label = __float_as_int(P.w);
    wid = __float_as_uint(J.org[w].w);
    if (MODE & NZ_MODE_SIG) sig = J.phi[w].w;
    if (MODE & NZ_MODE_PHI) {
      const float4 F = J.phi[w], C = J.comp[w];
      phi_sum = make_float4(F.x, F.y, F.z, C.x);
      phi_comp = make_float2(C.y, C.z);
    }
    if (!kPhi) origin = J.org[w];
    if (label < 0 || label > J.nstructures) label = J.nstructures;
    label_bounds<LK>(J, label, lo, hi);
    ds_label = label;
    ds = sqrtf(2 * __ldg(J.D + label) * dt);
    cell = step_cell(J, x, y, z, mx, my, mz);
    cell_list(J, true, cell, pstart, pcount, oob);
    jump_of(J, wid, s, 0, ds, jx, jy, jz);
  }
  while (__any_sync(0xffffffffu, s < s1)) {
    const bool act = s < s1;
    float jc = jr;
    float a = jx * jx + jy * jy + jz * jz;
    float reach = reach_of(a, jr);
    // Near list when everything this iteration can touch lies within its
    // margin of the step's cell: distance from the walker to the cell plus
    // the reach, with 2 % + 2 nm of slack against rounding
    // ((dist + reach) * 1.02 + tol + 2 nm <= margin, as dist^2 <= t^2 with
    // t = pack_cut - reach).
    const float dist_x = fmaxf(0.f, __fmaf_rn(-0.5f, J.g.dLx, fabsf(x - mx)));
    const float dist_y = fmaxf(0.f, __fmaf_rn(-0.5f, J.g.dLy, fabsf(y - my)));
    const float dist_z = fmaxf(0.f, __fmaf_rn(-0.5f, J.g.dLz, fabsf(z - mz)));
    const float t = J.pack_cut - reach;
    const bool near = t >= 0.f && __fmaf_rn(dist_x, dist_x, __fmaf_rn(dist_y, dist_y, dist_z * dist_z)) <= t * t;
    int start = pstart, count = act ? pcount : 0;
    if (act && !near) cell_list(J, false, cell, start, count, oob);
    // A sphere of the walker's structure whose safe ball (nz_cells_safe)
    // contains the segment's ends, and so all of it: the walker stays inside
    // that sphere and out of reach of every lower structure's, so it keeps
    // its label and takes the whole jump, and no list is scanned.  Tried: the
    // sphere that held the walker longest when its fractions were last
    // computed.
    bool deep = false;
    if (within >= lo && within < hi && near && a >= kTinyJump2) {
      const float4 c = SH ? s_stage[within] : __ldg(J.rec4 + within);
      const float safe = __ldg(J.rec_safe + within);
      const float dx = x - c.x, dy = y - c.y, dz = z - c.z;
      const float ux = __fmaf_rn(jr, jx, dx), uy = __fmaf_rn(jr, jy, dy), uz = __fmaf_rn(jr, jz, dz);
      deep = fmaxf(__fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz)), __fmaf_rn(ux, ux, __fmaf_rn(uy, uy, uz * uz))) < safe;
    }
    // The collision pass.  Each lane marks its near list's near entries 32 at
    // a time (near_bits_packed) and computes their fractions.  Where an
    // iteration needs the full list (1 walker in 100) the warp tests that list
    // together, an entry a lane, so the others do not wait for a lane's 20 and
    // more entries.
    ScanOut r;
    r.fin = 0.0f;
    r.fout = kBig;
    r.any_in = false;
    bool lower = false;
    bool more = act && !deep && count > 0;
    const bool tiny = a < kTinyJump2;  // every entry is marked; close_bits passes over the far ones
    const float inf = __int_as_float(0x7f800000);
    const void* list = near ? J.near_idx : J.idx;
    const unsigned full0 = __ballot_sync(kAll, more && !near);
    Reach g;
    if (full0) {
      const float f = 2.0f * jr;
      g.mx = f * jx;
      g.my = f * jy;
      g.mz = f * jz;
      g.m2 = a * (jr * jr);
      g.k = -0.5f * rcp_approx(g.m2);
      g.slack = tiny ? inf : kTol + 2e-3f + 0.02f * reach;
    }
    const float ir = rsqrt_approx(fmaxf(a, 1e-30f));
    const __half2 px = __float2half2_rn(x - mx), py = __float2half2_rn(y - my), pz = __float2half2_rn(z - mz);
    const __half2 ex = __float2half2_rn(jx * ir), ey = __float2half2_rn(jy * ir), ez = __float2half2_rn(jz * ir);
    const __half2 len = __float2half2_rn(reach), grow = __float2half2_rn(tiny ? inf : 0.02f * reach);
    const uint4* pk = J.near_pack + ((start + cell + 1) >> 1);
    for (int base = 0; __any_sync(kAll, more); base += 32) {
      uint32_t bits = 0u;
      if (more && near) {
        const int n = min(32, count - base);
        bits = near_bits_packed(pk + (base >> 1), (n + 1) >> 1, px, py, pz, ex, ey, ez, len, grow) &
               (((1u << ((n + 1) >> 1)) - 1u) | (((1u << (n >> 1)) - 1u) << 16));
      }
      unsigned full = full0 ? __ballot_sync(kAll, more && !near) : 0u;
      while (full) {
        const int o = __ffs(full) - 1;
        full &= full - 1;
        Reach go;
        go.mx = __shfl_sync(kAll, g.mx, o);
        go.my = __shfl_sync(kAll, g.my, o);
        go.mz = __shfl_sync(kAll, g.mz, o);
        go.m2 = __shfl_sync(kAll, g.m2, o);
        go.k = __shfl_sync(kAll, g.k, o);
        go.slack = __shfl_sync(kAll, g.slack, o);
        const float xo = __shfl_sync(kAll, x, o), yo = __shfl_sync(kAll, y, o), zo = __shfl_sync(kAll, z, o);
        const int so = __shfl_sync(kAll, start, o), no = __shfl_sync(kAll, count, o), ho = __shfl_sync(kAll, hi, o);
        // lane's entry: the one whose mark is bit `lane` (bit_entry)
        const int i = base + bit_entry(lane);
        bool yes = false;
        int bad = 0;
        if (i < no) {
          int key;
          float4 c;
          entry<LK, SH>(J.idx, J.rec4, nullptr, so + i, J.S, bad, key, c);
          yes = key < ho && is_near(go, xo, yo, zo, c);
        }
        const unsigned m = __ballot_sync(kAll, yes);
        if (kCheckBounds) bad = __any_sync(kAll, bad);
        if (lane == o) {
          bits = m;
          oob |= bad;
        }
      }
      if (tiny && bits) bits = close_bits<LK, SH>(bits, list, J.rec4, start + base, x, y, z, a, jr, J.S, oob);
      if (bits)
        fractions<LK, kT64, SH>(bits, list, J.rec4, start + base, lo, hi, x, y, z, a, jx, jy, jz, J.S, oob, r, lower, within);
      more = more && base + 32 < count;
    }
    if (!act) continue;
    niter++;
    if (deep) {
      r.any_in = true;
      r.fin = jr;
    }
    // the label carried from the previous iteration holds when no sphere of a
    // lower structure contains the walker and, outside the box, one of its own does
    if (lower || (label < J.nstructures && !r.any_in)) {
      label = label_of<LK, SH>(list, J.rec4, nullptr, J.rec_sid, start, count, J.nstructures, x, y, z, J.S, oob);
      if (kCheckBounds && (label < 0 || label > J.nstructures)) {
        oob = 1;
        label = J.nstructures;
      }
      label_bounds<LK>(J, label, lo, hi);
      if (niter == 1) {  // the first draw's length depends on the label
        ds = sqrtf(2 * __ldg(J.D + label) * dt);
        ds_label = label;
        jump_of(J, wid, s, 0, ds, jx, jy, jz);
        a = jx * jx + jy * jy + jz * jz;
      }
      // the full list: the near one was chosen for the old reach
      int fs, fc;
      cell_list(J, false, cell, fs, fc, oob);
      scan_lane<LK, kT64, SH>(J.idx, J.rec4, fs, fc, lo, hi, x, y, z, a, jx, jy, jz, jr, J.S, oob, r);
    }
    jc = ref_min(jc, r.any_in ? r.fin : kBig);
    jc = ref_min(jc, r.fout);
    x += jc * jx;
    y += jc * jy;
    z += jc * jz;
    // the next draw: the scatter draw of this step, or the first draw of the
    // next one; every iteration ends with one or the other, so one call site
    // serves all lanes of the warp
    // (the k-th iteration's scatter draw is draw k)
    int next_step = s, next_draw = niter;
    if (jc < jr) {
      jr = sqrtf(ref_max(0, jr * jr - jc * jc));
      if (MODE & NZ_MODE_SIG) sig *= t2_decay(-jc * jc * dt / __ldg(J.T2 + label));
    } else {
      jr -= jc;
      if (MODE & NZ_MODE_SIG) sig *= t2_decay(-jc * dt / __ldg(J.T2 + label));
    }
    if (!((jr > kTol) && (niter < kMaxIter))) {
      if (niter >= kMaxIter && jr > kTol) {
        float4* c = J.comp + w;
        c->w = __int_as_float(__float_as_int(c->w) | kFlagIterCap);
      }
      float fx, fy, fz, kx, ky, kz;
      if (MODE & NZ_MODE_PHI) {
        const float4 F = phi_sum;
        const float2 C = phi_comp;
        fx = F.x; fy = F.y; fz = F.z; kx = F.w; ky = C.x; kz = C.y;
        const float G = __ldg(J.G + s);
        kahan_add(fx, kx, G * x);
        kahan_add(fy, ky, G * y);
        kahan_add(fz, kz, G * z);
      }
      const float Lx = J.g.Lx, Ly = J.g.Ly, Lz = J.g.Lz;
      if (fabsf(x) > Lx / 2 || fabsf(y) > Ly / 2 || fabsf(z) > Lz / 2) {  // rare: a wrap
        const float Ga = (MODE & NZ_MODE_PHI) ? __ldg(J.Garea + s) : 0.0f;
        float4 O = kOrig ? origin : J.org[w];
        if (x < -Lx / 2) {
          x += Lx; O.x += Lx;
          if (MODE & NZ_MODE_PHI) kahan_add(fx, kx, Lx * Ga);
        } else if (x > Lx / 2) {
          x -= Lx; O.x -= Lx;
          if (MODE & NZ_MODE_PHI) kahan_add(fx, kx, -(Lx * Ga));
        }
        if (y < -Ly / 2) {
          y += Ly; O.y += Ly;
          if (MODE & NZ_MODE_PHI) kahan_add(fy, ky, Ly * Ga);
        } else if (y > Ly / 2) {
          y -= Ly; O.y -= Ly;
          if (MODE & NZ_MODE_PHI) kahan_add(fy, ky, -(Ly * Ga));
        }
        if (z < -Lz / 2) {
          z += Lz; O.z += Lz;
          if (MODE & NZ_MODE_PHI) kahan_add(fz, kz, Lz * Ga);
        } else if (z > Lz / 2) {
          z -= Lz; O.z -= Lz;
          if (MODE & NZ_MODE_PHI) kahan_add(fz, kz, -(Lz * Ga));
        }
        if (kOrig) origin = O;
        else J.org[w] = O;
      }
      if (MODE & NZ_MODE_PHI) {
        phi_sum = make_float4(fx, fy, fz, kx);
        phi_comp = make_float2(ky, kz);
      }
      if (kDisp) {  // coalesced across the warp's walkers of one step
        const size_t N = size_t(J.nwalkers);
        float* d = J.disp + size_t(s - s0) * 3 * N;
        const float4 O = origin;
        d[w] = x - O.x;
        d[N + w] = y - O.y;
        d[2 * N + w] = z - O.z;
      }
      if (kMom) {  // nz_moments' terms: float displacement, squared in FP64
        const float4 O = origin;
        const double ex = double(x - O.x), ey = double(y - O.y), ez = double(z - O.z);
        double* m = s_mom + 6 * (s - s0);
        const double ex2 = ex * ex, ey2 = ey * ey, ez2 = ez * ez;
        atomicAdd(m + 0, ex2);
        atomicAdd(m + 1, ey2);
        atomicAdd(m + 2, ez2);
        atomicAdd(m + 3, ex2 * ex2);
        atomicAdd(m + 4, ey2 * ey2);
        atomicAdd(m + 5, ez2 * ez2);
      }
      s++;
      niter = 0;
      jr = 1.0f;
      next_step = s;
      next_draw = 0;
      if (label != ds_label) {
        ds = sqrtf(2 * __ldg(J.D + label) * dt);
        ds_label = label;
      }
      cell = step_cell(J, x, y, z, mx, my, mz);
      cell_list(J, true, cell, pstart, pcount, oob);
    }
    if (s < s1) jump_of(J, kPhi ? wid : __float_as_uint(origin.w), next_step, next_draw, ds, jx, jy, jz);
  }
  if (!live) return;
  J.pos[w] = make_float4(x, y, z, __int_as_float(label));
  if (kOrig) J.org[w] = origin;
  if (MODE & NZ_MODE_PHI) {
    const float4 F = phi_sum;
    J.phi[w] = make_float4(F.x, F.y, F.z, (MODE & NZ_MODE_SIG) ? sig : J.phi[w].w);
    float4* c = J.comp + w;
    *c = make_float4(F.w, phi_comp.x, phi_comp.y, c->w);
  } else if (MODE & NZ_MODE_SIG) {
    J.phi[w].w = sig;
  }
  if (kCheckBounds && oob) {
    float4* c = J.comp + w;
    c->w = __int_as_float(__float_as_int(c->w) | kFlagBounds);
  }
}

// Steps [s0, s1) of walker w, by a lane on its own: lists without packed
// entries (on full lists of 25 entries, 1e8 walker-steps: 11.0 ms so, 11.7
// through walk_warp with single-precision marks, record lists 12.3 and 14.0).
// Registers hold position, label, Phi and its compensation and the step's
// jump; the origin (spins0) and the flag word stay in memory and are updated
// in place on the rare wrap / iteration-cap events (except with moments, which
// read the origin every step).
template <int MODE, int LK, bool SH, bool BOX>
__device__ __forceinline__ void walk_one(const JobDev& J, int w, int s0, int s1, double* s_mom) {
  constexpr bool kMom = (MODE & NZ_MODE_MOMENTS) != 0;
  constexpr bool kDisp = (MODE & kModeDisp) != 0;
  constexpr bool kOrig = kMom || kDisp;  // origin in registers
  const float4 P = J.pos[w];
  float x = P.x, y = P.y, z = P.z;
  int label = __float_as_int(P.w);
  const uint32_t wid = __float_as_uint(J.org[w].w);
  float fx = 0.f, fy = 0.f, fz = 0.f, sig = 1.f, kx = 0.f, ky = 0.f, kz = 0.f;
  if (MODE & (NZ_MODE_PHI | NZ_MODE_SIG)) {
    const float4 F = J.phi[w];
    fx = F.x; fy = F.y; fz = F.z; sig = F.w;
  }
  if (MODE & NZ_MODE_PHI) {
    const float4 C = J.comp[w];
    kx = C.x; ky = C.y; kz = C.z;
  }
  float x0 = 0.f, y0 = 0.f, z0 = 0.f;
  if (kOrig) {
    const float4 O = J.org[w];
    x0 = O.x; y0 = O.y; z0 = O.z;
  }
  if (label < 0 || label > J.nstructures) label = J.nstructures;
  int lo, hi;  // keys of structure `label`
  label_bounds<LK>(J, label, lo, hi);

  const float dt = J.dt;
  const bool has_near = (LK ? J.near_idx : static_cast<const void*>(J.near_sph4)) != nullptr;
  int s = s0;
  int niter = 0, draw = 0, cell = 0;
  // start and count of the step cell's primary list (the near list where
  // there is one), loaded as soon as the cell is known so that the load
  // overlaps the draw
  int pstart = 0, pcount = 0;
  float mx = 0.f, my = 0.f, mz = 0.f;  // centre of the step's cell
  float jr = 1.0f, jx = 0.0f, jy = 0.0f, jz = 0.0f;
  // ds depends on the label only; it is recomputed when the label at the
  // start of a step differs from the one it was computed for
  int ds_label = label;
  float ds = sqrtf(2 * __ldg(J.D + label) * dt);
  int oob = 0;  // bounds-checked build: an index was out of range
  if (s < s1) {
    cell = step_cell(J, x, y, z, mx, my, mz);
    cell_list(J, has_near, cell, pstart, pcount, oob);
    jump_of(J, wid, s, 0, ds, jx, jy, jz);
    draw = 1;
  }
  while (s < s1) {
    niter++;
    float jc = jr;
    float a = jx * jx + jy * jy + jz * jz;
    float reach = reach_of(a, jr);
    // Near list when everything this iteration can touch lies within its
    // margin of the step's cell: distance from the walker to the cell plus
    // the reach, with 2 % + 2 nm of slack against rounding
    // ((dist + reach) * 1.02 + tol + 2 nm <= margin, as dist^2 <= t^2 with
    // t = near_cut - reach).
    bool near = false;
    if (has_near) {
      const float ex = fmaxf(0.f, __fmaf_rn(-0.5f, J.g.dLx, fabsf(x - mx)));
      const float ey = fmaxf(0.f, __fmaf_rn(-0.5f, J.g.dLy, fabsf(y - my)));
      const float ez = fmaxf(0.f, __fmaf_rn(-0.5f, J.g.dLz, fabsf(z - mz)));
      const float t = J.near_cut - reach;
      near = t >= 0.f && ex * ex + ey * ey + ez * ez <= t * t;
    }
    const void* list = LK ? (near ? J.near_idx : J.idx) : nullptr;
    const float4* sph4 = LK ? J.rec4 : (near ? J.near_sph4 : J.sph4);
    const int* sidv = LK ? nullptr : (near ? J.near_sid : J.sid);
    int start = pstart, count = pcount;
    if (has_near && !near) cell_list(J, false, cell, start, count, oob);
    ScanOut r;
    constexpr bool kT64 = (MODE & NZ_MODE_TANGENT64) != 0;
    if (!scan_cell<LK, kT64, SH, BOX>(list, sph4, sidv, start, count, J.nstructures, lo, hi, x, y, z, label, a, jx, jy,
                                  jz, reach, J.S, oob, r)) {
      label = label_of<LK, SH>(list, sph4, sidv, J.rec_sid, start, count, J.nstructures, x, y, z, J.S, oob);
      if (kCheckBounds && (label < 0 || label > J.nstructures)) {
        oob = 1;
        label = J.nstructures;
      }
      label_bounds<LK>(J, label, lo, hi);
      if (niter == 1) {  // the first draw's length depends on the label
        ds = sqrtf(2 * __ldg(J.D + label) * dt);
        ds_label = label;
        jump_of(J, wid, s, 0, ds, jx, jy, jz);
        a = jx * jx + jy * jy + jz * jz;
        reach = reach_of(a, jr);
      }
      // the full list: the near one was chosen for the old reach
      int fs, fc;
      cell_list(J, false, cell, fs, fc, oob);
      scan_cell<LK, kT64, SH, BOX>(LK ? J.idx : nullptr, LK ? J.rec4 : J.sph4, LK ? nullptr : J.sid, fs, fc,
                               J.nstructures, lo, hi, x, y, z, label, a, jx, jy, jz, reach, J.S, oob, r);
    }
    jc = ref_min(jc, r.any_in ? r.fin : kBig);
    jc = ref_min(jc, r.fout);
    x += jc * jx;
    y += jc * jy;
    z += jc * jz;
    // the next draw: the scatter draw of this step, or the first draw of the
    // next one; every iteration ends with one or the other, so one call site
    // serves all lanes of the warp
    int next_step = s, next_draw = draw;
    if (jc < jr) {
      jr = sqrtf(ref_max(0, jr * jr - jc * jc));
      if (MODE & NZ_MODE_SIG) sig *= t2_decay(-jc * jc * dt / __ldg(J.T2 + label));
      draw++;
    } else {
      jr -= jc;
      if (MODE & NZ_MODE_SIG) sig *= t2_decay(-jc * dt / __ldg(J.T2 + label));
    }
    if (!((jr > kTol) && (niter < kMaxIter))) {
      if (niter >= kMaxIter && jr > kTol) {
        float4* c = J.comp + w;
        c->w = __int_as_float(__float_as_int(c->w) | kFlagIterCap);
      }
      if (MODE & NZ_MODE_PHI) {
        const float G = __ldg(J.G + s);
        kahan_add(fx, kx, G * x);
        kahan_add(fy, ky, G * y);
        kahan_add(fz, kz, G * z);
      }
      const float Lx = J.g.Lx, Ly = J.g.Ly, Lz = J.g.Lz;
      if (fabsf(x) > Lx / 2 || fabsf(y) > Ly / 2 || fabsf(z) > Lz / 2) {  // rare: a wrap
        const float Ga = (MODE & NZ_MODE_PHI) ? __ldg(J.Garea + s) : 0.0f;
        float4 O = kOrig ? make_float4(x0, y0, z0, 0.f) : J.org[w];
        if (x < -Lx / 2) {
          x += Lx; O.x += Lx;
          if (MODE & NZ_MODE_PHI) kahan_add(fx, kx, Lx * Ga);
        } else if (x > Lx / 2) {
          x -= Lx; O.x -= Lx;
          if (MODE & NZ_MODE_PHI) kahan_add(fx, kx, -(Lx * Ga));
        }
        if (y < -Ly / 2) {
          y += Ly; O.y += Ly;
          if (MODE & NZ_MODE_PHI) kahan_add(fy, ky, Ly * Ga);
        } else if (y > Ly / 2) {
          y -= Ly; O.y -= Ly;
          if (MODE & NZ_MODE_PHI) kahan_add(fy, ky, -(Ly * Ga));
        }
        if (z < -Lz / 2) {
          z += Lz; O.z += Lz;
          if (MODE & NZ_MODE_PHI) kahan_add(fz, kz, Lz * Ga);
        } else if (z > Lz / 2) {
          z -= Lz; O.z -= Lz;
          if (MODE & NZ_MODE_PHI) kahan_add(fz, kz, -(Lz * Ga));
        }
        if (kOrig) {
          x0 = O.x; y0 = O.y; z0 = O.z;
        } else {
          J.org[w] = O;
        }
      }
      if (kDisp) {  // coalesced across the warp's walkers of one step
        const size_t N = size_t(J.nwalkers);
        float* d = J.disp + size_t(s - s0) * 3 * N;
        d[w] = x - x0;
        d[N + w] = y - y0;
        d[2 * N + w] = z - z0;
      }
      if (kMom) {  // nz_moments' terms: float displacement, squared in FP64
        const double ex = double(x - x0), ey = double(y - y0), ez = double(z - z0);
        double* m = s_mom + 6 * (s - s0);
        const double ex2 = ex * ex, ey2 = ey * ey, ez2 = ez * ez;
        atomicAdd(m + 0, ex2);
        atomicAdd(m + 1, ey2);
        atomicAdd(m + 2, ez2);
        atomicAdd(m + 3, ex2 * ex2);
        atomicAdd(m + 4, ey2 * ey2);
        atomicAdd(m + 5, ez2 * ez2);
      }
      s++;
      niter = 0;
      jr = 1.0f;
      draw = 1;
      next_step = s;
      next_draw = 0;
      if (label != ds_label) {
        ds = sqrtf(2 * __ldg(J.D + label) * dt);
        ds_label = label;
      }
      cell = step_cell(J, x, y, z, mx, my, mz);
      cell_list(J, has_near, cell, pstart, pcount, oob);
    }
    if (s < s1) jump_of(J, wid, next_step, next_draw, ds, jx, jy, jz);
  }
  J.pos[w] = make_float4(x, y, z, __int_as_float(label));
  if (kOrig) J.org[w] = make_float4(x0, y0, z0, __uint_as_float(wid));
  if (MODE & (NZ_MODE_PHI | NZ_MODE_SIG)) J.phi[w] = make_float4(fx, fy, fz, sig);
  if (MODE & NZ_MODE_PHI) {
    float4* c = J.comp + w;
    *c = make_float4(kx, ky, kz, c->w);
  }
  if (kCheckBounds && oob) {
    float4* c = J.comp + w;
    c->w = __int_as_float(__float_as_int(c->w) | kFlagBounds);
  }
}

// One work item: walkers [first, first + count) of job J, steps [step0, step1)
// clamped to the job's protocol.
template <int MODE, int LK, bool SH, bool WARP, bool BOX = false>
__device__ __forceinline__ void run_item(const JobDev& J, int first, int count, int step0, int step1, double* s_mom,
                                         float4* s_phi, int flags = 0, int lanes = 32) {
  const int s0 = step0 + J.step_offset, s1 = min(step1 + J.step_offset, J.nsteps);
  if (MODE & NZ_MODE_MOMENTS) {
    for (int i = threadIdx.x; i < kMomentSteps * 6; i += blockDim.x) s_mom[i] = 0.0;
    __syncthreads();
  }
  const int slot = int(threadIdx.x >> 5) * lanes + int(threadIdx.x & 31);
  const bool live = int(threadIdx.x & 31) < lanes && slot < count && s0 < s1;
  if (WARP ? __any_sync(0xffffffffu, live) : live) {
    if constexpr (WARP) walk_warp<MODE, LK, SH>(J, live, first + slot, s0, s1, s_mom, s_phi);
    else walk_one<MODE, LK, SH, BOX>(J, first + slot, s0, s1, s_mom);
    if (live && flags) {
      float4* c = J.comp + first + slot;
      c->w = __int_as_float(__float_as_int(c->w) | flags);
    }
  }
  if (MODE & NZ_MODE_MOMENTS) {
    __syncthreads();
    if (J.moments)
      for (int i = threadIdx.x; i < (s1 - s0) * 6; i += blockDim.x)
        atomicAdd(J.moments + size_t(s0) * 6 + i, s_mom[i]);
    __syncthreads();
  }
}

// Staging a job's records into shared memory: one bulk copy (the TMA unit's
// cp.async.bulk, global -> shared) completing on an mbarrier.  Sizes are
// multiples of 16 bytes and both addresses 16-byte aligned (the host checks
// the records' address; s_stage is 16-byte aligned).  Every wait is bounded.
constexpr int kStageSpin = 1 << 20;  // try_wait polls before a copy is given up on

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
  for (int i = 0; i < kStageSpin; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
// Thread 0 only.  The CTA's generic-proxy reads of the previous contents of
// s_stage ended at a barrier before this call; the proxy fence orders them
// before the bulk copy's writes.
__device__ __forceinline__ void stage_records(uint32_t bar, const float4* src, uint32_t bytes) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(s_stage)),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// Work items are CTAs' worth of walkers of one job.  SINGLE: one job passed by
// value, stage_cap walkers a warp, item i = the i-th CTA's worth of them.
// Otherwise jobs and items come from device arrays; with queue != null the
// grid is persistent and each CTA takes items from *queue until none is left.
// STAGE (batched, index lists): a job whose S records fit in stage_cap
// records is walked with its records in shared memory (s_stage, stage_cap *
// 16 bytes of dynamic shared memory); the copy is made when a CTA's item
// belongs to a job other than the one already staged.  Larger jobs read
// their records from global memory as without STAGE.  The records are the
// same bytes either way, so the walk's results are identical.
#ifdef NZ_FUSED_MAXNREG
#define NZ_FUSED_BOUNDS __maxnreg__(NZ_FUSED_MAXNREG)
#else
#define NZ_FUSED_BOUNDS __launch_bounds__(kFusedMaxThreads, kFusedMinBlocks)
#endif
// kinds of launch: many jobs or one, their near lists packed (walk_warp) or not (walk_one)
enum : int { kBatch, kBatchPacked, kSingle, kSinglePacked };
template <int MODE, int LK, int KIND, bool STAGE>
__global__ void NZ_FUSED_BOUNDS
    walk_fused_kernel(const __grid_constant__ JobDev single, const nz_job* __restrict__ jobs,
                      const nz_item* __restrict__ items, int n_items, int step0, int step1, int* queue,
                      int stage_cap) {
  constexpr bool SINGLE = KIND == kSingle || KIND == kSinglePacked;
  constexpr bool PACKED = KIND == kBatchPacked || KIND == kSinglePacked;
  static_assert(!STAGE || (!SINGLE && LK != 0), "staging is for batched index-list walks");
  __shared__ int s_item;
  __shared__ double s_mom[(MODE & NZ_MODE_MOMENTS) ? kMomentSteps * 6 : 1];
  __shared__ JobDev s_job;
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ const float4* s_staged;  // the records now in s_stage (thread 0's bookkeeping)
  __shared__ int s_use, s_broken, s_pending;
  float4* const s_phi = s_stage + (STAGE ? stage_cap : 0);
  uint32_t phase = 0;  // parity of the barrier phase the next copy completes
  if (STAGE) {
    if (threadIdx.x == 0) {
      mbar_init(smem_addr(&s_bar));
      s_staged = nullptr;
      s_broken = s_pending = 0;
    }
    __syncthreads();
  }
  int it = blockIdx.x;
  for (;;) {
    if (queue) {
      if (threadIdx.x == 0) s_item = atomicAdd(queue, 1);
      __syncthreads();
      it = s_item;
      __syncthreads();
    }
    if (it >= n_items) {
      // a copy given up on may still be writing s_stage: wait for it (bounded)
      // before the CTA's shared memory is released
      if (STAGE && threadIdx.x == 0 && s_pending) mbar_wait_bounded(smem_addr(&s_bar), phase);
      return;
    }
    if (SINGLE) {
      const int lanes = stage_cap;  // walkers a warp
      const int per = int(blockDim.x >> 5) * lanes;
      const int first = it * per;
      const int count = min(per, single.nwalkers - first);
      run_item<MODE, LK, false, PACKED>(single, first, count, step0, step1, s_mom, s_phi, 0, lanes);
    } else {
      // every thread of the CTA works on the same job: its descriptor lives
      // in shared memory, not in each thread's registers
      const nz_item wi = items[it];
      if (threadIdx.x == 0) {
        const nz_job& a = jobs[wi.job];
        s_job = make_job(a.sub, a.G, a.Garea, a.nsteps, a.dt, a.draws, a.mode, a.state, a.moments);
        s_job.step_offset = a.step_offset;
        if (STAGE) {
          const float4* src = s_job.rec4;
          const int S = s_job.S;
          int use = 0;
          if (!s_broken && S > 0 && S <= stage_cap && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
            if (src == s_staged) {
              use = 1;
            } else {
              stage_records(smem_addr(&s_bar), src, uint32_t(S) * 16u);
              s_pending = 1;
              use = 2;
            }
          }
          s_use = use;
        }
      }
      __syncthreads();
      if (STAGE) {
        int use = s_use;
        int flags = 0;
        if (use == 2) {
          // every thread observes the copy's completion on the barrier
          const bool done = mbar_wait_bounded(smem_addr(&s_bar), phase);
          const int late = __syncthreads_or(!done);
          if (late) {  // walk from global memory; stage nothing more
            use = 0;
            flags = kFlagStageTimeout;
            if (threadIdx.x == 0) {
              s_broken = 1;
              s_staged = nullptr;
            }
          } else {
            phase ^= 1u;
            if (threadIdx.x == 0) {
              s_staged = s_job.rec4;
              s_pending = 0;
            }
          }
        }
        if (use) run_item<MODE, LK, true, PACKED>(s_job, wi.first, wi.count, step0, step1, s_mom, s_phi);
        else run_item<MODE, LK, false, false>(s_job, wi.first, wi.count, step0, step1, s_mom, s_phi, flags);
      } else {
        // Record lists: walkers in the box need no structure ids.  Leaving them
        // unread pays for full lists (four jobs, 1.5e5 walkers, 400 steps: 7.9
        // against 8.5 ms), costs a little for near lists (5.9, 5.7).
        if (LK == 0 && !s_job.near_sph4)
          run_item<MODE, LK, false, false, true>(s_job, wi.first, wi.count, step0, step1, s_mom, s_phi);
        else
          run_item<MODE, LK, false, PACKED>(s_job, wi.first, wi.count, step0, step1, s_mom, s_phi);
      }
      __syncthreads();
    }
    if (!queue) {
      if (STAGE && threadIdx.x == 0 && s_pending) mbar_wait_bounded(smem_addr(&s_bar), phase);
      return;
    }
  }
}

// ---------------------------------------------------------------------------
// packing between the reference layout and the fused state
// ---------------------------------------------------------------------------
__global__ void pack_kernel(nz_walkers wk, const uint32_t* __restrict__ ids, nz_state st) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= wk.N) return;
  const int N = wk.N;
  const int label = wk.label ? wk.label[w] : -1;
  reinterpret_cast<float4*>(st.pos)[w] =
      make_float4(wk.spins[w], wk.spins[N + w], wk.spins[2 * N + w], __int_as_float(label));
  reinterpret_cast<float4*>(st.org)[w] =
      make_float4(wk.spins0[w], wk.spins0[N + w], wk.spins0[2 * N + w], __uint_as_float(ids ? ids[w] : uint32_t(w)));
  float4 f = make_float4(0.f, 0.f, 0.f, wk.sig ? wk.sig[w] : 1.0f);
  float4 c = make_float4(0.f, 0.f, 0.f, __int_as_float(wk.flags ? wk.flags[w] : 0));
  if (wk.phi) {
    f.x = wk.phi[w]; f.y = wk.phi[N + w]; f.z = wk.phi[2 * N + w];
    c.x = wk.phi[3 * N + w]; c.y = wk.phi[4 * N + w]; c.z = wk.phi[5 * N + w];
  }
  reinterpret_cast<float4*>(st.phi)[w] = f;
  reinterpret_cast<float4*>(st.comp)[w] = c;
}

// by_id: walker w of the state goes to the reference-layout slot of its
// walker id (ids outside [0, N) are dropped and counted in *bad).
__global__ void unpack_kernel(nz_state st, nz_walkers wk, int by_id, int* bad) {
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= wk.N) return;
  int w = slot;
  if (by_id) {
    w = __float_as_int(reinterpret_cast<const float4*>(st.org)[slot].w);
    if (w < 0 || w >= wk.N) {
      if (bad) atomicAdd(bad, 1);
      return;
    }
  }
  const int N = wk.N;
  const float4 p = reinterpret_cast<const float4*>(st.pos)[slot];
  const float4 o = reinterpret_cast<const float4*>(st.org)[slot];
  const float4 f = reinterpret_cast<const float4*>(st.phi)[slot];
  const float4 c = reinterpret_cast<const float4*>(st.comp)[slot];
  wk.spins[w] = p.x; wk.spins[N + w] = p.y; wk.spins[2 * N + w] = p.z;
  wk.spins0[w] = o.x; wk.spins0[N + w] = o.y; wk.spins0[2 * N + w] = o.z;
  if (wk.label) wk.label[w] = __float_as_int(p.w);
  if (wk.sig) wk.sig[w] = f.w;
  if (wk.flags) wk.flags[w] = __float_as_int(c.w);
  if (wk.phi) {
    wk.phi[w] = f.x; wk.phi[N + w] = f.y; wk.phi[2 * N + w] = f.z;
    wk.phi[3 * N + w] = c.x; wk.phi[4 * N + w] = c.y; wk.phi[5 * N + w] = c.z;
  }
}

__host__ __device__ JobDev make_job(const nz_substrate& sub, const float* G, const float* Garea, int nsteps, float dt,
                                    const nz_draws& d, int mode, const nz_state& st, double* moments) {
  JobDev j;
  j.nwalkers = st.N;
  j.step_offset = 0;
  j.g = Grid{sub.grid.Lx, sub.grid.Ly, sub.grid.Lz, sub.grid.dLx, sub.grid.dLy, sub.grid.dLz,
             float(sub.grid.nx), float(sub.grid.ny), float(sub.grid.nz)};
  j.idLx = 1.0f / sub.grid.dLx;
  j.idLy = 1.0f / sub.grid.dLy;
  j.idLz = 1.0f / sub.grid.dLz;
  j.nx = sub.grid.nx;
  j.ny = sub.grid.ny;
  j.nstructures = sub.nstructures;
  j.ncell = sub.grid.nx * sub.grid.ny * sub.grid.nz;
  j.sph4 = reinterpret_cast<const float4*>(sub.cell_sph4);
  j.sid = sub.cell_sid;
  j.cell_start = sub.cell_start;
  j.cell_count = sub.cell_count;
  j.near_margin = sub.near_margin;
  j.near_cut = (sub.near_margin - kTol - 2e-3f) / 1.02f;
  j.near_start = sub.near_start;
  j.near_count = sub.near_count;
  j.near_sph4 = reinterpret_cast<const float4*>(sub.near_sph4);
  // packed near entries: the squared safe radius of every record, then the pairs
  const bool packed = (sub.idx_bytes & NZ_NEAR_PACKED) && sub.near_idx && sub.near_sph4;
  j.rec_safe = packed ? sub.near_sph4 : nullptr;
  j.near_pack = packed ? reinterpret_cast<const uint4*>(sub.near_sph4) + pack_radii(sub.S) : nullptr;
  // without packed entries walk_warp takes the full lists always
  j.pack_cut = packed ? j.near_cut : -1.0f;
  if (!j.near_start) j.near_start = j.cell_start;
  if (!j.near_count) j.near_count = j.cell_count;
  j.near_sid = sub.near_sid;
  j.idx = sub.idx_bytes ? sub.cell_idx : nullptr;
  j.near_idx = sub.idx_bytes ? sub.near_idx : nullptr;
  j.rec4 = reinterpret_cast<const float4*>(sub.rec4);
  j.rec_sid = sub.rec_sid;
  j.sid_start = sub.sid_start;
  j.S = sub.S;
  j.n_items = sub.n_items;
  j.near_items = sub.near_items;
  j.D = sub.D;
  j.T2 = sub.T2;
  j.G = G;
  j.Garea = Garea;
  j.nsteps = nsteps;
  j.dt = dt;
  j.key0 = d.key0;
  j.key1 = d.key1;
  j.stream = d.stream;
  j.mode = mode;
  j.pos = reinterpret_cast<float4*>(st.pos);
  j.org = reinterpret_cast<float4*>(st.org);
  j.phi = reinterpret_cast<float4*>(st.phi);
  j.comp = reinterpret_cast<float4*>(st.comp);
  j.moments = moments;
  j.disp = nullptr;
  return j;
}

// Shared memory carveout (percent) of the unstaged walk over packed lists:
// what the CTAs that the register budget allows need (and 1 KB each that the
// system takes); the rest stays L1, which the lists and records live in.
template <int MODE>
constexpr int fused_carveout() {
  constexpr size_t need = kFusedMinBlocks * phi_bytes<MODE>(kFusedMaxThreads) + 2 * kFusedMinBlocks * 1400;
  return int((100 * need + kSmemPerSm - 1) / kSmemPerSm);
}

// Dynamic shared memory of the staged kernel for stage_cap records, after
// setting its attributes: the largest allowed size (once per device) and a
// carveout that leaves room for the CTAs the register budget allows at this
// CTA size, the rest staying L1.
template <int MODE, int LK, int KIND>
size_t stage_setup(int stage_cap, int threads) {
  auto kernel = walk_fused_kernel<MODE, LK, KIND, true>;
  const size_t bytes = size_t(stage_cap) * 16 + (KIND == kBatchPacked ? phi_bytes<MODE>(threads) : 0);
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices) {
    static std::once_flag once[kMaxDevices];
    std::call_once(once[dev], [&] {
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kMaxStageRecords * 16 + int(phi_bytes<MODE>(kFusedMaxThreads)));
    });
  }
  const int ctas = std::max(1, kFusedMinBlocks * kFusedMaxThreads / threads);
  const size_t need = size_t(ctas) * (bytes + 2048);
  const int pct = int(std::min<size_t>(100, (100 * need + kSmemPerSm - 1) / kSmemPerSm));
  cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
  return bytes;
}

// packed: the near lists of all jobs (of the single one) are packed.
template <int MODE, int LK>
void launch_mode(const JobDev& single, const nz_job* jobs, const nz_item* items, int n_items, int step0, int step1,
                 int* queue, int grid, int threads, int stage_cap, bool packed, cudaStream_t st) {
  // walk_one keeps nothing in shared memory: the whole carveout for L1.
  // Function attributes belong to a device's context, so this is done once
  // per device (and once across threads).
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices) {
    static std::once_flag once[kMaxDevices];
    std::call_once(once[dev], [] {
      auto carve = [](auto kernel, int pct) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
      };
      carve(walk_fused_kernel<MODE, LK, kBatch, false>, 0);
      carve(walk_fused_kernel<MODE, LK, kSingle, false>, 0);
      if constexpr (LK != 0) {
        carve(walk_fused_kernel<MODE, LK, kBatchPacked, false>, fused_carveout<MODE>());
        carve(walk_fused_kernel<MODE, LK, kSinglePacked, false>, fused_carveout<MODE>());
      }
    });
  }
  auto run = [&](auto kernel, size_t smem) {
    kernel<<<grid, threads, smem, st>>>(single, jobs, items, n_items, step0, step1, queue, stage_cap);
  };
  if constexpr (LK != 0) {
    const size_t bytes = phi_bytes<MODE>(threads);
    if (jobs && stage_cap > 0)
      return packed ? run(walk_fused_kernel<MODE, LK, kBatchPacked, true>,
                          stage_setup<MODE, LK, kBatchPacked>(stage_cap, threads))
                    : run(walk_fused_kernel<MODE, LK, kBatch, true>, stage_setup<MODE, LK, kBatch>(stage_cap, threads));
    if (jobs && packed) return run(walk_fused_kernel<MODE, LK, kBatchPacked, false>, bytes);
    if (packed) return run(walk_fused_kernel<MODE, LK, kSinglePacked, false>, bytes);
  }
  if (jobs) run(walk_fused_kernel<MODE, LK, kBatch, false>, 0);
  else run(walk_fused_kernel<MODE, LK, kSingle, false>, 0);
}

template <int LK>
int launch_lk(int mode, const JobDev& single, const nz_job* jobs, const nz_item* items, int n_items, int step0,
              int step1, int* queue, int grid, int threads, int stage_cap, cudaStream_t st) {
  const bool packed = jobs ? (mode & NZ_LIST_PACKED) != 0 : single.near_pack != nullptr;
#define NZ_LAUNCH(M) \
  launch_mode<(M), LK>(single, jobs, items, n_items, step0, step1, queue, grid, threads, stage_cap, packed, st)
  switch (mode & (NZ_MODE_PHI | NZ_MODE_SIG | NZ_MODE_MOMENTS | NZ_MODE_TANGENT64 | kModeDisp)) {
    case NZ_MODE_PHI | NZ_MODE_TANGENT64: NZ_LAUNCH(NZ_MODE_PHI | NZ_MODE_TANGENT64); break;
    case NZ_MODE_PHI | NZ_MODE_SIG | NZ_MODE_TANGENT64: NZ_LAUNCH(NZ_MODE_PHI | NZ_MODE_SIG | NZ_MODE_TANGENT64); break;
    case NZ_MODE_PHI: NZ_LAUNCH(NZ_MODE_PHI); break;
    case NZ_MODE_SIG: NZ_LAUNCH(NZ_MODE_SIG); break;
    case NZ_MODE_PHI | NZ_MODE_SIG: NZ_LAUNCH(NZ_MODE_PHI | NZ_MODE_SIG); break;
    case NZ_MODE_SIG | NZ_MODE_MOMENTS: NZ_LAUNCH(NZ_MODE_SIG | NZ_MODE_MOMENTS); break;
    case NZ_MODE_MOMENTS: NZ_LAUNCH(NZ_MODE_MOMENTS); break;
    case NZ_MODE_SIG | kModeDisp: NZ_LAUNCH(NZ_MODE_SIG | kModeDisp); break;
    case kModeDisp: NZ_LAUNCH(kModeDisp); break;
    case 0: NZ_LAUNCH(0); break;
    default: return set_error(NZ_ERR_ARG, "fused walk: unsupported mode %d", mode);
  }
#undef NZ_LAUNCH
  return check_launch("walk_fused_kernel");
}

// jobs == null: the single job `single`, stage_cap walkers a warp, n_items CTAs
// of kFusedThreads threads.  Batched index-list walks: stage_cap > 0 stages the
// records of jobs of at most that many in shared memory; NZ_LIST_PACKED in
// mode takes the walk over packed near lists.  Without that bit each lane
// walks by itself: unpacked index lists of four jobs, 1.5e5 walkers, 400
// steps, 256 (128) threads a CTA: 7.2 (6.9) ms so, 8.1 (8.0) through walk_warp;
// with their records staged 8.5 (9.5) and 9.9 (11.8).
int launch_fused(int mode, int lk, const JobDev& single, const nz_job* jobs, const nz_item* items, int n_items,
                 int step0, int step1, int* queue, int grid, int threads, cudaStream_t st, int stage_cap) {
  switch (lk) {
    case 0:
      return launch_lk<0>(mode, single, jobs, items, n_items, step0, step1, queue, grid, threads, jobs ? 0 : stage_cap,
                          st);
    case 2:
      return launch_lk<2>(mode, single, jobs, items, n_items, step0, step1, queue, grid, threads, stage_cap, st);
    case 4:
      return launch_lk<4>(mode, single, jobs, items, n_items, step0, step1, queue, grid, threads, stage_cap, st);
    default: return set_error(NZ_ERR_ARG, "fused walk: list kind %d is not 0, 2 or 4", lk);
  }
}

template <int MODE, int LK>
cudaError_t occupancy_mode(int threads, int stage_cap, bool packed, int* blocks_per_sm) {
  auto fit = [&](auto kernel, size_t smem) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel, threads, smem);
  };
  if constexpr (LK != 0) {
    if (stage_cap > 0)
      return packed ? fit(walk_fused_kernel<MODE, LK, kBatchPacked, true>,
                          stage_setup<MODE, LK, kBatchPacked>(stage_cap, threads))
                    : fit(walk_fused_kernel<MODE, LK, kBatch, true>, stage_setup<MODE, LK, kBatch>(stage_cap, threads));
    if (packed) return fit(walk_fused_kernel<MODE, LK, kBatchPacked, false>, phi_bytes<MODE>(threads));
  }
  return fit(walk_fused_kernel<MODE, LK, kBatch, false>, 0);
}

template <int LK>
cudaError_t occupancy_lk(int mode, int threads, int stage_cap, int* blocks_per_sm) {
  const bool packed = (mode & NZ_LIST_PACKED) != 0;
  switch (mode & (NZ_MODE_PHI | NZ_MODE_SIG | NZ_MODE_MOMENTS)) {
    case NZ_MODE_PHI: return occupancy_mode<NZ_MODE_PHI, LK>(threads, stage_cap, packed, blocks_per_sm);
    case NZ_MODE_SIG: return occupancy_mode<NZ_MODE_SIG, LK>(threads, stage_cap, packed, blocks_per_sm);
    case NZ_MODE_PHI | NZ_MODE_SIG: return occupancy_mode<NZ_MODE_PHI | NZ_MODE_SIG, LK>(threads, stage_cap, packed, blocks_per_sm);
    default: return cudaErrorInvalidValue;
  }
}

int occupancy_fused(int mode, int lk, int threads, int* blocks_per_sm, int stage_cap) {
  const int m = mode & (NZ_MODE_PHI | NZ_MODE_SIG | NZ_MODE_MOMENTS);
  if (m != NZ_MODE_PHI && m != NZ_MODE_SIG && m != (NZ_MODE_PHI | NZ_MODE_SIG))
    return set_error(NZ_ERR_ARG, "occupancy: unsupported batch mode %d", mode);
  cudaError_t e;
  switch (lk) {
    case 0: e = occupancy_lk<0>(mode, threads, 0, blocks_per_sm); break;
    case 2: e = occupancy_lk<2>(mode, threads, stage_cap, blocks_per_sm); break;
    case 4: e = occupancy_lk<4>(mode, threads, stage_cap, blocks_per_sm); break;
    default: return set_error(NZ_ERR_ARG, "occupancy: list kind %d is not 0, 2 or 4", lk);
  }
  if (e != cudaSuccess) return set_error(NZ_ERR_CUDA, "occupancy: %s", cudaGetErrorString(e));
  return NZ_OK;
}

}  // namespace nz
