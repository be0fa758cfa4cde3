// Plain walk kernel: one time step per launch, one thread per walker, walker
// state in HBM in the reference's layout (spins [3,N], spins0 [3,N],
// phase [ndir,N], sig [N]).  It is the drop-in for the reference's
// randomWalk3d (sim3d_kernel.cu:340-522), randomWalk3d_phase (:524-717) and
// randomWalk3d_phase_multidirr (:719-943) and the per-substrate baseline that
// the fused and batched paths are measured against.
//
// Differences from the reference kernel that do not change any result:
// a bounds guard (the reference needs N to be a multiple of its 1000-thread
// block), counter-based draws instead of a 48-byte cuRAND state per walker,
// compact cell lists (start, count) in place of the padded table (the padded
// table is the case start = c*K, count = K), runtime geometry instead of
// compile-time constants.
#include "kernels.cuh"

namespace nz {


__global__ void __launch_bounds__(256) walk_plain_kernel(const PlainArgs a) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= a.N) return;
  const int S = a.S, N = a.N;
  const float* __restrict__ cx = a.spheres;
  const float* __restrict__ cy = a.spheres + S;
  const float* __restrict__ cz = a.spheres + 2 * S;
  const float* __restrict__ rr = a.spheres + 3 * S;
  const float* __restrict__ sphSID = a.spheres + 4 * S;

  float x = a.spins[w], y = a.spins[N + w], z = a.spins[2 * N + w];
  int flags = a.flags ? a.flags[w] : 0;
  float sig = (a.mode & NZ_MODE_SIG) ? a.sig[w] : 1.0f;

  float ds = 0, jx = 0, jy = 0, jz = 0;
  float jump_current, jump_remaining = 1.0f;

  const int idxSeg = cell_of(a.g, x, y, z);
  int start = 0, count = 0;
  if (!kCheckBounds || (idxSeg >= 0 && idxSeg < a.ncell)) {
    start = __ldg(a.cell_start + idxSeg);
    count = __ldg(a.cell_count + idxSeg);
  } else {
    flags |= kFlagBounds;
  }
  if (kCheckBounds && (start < 0 || count < 0 || (a.n_items > 0 && start + count > a.n_items))) {
    flags |= kFlagBounds;
    start = count = 0;
  }
  const int* __restrict__ items = a.cell_items + start;

  int niter = 0, nscatter = 0, draw = 0;
  int spinSID = a.nstructures;
  while ((jump_remaining > kTol) && (niter < kMaxIter)) {
    niter++;
    jump_current = jump_remaining;

    // label: lowest structure id among the spheres containing the walker
    spinSID = a.nstructures;
    for (int n = 0; n < count; n++) {
      const int s = __ldg(items + n);
      if (kCheckBounds && (s < 0 || s >= S)) {
        flags |= kFlagBounds;
        continue;
      }
      const float sid = __ldg(sphSID + s);
      if (sid < spinSID) {
        const float isIn = inside_test(x - __ldg(cx + s), y - __ldg(cy + s), z - __ldg(cz + s), __ldg(rr + s));
        if (isIn < 0) spinSID = int(sid);
      }
    }
    if (kCheckBounds && (spinSID < 0 || spinSID > a.nstructures)) {
      flags |= kFlagBounds;
      spinSID = a.nstructures;
    }

    if (niter == 1) {
      float n0, n1, n2;
      draw3(a.draws, uint32_t(w), a.step, draw++, n0, n1, n2, flags);
      ds = sqrtf(2 * __ldg(a.D + spinSID) * a.dt);
      jx = ds * n0;
      jy = ds * n1;
      jz = ds * n2;
    }

    const float aa = jx * jx + jy * jy + jz * jz;
    float isInsideAny = 0;
    float furthest_fstep_in = 0;
    float closest_fstep_out = kBig;
    for (int n = 0; n < count; n++) {
      const int s = __ldg(items + n);
      if (kCheckBounds && (s < 0 || s >= S)) continue;  // flagged in the label pass
      const float sid = __ldg(sphSID + s);
      if (sid > spinSID) continue;
      const float dx = x - __ldg(cx + s), dy = y - __ldg(cy + s), dz = z - __ldg(cz + s);
      const float r = __ldg(rr + s);
      const float isIn = inside_test(dx, dy, dz, r);
      if (isIn < 0) {
        isInsideAny = 1;
        const float f = step_in(dx, dy, dz, r, aa, jx, jy, jz);
        if (furthest_fstep_in < f) furthest_fstep_in = f;
      } else if (sid < spinSID) {
        const float f = step_out(dx, dy, dz, r, aa, jx, jy, jz);
        if (f < closest_fstep_out) closest_fstep_out = f;
      }
    }

    jump_current = ref_min(jump_current, isInsideAny ? furthest_fstep_in : kBig);
    jump_current = ref_min(jump_current, closest_fstep_out);
    x += jump_current * jx;
    y += jump_current * jy;
    z += jump_current * jz;

    if (jump_current < jump_remaining) {
      jump_remaining = sqrtf(ref_max(0, jump_remaining * jump_remaining - jump_current * jump_current));
      if (a.mode & NZ_MODE_SIG) sig *= t2_decay(-jump_current * jump_current * a.dt / __ldg(a.T2 + spinSID));
      float n0, n1, n2;
      draw3(a.draws, uint32_t(w), a.step, draw++, n0, n1, n2, flags);
      jx = ds * n0;
      jy = ds * n1;
      jz = ds * n2;
      nscatter++;
    } else {
      jump_remaining -= jump_current;
      if (a.mode & NZ_MODE_SIG) sig *= t2_decay(-jump_current * a.dt / __ldg(a.T2 + spinSID));
    }
  }
  if (niter >= kMaxIter && jump_remaining > kTol) flags |= kFlagIterCap;

  // phase of every direction from the post-step, pre-wrap position
  const int nd = a.ndir;
  if (a.mode & NZ_MODE_PHASE) {
    for (int d = 0; d < nd; ++d) {
      const float proj = x * __ldg(a.diffdir + d) + y * __ldg(a.diffdir + nd + d) + z * __ldg(a.diffdir + 2 * nd + d);
      a.phase[w + size_t(d) * N] += proj * a.G;
    }
  }
  float fx = 0, fy = 0, fz = 0, kx = 0, ky = 0, kz = 0;
  if (a.mode & NZ_MODE_PHI) {
    fx = a.phi[w]; fy = a.phi[N + w]; fz = a.phi[2 * N + w];
    kx = a.phi[3 * N + w]; ky = a.phi[4 * N + w]; kz = a.phi[5 * N + w];
    kahan_add(fx, kx, a.G * x);
    kahan_add(fy, ky, a.G * y);
    kahan_add(fz, kz, a.G * z);
  }

  // periodic wrap; spins0 and phase follow the walker
  const float Lx = a.g.Lx, Ly = a.g.Ly, Lz = a.g.Lz;
  if (x < -Lx / 2) {
    x += Lx; a.spins0[w] += Lx;
    if (a.mode & NZ_MODE_PHASE) for (int d = 0; d < nd; ++d) a.phase[w + size_t(d) * N] += Lx * __ldg(a.diffdir + d) * a.Garea;
    if (a.mode & NZ_MODE_PHI) kahan_add(fx, kx, Lx * a.Garea);
  } else if (x > Lx / 2) {
    x -= Lx; a.spins0[w] -= Lx;
    if (a.mode & NZ_MODE_PHASE) for (int d = 0; d < nd; ++d) a.phase[w + size_t(d) * N] -= Lx * __ldg(a.diffdir + d) * a.Garea;
    if (a.mode & NZ_MODE_PHI) kahan_add(fx, kx, -(Lx * a.Garea));
  }
  if (y < -Ly / 2) {
    y += Ly; a.spins0[N + w] += Ly;
    if (a.mode & NZ_MODE_PHASE) for (int d = 0; d < nd; ++d) a.phase[w + size_t(d) * N] += Ly * __ldg(a.diffdir + nd + d) * a.Garea;
    if (a.mode & NZ_MODE_PHI) kahan_add(fy, ky, Ly * a.Garea);
  } else if (y > Ly / 2) {
    y -= Ly; a.spins0[N + w] -= Ly;
    if (a.mode & NZ_MODE_PHASE) for (int d = 0; d < nd; ++d) a.phase[w + size_t(d) * N] -= Ly * __ldg(a.diffdir + nd + d) * a.Garea;
    if (a.mode & NZ_MODE_PHI) kahan_add(fy, ky, -(Ly * a.Garea));
  }
  if (z < -Lz / 2) {
    z += Lz; a.spins0[2 * N + w] += Lz;
    if (a.mode & NZ_MODE_PHASE) for (int d = 0; d < nd; ++d) a.phase[w + size_t(d) * N] += Lz * __ldg(a.diffdir + 2 * nd + d) * a.Garea;
    if (a.mode & NZ_MODE_PHI) kahan_add(fz, kz, Lz * a.Garea);
  } else if (z > Lz / 2) {
    z -= Lz; a.spins0[2 * N + w] -= Lz;
    if (a.mode & NZ_MODE_PHASE) for (int d = 0; d < nd; ++d) a.phase[w + size_t(d) * N] -= Lz * __ldg(a.diffdir + 2 * nd + d) * a.Garea;
    if (a.mode & NZ_MODE_PHI) kahan_add(fz, kz, -(Lz * a.Garea));
  }

  a.spins[w] = x;
  a.spins[N + w] = y;
  a.spins[2 * N + w] = z;
  if (a.mode & NZ_MODE_SIG) a.sig[w] = sig;
  if (a.mode & NZ_MODE_PHI) {
    a.phi[w] = fx; a.phi[N + w] = fy; a.phi[2 * N + w] = fz;
    a.phi[3 * N + w] = kx; a.phi[4 * N + w] = ky; a.phi[5 * N + w] = kz;
  }
  if (a.label) a.label[w] = spinSID;
  if (a.n_iter) a.n_iter[w] += niter;
  if (a.n_scatter) a.n_scatter[w] += nscatter;
  if (a.flags) a.flags[w] = flags;
}

// The same step over index lists (records by structure, a cell's entries
// ascending): G lanes share a walker.  They take every G-th entry of its list
// and agree by shuffles; the rest of the step each of them does alike.  One
// pass finds the first containing entry, which gives the label (structures
// ascend), and marks the near spheres; a sphere whose (r + tol) ball lies
// more than 2 % + 2 nm beyond the iteration's reach is not solved (it neither
// contains the walker nor lowers the jump fraction).  Phases, positions and counters are written by the
// block's threads walker by walker, whole lines at a time.
//
// Bound by the loads of the list's records (L1 and L2) and the scan's issue
// slots.  5e4 walkers x 30 directions on lists of about 100 entries took 272
// us a step with one lane a walker and the spheres' five arrays (7 of 32 lanes
// active, 12 % of the warps), 58 us so.
template <int G, typename T>
__global__ void __launch_bounds__(256) walk_plain_lists_kernel(const PlainArgs a, const PlainLists l) {
  constexpr int kWalkers = 256 / G;
  __shared__ float4 s_pos[kWalkers];  // position before the wrap; T2 weight
  __shared__ int4 s_out[kWalkers];    // label, iterations, scatterings, flags
  const int lane = threadIdx.x & 31, sub = threadIdx.x % G, slot = threadIdx.x / G;
  const unsigned group = (G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u)) << (lane & ~(G - 1));
  const int w0 = blockIdx.x * kWalkers, w = w0 + slot;
  const int S = a.S, N = a.N;
  if (w < N) {
    float x = a.spins[w], y = a.spins[size_t(N) + w], z = a.spins[2 * size_t(N) + w];
    int flags = a.flags ? a.flags[w] : 0;
    float sig = (a.mode & NZ_MODE_SIG) ? a.sig[w] : 1.0f;
    const int cell = cell_of(a.g, x, y, z);
    int start = 0, count = 0;
    if (!kCheckBounds || (cell >= 0 && cell < a.ncell)) {
      start = __ldg(a.cell_start + cell);
      count = __ldg(a.cell_count + cell);
    } else {
      flags |= kFlagBounds;
    }
    if (kCheckBounds && (start < 0 || count < 0 || (a.n_items > 0 && start + count > a.n_items))) {
      flags |= kFlagBounds;
      start = count = 0;
    }
    const T* __restrict__ idx = static_cast<const T*>(l.idx) + start;
    int bad = 0;
    auto entry = [&](int i, int& key, float4& c) {
      key = int(__ldg(idx + i));
      if (kCheckBounds && (key < 0 || key >= S)) {
        bad = 1;
        key = 0x7fffffff;
        c = make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
        return;
      }
      c = __ldg(l.rec4 + key);
    };
    // how far beyond a sphere's surface the filter keeps it; a jump too short
    // for the filter's arithmetic keeps every one
    auto slack_of = [](float aa, float jr) {
      return aa < 1e-8f ? __int_as_float(0x7f800000) : kTol + sqrtf(aa) * jr * 1.02f + 2e-3f;
    };
    const float ds_box = sqrtf(2 * __ldg(a.D + a.nstructures) * a.dt);
    float ds = 0, jx = 0, jy = 0, jz = 0, jr = 1.0f, n0 = 0, n1 = 0, n2 = 0;
    int niter = 0, nscatter = 0, draw = 0, label = a.nstructures;
    while (jr > kTol && niter < kMaxIter) {
      niter++;
      // the iteration's jump, which the filter needs; the first one's length
      // depends on the label, so the box's stands in for it until that is
      // known
      if (niter == 1) {
        draw3(a.draws, uint32_t(w), a.step, draw++, n0, n1, n2, flags);
        ds = ds_box;
        jx = ds * n0;
        jy = ds * n1;
        jz = ds * n2;
      }
      float aa = jx * jx + jy * jy + jz * jz;
      float slack = slack_of(aa, jr);
      // one pass: the first containing entry (the label), and which of the
      // lane's first 32 entries are near
      int best = 0x7fffffff, stop = 0x7fffffff;
      unsigned near = 0u;
      int k = 0;
      for (int i = sub; i < count; i += G, ++k) {
        int key;
        float4 c;
        entry(i, key, c);
        if (key >= stop) break;
        const float dx = x - c.x, dy = y - c.y, dz = z - c.z;
        const float d2 = dx * dx + dy * dy + dz * dz, ro = c.w + slack;
        if (d2 <= ro * ro) {
          near |= k < 32 ? 1u << k : 0u;
          if (best == 0x7fffffff && d2 - c.w * c.w < 0) {
            best = key;  // nothing above this structure counts
            stop = __ldg(l.sid_start + __ldg(l.rec_sid + key) + 1);
          }
        }
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(group, best, o));
      int lo, hi;
      if (best == 0x7fffffff) {
        label = a.nstructures;
        lo = hi = S;
      } else {
        label = __ldg(l.rec_sid + best);
        lo = __ldg(l.sid_start + label);
        hi = __ldg(l.sid_start + label + 1);
      }
      bool marked = count <= 32 * G;  // the marks cover the list
      if (niter == 1) {
        ds = sqrtf(2 * __ldg(a.D + label) * a.dt);
        jx = ds * n0;
        jy = ds * n1;
        jz = ds * n2;
        aa = jx * jx + jy * jy + jz * jz;
        const float now = slack_of(aa, jr);
        marked &= now <= slack;  // and this jump
        slack = now;
      }
      float fin = -1.0f, fout = kBig;  // fin -1: no containing sphere
      auto solve = [&](int key, float4 c) {
        const float dx = x - c.x, dy = y - c.y, dz = z - c.z;
        const float d2 = dx * dx + dy * dy + dz * dz, ro = c.w + slack;
        if (!(d2 <= ro * ro)) return;
        const bool inside = d2 - c.w * c.w < 0;
        if (inside || key < lo) {
          const float f = step_either(inside, dx, dy, dz, c.w, aa, jx, jy, jz);
          if (inside) fin = fmaxf(fin, f > 0.0f ? f : 0.0f);
          else if (f < fout) fout = f;
        }
      };
      if (marked) {
        while (near) {
          int key;
          float4 c;
          entry(sub + G * (__ffs(near) - 1), key, c);
          near &= near - 1u;
          if (key < hi) solve(key, c);
        }
      } else {
        for (int i = sub; i < count; i += G) {
          int key;
          float4 c;
          entry(i, key, c);
          if (key >= hi) break;
          solve(key, c);
        }
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) {
        fin = fmaxf(fin, __shfl_xor_sync(group, fin, o));
        fout = fminf(fout, __shfl_xor_sync(group, fout, o));
      }
      float jc = ref_min(jr, fin >= 0.0f ? fin : kBig);
      jc = ref_min(jc, fout);
      x += jc * jx;
      y += jc * jy;
      z += jc * jz;
      if (jc < jr) {
        jr = sqrtf(ref_max(0, jr * jr - jc * jc));
        if (a.mode & NZ_MODE_SIG) sig *= t2_decay(-jc * jc * a.dt / __ldg(a.T2 + label));
        draw3(a.draws, uint32_t(w), a.step, draw++, n0, n1, n2, flags);
        jx = ds * n0;
        jy = ds * n1;
        jz = ds * n2;
        nscatter++;
      } else {
        jr -= jc;
        if (a.mode & NZ_MODE_SIG) sig *= t2_decay(-jc * a.dt / __ldg(a.T2 + label));
      }
    }
    if (niter >= kMaxIter && jr > kTol) flags |= kFlagIterCap;
    if (kCheckBounds) {
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) bad |= __shfl_xor_sync(group, bad, o);
      if (bad) flags |= kFlagBounds;
    }
    if (sub == 0) {
      s_pos[slot] = make_float4(x, y, z, sig);
      s_out[slot] = make_int4(label, niter, nscatter, flags);
    }
  }
  __syncthreads();
  const int here = min(kWalkers, N - w0);
  const float Lx = a.g.Lx, Ly = a.g.Ly, Lz = a.g.Lz;
  // phase of every direction from the position before the wrap, then the
  // wrap's terms, axis by axis
  if (a.mode & NZ_MODE_PHASE) {
    const int nd = a.ndir;
    for (int k = threadIdx.x; k < kWalkers * nd; k += 256) {
      const int i = k % kWalkers, d = k / kWalkers;
      if (i >= here) continue;
      const float4 p = s_pos[i];
      const float ux = __ldg(a.diffdir + d), uy = __ldg(a.diffdir + nd + d), uz = __ldg(a.diffdir + 2 * nd + d);
      float* const at = a.phase + size_t(d) * N + w0 + i;
      float ph = *at;
      const float proj = p.x * ux + p.y * uy + p.z * uz;
      ph += proj * a.G;
      if (p.x < -Lx / 2) ph += Lx * ux * a.Garea;
      else if (p.x > Lx / 2) ph -= Lx * ux * a.Garea;
      if (p.y < -Ly / 2) ph += Ly * uy * a.Garea;
      else if (p.y > Ly / 2) ph -= Ly * uy * a.Garea;
      if (p.z < -Lz / 2) ph += Lz * uz * a.Garea;
      else if (p.z > Lz / 2) ph -= Lz * uz * a.Garea;
      *at = ph;
    }
  }
  for (int i = threadIdx.x; i < here; i += 256) {
    const int v = w0 + i;
    const float4 p = s_pos[i];
    const int4 o = s_out[i];
    const float pos[3] = {p.x, p.y, p.z}, len[3] = {Lx, Ly, Lz};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float q = pos[k], term = 0.0f;
      float *const org = a.spins0 + size_t(k) * N + v;
      if (q < -len[k] / 2) {
        q += len[k];
        *org += len[k];
        term = len[k] * a.Garea;
      } else if (q > len[k] / 2) {
        q -= len[k];
        *org -= len[k];
        term = -(len[k] * a.Garea);
      }
      a.spins[size_t(k) * N + v] = q;
      if (a.mode & NZ_MODE_PHI) {
        float* const f = a.phi + size_t(k) * N + v;
        float* const c = a.phi + size_t(3 + k) * N + v;
        float fs = *f, cs = *c;
        kahan_add(fs, cs, a.G * pos[k]);
        if (q != pos[k]) kahan_add(fs, cs, term);
        *f = fs;
        *c = cs;
      }
    }
    if (a.mode & NZ_MODE_SIG) a.sig[v] = p.w;
    if (a.label) a.label[v] = o.x;
    if (a.n_iter) a.n_iter[v] += o.y;
    if (a.n_scatter) a.n_scatter[v] += o.z;
    if (a.flags) a.flags[v] = o.w;
  }
}

// Lanes a walker: eight while that many threads still fit the GPU about once
// and a half (148 SMs of 2048), else four.  A step of 5e4 walkers on lists of
// about 100 takes 58 us with eight, 61 with four; of 7.5e4 on lists of 17, 70
// and 66 us; of 1e6 on lists of 17 / 44 entries 654 / 795 us with eight, 520 /
// 710 with four, 467 / 846 with two (955 / 1950 with one lane and the spheres'
// arrays).
int launch_plain_lists(const PlainArgs& a, const PlainLists& l, int idx_bytes, cudaStream_t st) {
  const bool eight = 8ll * a.N <= 148ll * 2048 * 3 / 2;
  const int per = eight ? 32 : 64;
  const unsigned blocks = unsigned((a.N + per - 1) / per);
  if (idx_bytes == 2) {
    if (eight) walk_plain_lists_kernel<8, uint16_t><<<blocks, 256, 0, st>>>(a, l);
    else walk_plain_lists_kernel<4, uint16_t><<<blocks, 256, 0, st>>>(a, l);
  } else {
    if (eight) walk_plain_lists_kernel<8, int><<<blocks, 256, 0, st>>>(a, l);
    else walk_plain_lists_kernel<4, int><<<blocks, 256, 0, st>>>(a, l);
  }
  return check_launch("walk_plain_lists_kernel");
}

}  // namespace nz
