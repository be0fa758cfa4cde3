// Device probes: the draws' transform on given words and its division and root
// on all words, for tests; and the peak used by the benchmark to state the
// FP32 roofline it reports against: each thread runs 8 independent fused
// multiply-add chains.
#include "kernels.cuh"

namespace nz {

__global__ void __launch_bounds__(256) fma_probe_kernel(int iters, float seed, float* __restrict__ out) {
  float a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = seed + float(threadIdx.x + i);
  const float m = 0.999999f, c = 1e-7f;
  for (int k = 0; k < iters; ++k) {
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = __fmaf_rn(a[i], m, c);
  }
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) s += a[i];
  if (s == 12345.678f) out[blockIdx.x] = s;  // keeps the chains live
}

// Box-Muller of each pair of word pairs, as the walks' draws transform them.
__global__ void __launch_bounds__(256) box_muller_probe_kernel(const uint4* __restrict__ words, int n,
                                                               float4* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint4 w = words[i];
  float4 v;
  box_muller2(w.x, w.y, w.z, w.w, v.x, v.y, v.z, v.w);
  out[i] = v;
}

// The draws' division and root of word w and of another word beside it (each
// word comes once on either side), against the IEEE operators.
__global__ void __launch_bounds__(256) draw_operators_probe_kernel(unsigned long long* __restrict__ differ) {
  unsigned long long bad = 0;
  const uint32_t step = gridDim.x * blockDim.x;  // divides 2^32
  uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
  for (uint32_t k = 0; k < uint32_t((1ull << 32) / step); ++k, w += step) {
    const F2 u = unit2(w, w * 0x9E3779B1u);
    float x[2], m[2], e[2], got[2], l[2];
    split(u, x[0], x[1]);
    for (int i = 0; i < 2; ++i) log_parts(x[i], m[i], e[i]);
    split(log_ratio2(f2(m[0], m[1])), got[0], got[1]);
    for (int i = 0; i < 2; ++i) bad += __float_as_uint(got[i]) != __float_as_uint((m[i] - 1.0f) / (m[i] + 1.0f));
    const F2 l2 = mul2(f2(-2.0f), log_series2(u));
    split(l2, l[0], l[1]);
    split(sqrt2_plain(l2), got[0], got[1]);
    for (int i = 0; i < 2; ++i)  // box_muller2 takes l itself where it is not above 0
      bad += l[i] > 0.0f && __float_as_uint(got[i]) != __float_as_uint(sqrtf(l[i]));
  }
  if (bad) atomicAdd(differ, bad);
}

}  // namespace nz

using namespace nz;

// FP32 FMA throughput probe: grid x 256 threads x iters x 8 FMAs (2 flops each).
extern "C" int nz_probe_fma(int grid, int iters, float* out, void* stream) {
  if (grid <= 0 || iters <= 0 || !out) return set_error(NZ_ERR_ARG, "nz_probe_fma: bad arguments");
  fma_probe_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(iters, 1.0f, out);
  return check_launch("fma_probe_kernel");
}

extern "C" int nz_probe_box_muller(const uint32_t* words, int n, float* out, void* stream) {
  if (n < 0 || (n > 0 && (!words || !out)) || (reinterpret_cast<uintptr_t>(words) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 15))
    return set_error(NZ_ERR_ARG, "nz_probe_box_muller: bad arguments (n=%d)", n);
  if (n == 0) return NZ_OK;
  box_muller_probe_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const uint4*>(words), n, reinterpret_cast<float4*>(out));
  return check_launch("box_muller_probe_kernel");
}

extern "C" int nz_probe_draw_operators(unsigned long long* differ, void* stream) {
  if (!differ) return set_error(NZ_ERR_ARG, "nz_probe_draw_operators: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(differ, 0, sizeof(*differ), st) != cudaSuccess)
    return check_launch("nz_probe_draw_operators memset");
  draw_operators_probe_kernel<<<1024, 256, 0, st>>>(differ);
  return check_launch("draw_operators_probe_kernel");
}
