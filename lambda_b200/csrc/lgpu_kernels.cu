// lgpu_kernels.cu — closest-hit, render and tone-map kernels.
#include <float.h>
#include <stdint.h>

#include "lgpu_counters.cuh"
#include "lgpu_kernels.cuh"

namespace lgpu {

namespace {

// ---- tone map (src/renderer.cpp:149-176) -------------------------------------

constexpr int kTmThreads = 256;
constexpr uint32_t kTmMaxBlocks = kTonemapMaxPartials;

__device__ __forceinline__ float log2f_approx(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float exp2f_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ double log_luminance(float r, float g, float b) {
  float const Yl = 0.2126f * r + 0.7152f * g + 0.0722f * b;
  float const y = Yl >= kEps ? Yl : kEps;
  return double(logf(y));
}

// Sum over the block, in thread 0 (the same order for the same values).
__device__ __forceinline__ double block_sum(double s) {
  __shared__ double red[kTmThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kTmThreads / 32; w++) t += red[w];
  return t;
}

// log-average luminance: per-block sums of log(max(Y, ε)) in double, four
// pixels (three 16-byte words) at a time where the image is 16-byte aligned
__global__ void __launch_bounds__(kTmThreads) tm_logsum_kernel(const float* __restrict__ rgb, uint64_t n, bool vec,
                                                               double* __restrict__ partials) {
  // the map kernel may be scheduled as soon as blocks leave; it waits for
  // the sums itself
  cudaTriggerProgrammaticLaunchCompletion();
  uint64_t const t0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x, dt = uint64_t(gridDim.x) * blockDim.x;
  uint64_t const n4 = vec ? n / 4 : 0;
  double s = 0.0;
  const float4* const v = reinterpret_cast<const float4*>(rgb);
  for (uint64_t p = t0; p < n4; p += dt) {
    float4 const a = v[3 * p], b = v[3 * p + 1], c = v[3 * p + 2];
    s += log_luminance(a.x, a.y, a.z);
    s += log_luminance(a.w, b.x, b.y);
    s += log_luminance(b.z, b.w, c.x);
    s += log_luminance(c.y, c.z, c.w);
  }
  for (uint64_t p = 4 * n4 + t0; p < n; p += dt) s += log_luminance(rgb[3 * p], rgb[3 * p + 1], rgb[3 * p + 2]);
  s = block_sum(s);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// tonemapping::koiFilmic (cg.hpp:181-194)
__device__ __forceinline__ float koi_filmic(float L) {
  float const x = 10.f * L;
  return (x * (0.3f * x + 0.14f)) / (x * (0.3f * x + 2.8f) + 10.f);
}
// linRGB2sRGB (cg.hpp:149-154) and float2byte (numli.hpp:105-106)
__device__ __forceinline__ int srgb_byte_exact(float c) {
  float const s = c > 0.0031308f ? 1.055f * powf(c, 1.f / 2.4f) - 0.055f : 12.92f * c;
  int const v = int(255.f * s + 0.5f);
  return v < 0 ? 0 : (v > 255 ? 255 : v);
}
// The same byte: 255 s + 0.5 with the power by the hardware's base-2
// logarithm and exponential, which is within 3e-4 of it for c in (0.003, 1]
// (their relative errors are 2^-22; the logarithm is at most 8.4 in size),
// and powf only where that lies within kByteMargin of a whole number: one
// value in 500.  The whole part by adding 1.5 * 2^23: conversions run on the
// same quarter-rate unit as the logarithm and bounded the kernel.
constexpr float kByteMargin = 0.001f;
__device__ __forceinline__ uint32_t srgb_byte(float c) {
  float const hi = fmaf(269.025f, exp2f_approx(log2f_approx(c) * (1.f / 2.4f)), -13.525f);
  float const v = c > 0.0031308f ? hi : fmaxf(255.f * (12.92f * c) + 0.5f, 0.25f);
  float const m = (v - 0.5f) + 12582912.f;
  float const f = v - (m - 12582912.f);
  // false for NaN, too
  bool const sure = c <= 1.f && fabsf(f - 0.5f) < 0.5f - kByteMargin;
  return sure ? __float_as_uint(m) & 0xFFu : uint32_t(srgb_byte_exact(c));
}

// Exposure from the sums (each block adds them up for itself: 1,184 values
// from L2 cost less than a launch of their own), then tone curve and sRGB
// byte per channel, four channels at a time where all arrays are aligned.
// Bound by issue (69 %; 64 instructions per channel, of which the division
// and the power are most).  1920x1080: 27 + 3 (exposure launch) -> 16 us,
// the call 57 -> 38 us.
__global__ void __launch_bounds__(kTmThreads) tm_map_kernel(const float* __restrict__ rgb, uint64_t n, bool vec,
                                                            const double* __restrict__ partials, uint32_t nb,
                                                            float y_mid, float* __restrict__ out_tm,
                                                            uint8_t* __restrict__ out24) {
  uint64_t const t0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x, dt = uint64_t(gridDim.x) * blockDim.x;
  uint64_t const n4 = vec ? 3 * n / 4 : 0;
  const float4* const in4 = reinterpret_cast<const float4*>(rgb);
  // the first word does not depend on the sums
  float4 v = t0 < n4 ? in4[t0] : make_float4(0.f, 0.f, 0.f, 0.f);
  cudaGridDependencySynchronize();
  __shared__ float exposure;
  double s = 0.0;
  for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) s += partials[b];
  s = block_sum(s);
  if (threadIdx.x == 0) exposure = y_mid / expf(float(s / double(n)));
  __syncthreads();
  float const e = exposure;
  for (uint64_t q = t0; q < n4; q += dt) {
    float4 const next = q + dt < n4 ? in4[q + dt] : v;
    float4 const L = make_float4(koi_filmic(e * v.x), koi_filmic(e * v.y), koi_filmic(e * v.z), koi_filmic(e * v.w));
    if (out_tm) reinterpret_cast<float4*>(out_tm)[q] = L;
    if (out24)
      reinterpret_cast<uint32_t*>(out24)[q] =
          srgb_byte(L.x) | (srgb_byte(L.y) << 8) | (srgb_byte(L.z) << 16) | (srgb_byte(L.w) << 24);
    v = next;
  }
  for (uint64_t q = 4 * n4 + t0; q < 3 * n; q += dt) {
    float const L = koi_filmic(e * rgb[q]);
    if (out_tm) out_tm[q] = L;
    if (out24) out24[q] = uint8_t(srgb_byte(L));
  }
}

}  // namespace

cudaError_t launch_render(const DevScene& S, const RenderArgs& a, WaveState* wave, float* d_out,
                          DevCounters* d_cnt, cudaStream_t st, WaveLaunch* run) {
  if (a.pixel_count == 0) return cudaSuccess;
  switch (S.hero_k) {
    case 4: return launch_render_k<4>(S, a, wave, d_out, d_cnt, st, run);
    case 8: return launch_render_k<8>(S, a, wave, d_out, d_cnt, st, run);
    case 16: return launch_render_k<16>(S, a, wave, d_out, d_cnt, st, run);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_batch(uint32_t hero_k, const JobTable& jobs, uint64_t n_items, uint64_t chunk_items, bool linear,
                         WaveState* wave, DevCounters* d_cnt, cudaStream_t st, WaveLaunch* run) {
  if (jobs.n == 0 || n_items == 0) return cudaSuccess;
  switch (hero_k) {
    case 4: return launch_batch_k<4>(jobs, n_items, chunk_items, linear, wave, d_cnt, st, run);
    case 8: return launch_batch_k<8>(jobs, n_items, chunk_items, linear, wave, d_cnt, st, run);
    case 16: return launch_batch_k<16>(jobs, n_items, chunk_items, linear, wave, d_cnt, st, run);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_adjoint(uint32_t hero_k, const DevScene& S, const RenderArgs& a, WaveState* wave,
                           uint64_t chunk_items, float* d_img, const AdjointArgs& g, DevCounters* d_cnt,
                           cudaStream_t st, WaveLaunch* run) {
  switch (hero_k) {
    case 4: return launch_adjoint_k<4>(S, a, wave, chunk_items, d_img, g, d_cnt, st, run);
    case 8: return launch_adjoint_k<8>(S, a, wave, chunk_items, d_img, g, d_cnt, st, run);
    case 16: return launch_adjoint_k<16>(S, a, wave, chunk_items, d_img, g, d_cnt, st, run);
  }
  return cudaErrorInvalidValue;
}

uint32_t tonemap_partials_needed(uint64_t n_pixels) {
  uint64_t const b = (n_pixels + kTmThreads - 1) / kTmThreads;
  return uint32_t(b < kTmMaxBlocks ? (b ? b : 1) : kTmMaxBlocks);
}

cudaError_t launch_tonemap(const float* d_rgb, uint64_t n_pixels, float y_mid, double* d_partials,
                           uint32_t n_partials, float* d_out_tm, uint8_t* d_out24, cudaStream_t st) {
  uint32_t const nb = tonemap_partials_needed(n_pixels);
  if (n_partials < nb) return cudaErrorInvalidValue;
  auto aligned = [](const void* p, uintptr_t to) { return (reinterpret_cast<uintptr_t>(p) & (to - 1)) == 0; };
  bool const vec_in = aligned(d_rgb, 16), vec = vec_in && aligned(d_out_tm, 16) && aligned(d_out24, 4);
  tm_logsum_kernel<<<nb, kTmThreads, 0, st>>>(d_rgb, n_pixels, vec_in, d_partials);
  uint64_t const mb = ((vec ? (3 * n_pixels + 3) / 4 : 3 * n_pixels) + kTmThreads - 1) / kTmThreads;
  // the map kernel's launch overlaps the sums (it waits for them on the device)
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(uint32_t(mb < kTmMaxBlocks ? (mb ? mb : 1) : kTmMaxBlocks));
  cfg.blockDim = dim3(kTmThreads);
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaError_t const e = cudaLaunchKernelEx(&cfg, tm_map_kernel, d_rgb, n_pixels, vec,
                                           static_cast<const double*>(d_partials), nb, y_mid, d_out_tm, d_out24);
  return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace lgpu
