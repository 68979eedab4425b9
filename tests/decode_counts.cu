// The counts' decode of the sweeps (ptx_counts.cuh) against CUDA's sqrtf on the GPU: all 2^24 floats
// of [1, 4) as the scale of one count, then every count at a list of scales over the whole range,
// one and two counts at a time.  minus_amplitude(0, ...) is the negated amplitude.  Prints the
// number of values compared and of those that differ (a NaN equals a NaN).
#include <cstdio>
#include <vector>

#include "ptx_counts.cuh"

__device__ bool same(float got, float want) { return got == want || (isnan(got) && isnan(want)); }

__global__ void all_mantissas(unsigned long long* bad) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;  // 2^24 threads
  const float x = __uint_as_float(0x3f800000u + i);
  const ptx::CountScale s(x);
  const float2 both = ptx::minus_amplitudes<true>(make_float2(0.f, 0.f), 0x10001u, x);
  const float want = sqrtf(x);
  if (!same(-ptx::minus_amplitude(0.f, 1u, s), want) || !same(-both.x, want) || !same(-both.y, want)) atomicAdd(bad, 1ull);
}

__global__ void all_counts(const float* scales, unsigned long long* bad) {
  const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;  // 2^16 threads in x, one scale per y
  const float scale = scales[blockIdx.y];
  const ptx::CountScale s(scale);
  const unsigned other = 65535u - c;
  const float2 zero = make_float2(0.f, 0.f);
  const float2 both = ptx::plain_scale(scale) ? ptx::minus_amplitudes<true>(zero, c | other << 16, scale)
                                              : ptx::minus_amplitudes<false>(zero, c | other << 16, scale);
  const float want = sqrtf(static_cast<float>(c) * scale), want2 = sqrtf(static_cast<float>(other) * scale);
  if (!same(-ptx::minus_amplitude(0.f, c, s), want) || !same(-both.x, want) || !same(-both.y, want2)) atomicAdd(bad, 1ull);
  // the difference is rounded once
  const float a = 1.25f * want + scale;
  if (!same(ptx::minus_amplitude(a, c, s), a - want)) atomicAdd(bad, 1ull);
}

int main() {
  std::vector<float> scales;
  for (int e = -149; e <= 127; ++e) {
    for (float m : {1.f, 1.9999999f, 1.3333334f, 1.7320508f}) {
      const float v = ldexpf(m, e);
      if (v > 0.f && !isinf(v)) scales.push_back(v);
    }
  }
  for (float v : {1e-45f, 1.1754942e-38f, 1.1754944e-38f, 3.4028235e38f / 65535.f, 3.4028235e38f, INFINITY}) scales.push_back(v);
  const unsigned ns = static_cast<unsigned>(scales.size());
  float* d_scales = nullptr;
  unsigned long long* bad = nullptr;
  unsigned long long host[2] = {0, 0};
  if (cudaMalloc(&d_scales, ns * sizeof(float)) || cudaMalloc(&bad, sizeof(host)) ||
      cudaMemcpy(d_scales, scales.data(), ns * sizeof(float), cudaMemcpyHostToDevice) ||
      cudaMemcpy(bad, host, sizeof(host), cudaMemcpyHostToDevice)) {
    return 1;
  }
  all_mantissas<<<(1u << 24) / 256, 256>>>(bad);
  all_counts<<<dim3(65536 / 256, ns), 256>>>(d_scales, bad + 1);
  if (cudaDeviceSynchronize() || cudaMemcpy(host, bad, sizeof(host), cudaMemcpyDeviceToHost)) return 1;
  std::printf("%u %llu\n%u %llu\n", 1u << 24, host[0], ns * 65536u, host[1]);
  return 0;
}
