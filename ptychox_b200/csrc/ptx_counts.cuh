// Observed amplitudes of photon counts.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx_pairfft.cuh"

namespace ptx {

// The amplitude observed at a detector pixel, sqrt(count scale): a reciprocal square root refined by
// one step of g + (x - g^2) h, h ~ 1 / (2 sqrt x) (P. Markstein, IBM J. Res. Dev. 34, 111 (1990)).
// It is the rounded square root of the rounded product, as sqrtf gives it, where x and the residual
// x - g^2 are normal numbers: for scales of plain_scale (all 2^24 values of [1, 4) and all counts at
// scales over the whole range were compared).  A table of all 65536 counts read by the epilogues
// instead cost their warps the loads' latency (Fourier columns of 225 x 256^2: 65.9 against 59.3 us)
// and each sweep its making.
__host__ __device__ inline bool plain_scale(float scale) { return scale >= 0x1p-64f && scale <= 0x1p64f; }

__device__ __forceinline__ float rsqrt_floor(float x) {  // 1 / sqrt(max(x, the least normal number))
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(fmaxf(x, 1.1754944e-38f)));
  return y;
}
// a - sqrt(count scale) of the two counts of a 32-bit word.  Two compilations, chosen on the host by
// the scale: the factors that minus_amplitude takes for any scale cost the packed columns 3% (225
// frames of 256^2: 167.4 us a sweep, 172.2).
template <bool PLAIN>
__device__ __forceinline__ float2 minus_amplitudes(float2 a, uint32_t counts, float scale) {
  const float2 x = mul2(make_float2(static_cast<float>(counts & 0xffffu), static_cast<float>(counts >> 16)), f2(scale));
  if constexpr (PLAIN) {
    const float2 y = make_float2(rsqrt_floor(x.x), rsqrt_floor(x.y)), g = mul2(x, y);
    return sub2(a, fma2(fma2(neg2(g), g, x), mul2(f2(0.5f), y), g));
  } else {
    return sub2(a, make_float2(sqrtf(x.x), sqrtf(x.y)));
  }
}

// For one count at a time: a scale outside plain_scale is taken by a power of four nearer to 1 and the
// root brought back: sqrt(count scale) = -minus_down (up root(count in)).  `up` reaches infinity
// exactly where the product count scale does.  Made on the host: as kernel arguments the factors are
// constant operands and hold no registers.
struct CountScale {
  float in, up, minus_down;
  CountScale() = default;
  __host__ __device__ CountScale(float scale) : in(scale), up(1.f), minus_down(-1.f) {
    if (scale < 0x1p-64f) {
      in = scale * 0x1p64f;
      minus_down = -0x1p-32f;
    } else if (scale > 3.4028235e38f) {  // every count above 0 is infinite, 0 a NaN
      in = 1.f;
      up = scale;
    } else if (scale > 0x1p64f) {
      in = scale * 0x1p-64f;
      up = 0x1p96f;
      minus_down = -0x1p-64f;
    }
  }
};
// a - sqrt(count scale)
__device__ __forceinline__ float minus_amplitude(float a, uint32_t count, const CountScale& s) {
  const float x = static_cast<float>(count) * s.in;
  const float y = rsqrt_floor(x), g = x * y;
  return fmaf(s.minus_down, s.up * fmaf(fmaf(-g, g, x), 0.5f * y, g), a);
}

}  // namespace ptx
