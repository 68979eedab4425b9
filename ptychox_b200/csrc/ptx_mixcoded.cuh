// Coded and near-field ptychography passes for field sides that are {2,3,5}-smooth but not
// powers of two, on the mixed-radix register FFT (ptx_mixfft.cuh).
//
// Same math, seven-pass structure and workspace layout as the power-of-two coded kernels
// (ptx_coded.cu; python/ptychoX/coded/ops.py:136-171, the adjoint in the step order of
// coded_kernel.cu:347-424).  Row passes that run two transforms (2, 4, 6) take the line from
// the space layout to the frequency layout with the inverse DFT, apply their pointwise step
// there (where thread u < A holds spatial columns u + A k) and return with the forward DFT;
// single-transform column passes (1, 7) store or consume the frequency layout directly.
// Signed frequencies follow numpy's fftfreq for odd sides too (k <= (n - 1) / 2 is
// non-negative).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <stdint.h>

#include "ptx_mix.cuh"

namespace ptx {
namespace mixcoded {

using mixk::ColCfg;
using mixk::RowCfg;

constexpr float kAmpFloor = 1e-30f;  // keeps g / A finite when a pooled amplitude is exactly 0

// numpy fftfreq(n) * n: k for k <= (n - 1) / 2, k - n above
__device__ __forceinline__ int signed_freq(int k, int n) { return k <= (n - 1) / 2 ? k : k - n; }

// exp(2 pi i (dx fx + dy fy)) for signed integer frequencies fx, fy: the argument reduced
// exactly in FP32 (FMA two-product remainders, integer turns removed) before sincospif.
__device__ __forceinline__ float2 shift_ramp(float dx, float dy, int fx, int fy) {
  const float ffx = static_cast<float>(fx), ffy = static_cast<float>(fy);
  const float px = dx * ffx, py = dy * ffy;
  const float ex = fmaf(dx, ffx, -px), ey = fmaf(dy, ffy, -py);
  const float t = (px - rintf(px)) + (py - rintf(py)) + (ex + ey);
  float s, c;
  sincospif(2.0f * t, &s, &c);
  return make_float2(c, s);
}

template <int N>
__device__ __forceinline__ size_t frame_elem(int f, int r, int c) {
  return ((size_t)f * num_tiles(N) + c / kTile) * N * kTile + (size_t)r * kTile + (c % kTile);
}

// All passes are persistent: work units (strip of 8 columns or group of rows, frame) in
// frame-fastest order over one wave of resident CTAs, CTA b taking the contiguous units
// [u0, u1).  A unit's data lands by cp.async in the exchange buffer once the previous unit's last
// exchange has been read, so it arrives while that unit finishes, and the twiddles sit in shared
// memory.  A CTA per unit with loads on demand and twiddles from global memory left the passes
// waiting for memory; per sweep of 32 near-field frames of 960^2 with the shift gradient (us):
//   pass         1    2    3    4    5    6    7    all
//   before     153  229  166  274  166  434  167   1590
//   now         97  171  169  246  172  189  144   1190
// DRAM alone would take 36 to 110 each.  What bounds them is the latency between the steps of a
// line at 8 to 16 warps per SM (registers: up to 32 complex values a thread): 40 to 45% of the
// issue slots and 35 to 39% of the FMA pipe are busy.

// A thread's index, taken anew for each unit: quotients and addresses that follow from it (a
// value per DFT element) stay within the unit; kept across units they spill.
__device__ __forceinline__ int this_unit(int v) {
  asm volatile("" : "+r"(v));
  return v;
}

// Units of a CTA and the walk over them
struct Units {
  long long u, end;
  int group, frame, nframes;
  __device__ __forceinline__ Units(int groups, int nf) : nframes(nf) {
    const long long total = (long long)groups * nf;
    u = total * blockIdx.x / gridDim.x;
    end = total * (blockIdx.x + 1) / gridDim.x;
    group = static_cast<int>(u / nf);
    frame = static_cast<int>(u - (long long)group * nf);
  }
  __device__ __forceinline__ bool more() const { return u < end; }
  __device__ __forceinline__ void next() {
    ++u;
    if (++frame == nframes) {
      frame = 0;
      ++group;
    }
  }
};

// The one twiddle table of a CTA, tw[u * P + t] = exp(-2 pi i t u / N) at the odd pitch P
template <int N>
struct Twiddles {
  using S = mix::Shape<N>;
  static constexpr int SIZE = (S::A * S::P + 1) / 2 * 2;
  static __device__ __forceinline__ void load(float2* dst, const float2* __restrict__ twt) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) dst[i / S::B * S::P + i % S::B] = __ldg(twt + i);
  }
};

// ---- column passes ----------------------------------------------------------------------
// STAGE 1: load O^ T1 R, inverse column DFT, store.  STAGE 3: forward DFT, x T2 (CONJ: x
// conj(T2) / n), inverse DFT, store.  STAGE 7: forward DFT, / n, grad += . conj(R) (float2
// atomics; T1's conjugate follows in the spectrum gradient's own transform) and, with
// grad_shifts, dL/d(dx, dy) += -2 pi sum (fx, fy) Im(conj(G) u).
template <int N>
struct StripCfg {
  using CC = ColCfg<N>;
  static constexpr int C = CC::C, THREADS = CC::THREADS;
  static constexpr int STRIPS = (N + C - 1) / C;
  static constexpr int BUF = ((CC::BUF > N * C ? CC::BUF : N * C) + 1) / 2 * 2;
  static constexpr int TAB = (N + 1) / 2 * 2;
  // exchange buffer, twiddles, two y ramps
  static constexpr int smem(bool table) {
    return (BUF + Twiddles<N>::SIZE + (table ? 2 * TAB : 0)) * (int)sizeof(float2);
  }
  // 16 warps per SM where the line's values leave the registers
  static constexpr int BLOCKS = CC::B <= 32 ? (THREADS <= 256 ? 512 / THREADS : 1) : 1;
};

template <int STAGE, bool CONJ, bool TABLE, int N>
__global__ void __launch_bounds__(StripCfg<N>::THREADS, StripCfg<N>::BLOCKS > 2 ? 2 : StripCfg<N>::BLOCKS)
    mix_coded_cols(MixCodedArgs a) {
  pdl_wait();
  using Cfg = ColCfg<N>;
  using Strip = StripCfg<N>;
  constexpr int A = Cfg::A, B = Cfg::B, C = Cfg::C;
  constexpr bool kRamp = STAGE != 3;
  extern __shared__ __align__(16) float2 sm[];
  float2* tws = sm + Strip::BUF;
  float2* rys = tws + Twiddles<N>::SIZE;  // [2][TAB], TABLE only
  const int tid = threadIdx.x;
  const int t0 = tid / C;
  const int c = tid - t0 * C;
  constexpr int kSubs = kTile / C;
  Units it(Strip::STRIPS, a.nframes);
  if (!it.more()) return;
  Twiddles<N>::load(tws, a.twt);
  float2* buf = sm + c;
  const uint64_t pol = STAGE == 1 ? policy_evict_last() : policy_evict_first();
  auto strip_at = [&](int strip, int f) {
    return a.scratch + ((size_t)f * num_tiles(N) + strip / kSubs) * N * kTile + (strip % kSubs) * C;
  };
  auto request = [&](int strip, int f, int slot) {
    if (STAGE == 1 && (N % 2 || (N % C && strip == Strip::STRIPS - 1))) {
      // odd rows start off 16 bytes, a last strip ends early: single elements
      for (int i = tid; i < N * C; i += Strip::THREADS) {
        const int r = i / C, q = i % C;
        if (strip * C + q < N) cp_async8_hint(sm + i, a.ospec + (size_t)r * N + strip * C + q, pol);
      }
    } else {
      const float2* src = STAGE == 1 ? a.ospec + strip * C : strip_at(strip, f);
      constexpr int pitch = STAGE == 1 ? N : kTile;
#pragma unroll 4
      for (int i = tid; i < N * C / 2; i += Strip::THREADS) {
        const int r = i / (C / 2), q = i % (C / 2);
        cp_async16_hint(sm + 2 * i, src + (size_t)r * pitch + 2 * q, pol);
      }
    }
    if constexpr (kRamp && TABLE) {
      const float2* ry = a.ramps + ((size_t)2 * f + 1) * N;
      for (int i = tid; i < N; i += Strip::THREADS) cp_async8(rys + slot * Strip::TAB + i, ry + i);
    }
    cp_async_commit();
  };
  request(it.group, it.frame, 0);
  for (int slot = 0; it.more(); slot ^= 1) {
    const int strip = it.group, f = it.frame, t = this_unit(t0);
    const int kc = strip * C + c;
    const bool col_ok = N % C == 0 || kc < N;
    const int fx = signed_freq(kc, N);
    float2 ex = make_float2(1.f, 0.f);
    float dx = 0.f, dy = 0.f;
    if constexpr (kRamp) {
      if constexpr (TABLE) {
        if (col_ok) ex = __ldg(&a.ramps[(size_t)2 * f * N + kc]);
      } else {
        dx = a.shifts[2 * f];
        dy = a.shifts[2 * f + 1];
      }
    }
    auto ramp = [&](int kr) {
      if constexpr (TABLE) {
        return cmul(ex, rys[slot * Strip::TAB + kr]);
      } else {
        return shift_ramp(dx, dy, fx, signed_freq(kr, N));
      }
    };
    cp_async_wait_all();
    __syncthreads();
    float2 y[A];
#pragma unroll
    for (int j = 0; j < A; ++j) {
      const int kr = t + B * j;
      y[j] = col_ok ? sm[kr * C + c] : make_float2(0.f, 0.f);
      if constexpr (STAGE == 1) y[j] = cmul(y[j], ramp(kr));
    }
    __syncthreads();  // the strip is read
    mix::fwd_step1<N, Cfg::RS, C, STAGE == 1, Cfg::S::P>(y, buf, t, tws);
    __syncthreads();
    float2 z[B];
    if (t < A) mix::fwd_step2<N, Cfg::RS, C, STAGE == 1>(z, buf, t);
    if constexpr (STAGE == 3) {
      if (t < A) {
#pragma unroll
        for (int k = 0; k < B; ++k) {
          if (col_ok) {
            const float2 h = __ldg(&a.t2[(size_t)(t + A * k) * N + kc]);
            z[k] = CONJ ? cscale(cmulc(z[k], h), a.inv_n) : cmul(z[k], h);
          }
        }
        // thread u wrote and reads only row u of the exchange buffer since the barrier
        mix::inv_step1<N, Cfg::RS, C, true, Cfg::S::P>(z, buf, t, tws);
      }
      __syncthreads();
      mix::inv_step2<N, Cfg::RS, C, true>(y, buf, t);
    }
    __syncthreads();  // the exchange is read
    it.next();
    if (it.more()) request(it.group, it.frame, slot ^ 1);
    if constexpr (STAGE == 3) {
      float2* out = strip_at(strip, f);
      if (col_ok) {
#pragma unroll
        for (int j = 0; j < A; ++j) out[(t + B * j) * kTile + c] = y[j];
      }
    } else if constexpr (STAGE == 1) {
      float2* out = strip_at(strip, f);
      if (t < A && col_ok) {
#pragma unroll
        for (int k = 0; k < B; ++k) out[(t + A * k) * kTile + c] = z[k];
      }
    } else {
      float sx = 0.f, sy = 0.f;
      if (t < A && col_ok) {
#pragma unroll
        for (int k = 0; k < B; ++k) {
          const int kr = t + A * k;
          const size_t idx = (size_t)kr * N + kc;
          const float2 w = ramp(kr);
          const float2 G = cscale(z[k], a.inv_n);
          atomicAdd(&a.grad_ospec[idx], cmulc(G, w));
          if (a.grad_shifts) {
            const float2 u = cmul(a.ospec[idx], w);
            const float im = fmaf(G.x, u.y, -G.y * u.x);  // Im(conj(G) u)
            sx = fmaf(static_cast<float>(fx), im, sx);
            sy = fmaf(static_cast<float>(signed_freq(kr, N)), im, sy);
          }
        }
      }
      if (a.grad_shifts) {
        constexpr double kTwoPi = 6.283185307179586476925286766559;
        block_add_double(static_cast<double>(sx), -kTwoPi, &a.grad_shifts[2 * f]);
        block_add_double(static_cast<double>(sy), -kTwoPi, &a.grad_shifts[2 * f + 1]);
      }
    }
  }
}

// ---- row passes ----------------------------------------------------------------------------
// Up to 128 threads, B per line, so that three CTAs of pass 2 fit an SM (two with 256 threads: 193
// us against 171); a line's frame row lands in its exchange buffer.
template <int N>
struct CodedRows {
  using RC = RowCfg<N>;
  static constexpr int A = RC::A, B = RC::B;
  static constexpr int LINES = 128 / B > 0 ? 128 / B : 1;
  // line buffers: an exchange or a landing row, 16-byte aligned
  static constexpr int NEED = RC::BUF > N + 1 ? RC::BUF : N + 1;
  static constexpr int BUF = (NEED + 1) / 2 * 2;
  static constexpr int ROW = (N + 1) / 2 * 2;
  static constexpr int smem(int lines, int rows) { return (lines * (BUF + rows * ROW) + Twiddles<N>::SIZE) * (int)sizeof(float2); }
};

// Frame row r of frame f into dst[0, N) (or, of a natural array, src[0, N)) by the line's B threads.
template <int N>
__device__ __forceinline__ void land_frame_row(float2* dst, const float2* scratch, int f, int r, int t, uint64_t pol) {
  constexpr int B = RowCfg<N>::B;
  const float2* base = scratch + (size_t)f * num_tiles(N) * N * kTile + (size_t)r * kTile;
#pragma unroll 4
  for (int i = t; i < (N + 1) / 2; i += B) {  // an odd row's last pair ends in the tile's padding
    const int c = 2 * i;
    cp_async16_hint(dst + c, base + (size_t)(c / kTile) * N * kTile + (c % kTile), pol);
  }
  cp_async_commit();
}
// A row src[0, N): in pairs where it starts on 16 bytes (odd sides: every other one), else one
// element at a time.
template <int N>
__device__ __forceinline__ void land_row(float2* dst, const float2* src, int t, uint64_t pol) {
  constexpr int B = RowCfg<N>::B;
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll 4
    for (int i = t; i < N / 2; i += B) cp_async16_hint(dst + 2 * i, src + 2 * i, pol);
    if (N % 2 && t == 0) cp_async8_hint(dst + N - 1, src + N - 1, pol);
  } else {
    for (int i = t; i < N; i += B) cp_async8_hint(dst + i, src + i, pol);
  }
  cp_async_commit();
}

// Pass 2: inverse row DFT, x = . / n (stored to xstore), a = x M, forward row DFT.
template <int N>
__global__ void __launch_bounds__(CodedRows<N>::LINES * CodedRows<N>::B, CodedRows<N>::B <= 32 ? 3 : 2)
    mix_coded_rows_mask(MixCodedArgs a, int lines) {
  pdl_wait();
  using Cfg = RowCfg<N>;
  using R = CodedRows<N>;
  constexpr int A = Cfg::A, B = Cfg::B;
  extern __shared__ __align__(16) float2 sm[];
  const int tid = threadIdx.x;
  const int l = tid / B;
  const int t0 = tid - l * B;
  float2* buf = sm + l * R::BUF;
  float2* mbuf = sm + lines * R::BUF + l * R::ROW;
  float2* tws = sm + lines * (R::BUF + R::ROW);
  Units it((N + lines - 1) / lines, a.nframes);
  if (!it.more()) return;
  Twiddles<N>::load(tws, a.twt);
  const uint64_t pol_first = policy_evict_first();
  int group = -1;
  if (it.group * lines + l < N) land_frame_row<N>(buf, a.scratch, it.frame, it.group * lines + l, t0, pol_first);
  while (it.more()) {
    const int t = this_unit(t0);
    const int f = it.frame, r = it.group * lines + l;
    const bool row_ok = r < N;
    if (it.group != group) {
      group = it.group;
      // read back by the thread's own lanes of the frequency layout after the next barrier
      if (row_ok) {
        for (int c = t; c < N; c += B) mbuf[c] = __ldg(&a.mask[(size_t)r * N + c]);
      }
    }
    cp_async_wait_all();
    __syncthreads();
    float2 y[A];
#pragma unroll
    for (int j = 0; j < A; ++j) y[j] = row_ok ? buf[t + B * j] : make_float2(0.f, 0.f);
    __syncthreads();  // the landing rows are read
    mix::fwd_step1<N, Cfg::P, 1, true, Cfg::P>(y, buf, t, tws);
    __syncthreads();
    if (t < A) {
      float2 z[B];
      mix::fwd_step2<N, Cfg::P, 1, true>(z, buf, t);
      float2* xrow = a.xstore + ((size_t)f * N + (row_ok ? r : 0)) * N;
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const int c = t + A * k;
        const float2 x = cscale(z[k], a.inv_n);
        if (row_ok) xrow[c] = x;
        z[k] = cmul(x, mbuf[c]);
      }
      mix::inv_step1<N, Cfg::P, 1, false, Cfg::P>(z, buf, t, tws);
    }
    __syncthreads();
    mix::inv_step2<N, Cfg::P, 1, false>(y, buf, t);
    __syncthreads();  // the exchange rows are read
    it.next();
    if (it.more() && it.group * lines + l < N) {
      land_frame_row<N>(buf, a.scratch, it.frame, it.group * lines + l, t, pol_first);
    }
    if (row_ok) {
#pragma unroll
      for (int j = 0; j < A; ++j) a.scratch[frame_elem<N>(f, r, t + B * j)] = y[j];
    }
  }
}

// Pass 4; `lines` a multiple of ds.  kMixColSweep: inverse row DFT, s = . / n, RMS pool over ds x
// ds, FP64 loss, g_s = gA / (A ds^2) s, forward row DFT.  kMixColForward: inverse row DFT, write
// s and the pooled amplitude.  kMixColBackward: g_s from the saved s, amplitude and grad_output,
// forward DFT.
template <int MODE, int N>
__global__ void __launch_bounds__(512) mix_coded_rows_pool(MixCodedArgs a, int lines) {
  pdl_wait();
  using Cfg = RowCfg<N>;
  using R = CodedRows<N>;
  constexpr int A = Cfg::A, B = Cfg::B;
  extern __shared__ __align__(16) float2 sm[];
  float2* tws = sm + lines * R::BUF;
  float* pool = reinterpret_cast<float*>(tws + Twiddles<N>::SIZE);  // [lines][N] |s|^2
  float* factor = pool + lines * N;                        // per pooled pixel
  const int tid = threadIdx.x;
  const int l = tid / B;
  const int t0 = tid - l * B;
  const int lw = N / a.ds;
  // c / ds = c inv_ds >> 20 for c, ds < 1024: c (inv_ds ds - 2^20) <= 1023^2 < 2^20
  const int inv_ds = ((1 << 20) + a.ds - 1) / a.ds;
  float2* buf = sm + l * R::BUF;
  Units it((N + lines - 1) / lines, a.nframes);
  Twiddles<N>::load(tws, a.twt);
  if (MODE == kMixColBackward) __syncthreads();
  const uint64_t pol_first = policy_evict_first();
  double acc = 0.0;
  if (MODE != kMixColBackward && it.more() && it.group * lines + l < N) {
    land_frame_row<N>(buf, a.scratch, it.frame, it.group * lines + l, t0, pol_first);
  }
  while (it.more()) {
    const int t = this_unit(t0);
    const int f = it.frame, r0 = it.group * lines, r = r0 + l;
    const bool row_ok = r < N;
    const size_t g = (size_t)a.frame0 + f;
    const int ds = this_unit(a.ds);
    const int per = this_unit(inv_ds);
    auto block_of = [&](int c) { return c * per >> 20; };
    const int nb = min(lines / ds, lw - r0 / ds) * lw;
    const size_t block0 = (g * lw + r0 / ds) * lw;
    float2 z[B];
    if (MODE == kMixColBackward) {
      if (t < A) {
        const int rr = row_ok ? r : 0;
        const float2* srow = a.sensor + (g * N + rr) * N;
        const float* arow = a.amplitude + (g * lw + rr / ds) * lw;
        const float* grow = a.grad_output + (g * lw + rr / ds) * lw;
#pragma unroll
        for (int k = 0; k < B; ++k) {
          const int c = t + A * k;
          const float am = fmaxf(arow[block_of(c)], kAmpFloor);
          z[k] = row_ok ? cscale(srow[c], grow[block_of(c)] / (am * static_cast<float>(ds * ds))) : make_float2(0.f, 0.f);
        }
      }
    } else {
      uint16_t first = 0;  // the count of the thread's first block, on its way meanwhile
      if (MODE == kMixColSweep && tid < nb) first = __ldg(a.measured + block0 + tid);
      cp_async_wait_all();
      __syncthreads();
      float2 y[A];
#pragma unroll
      for (int j = 0; j < A; ++j) y[j] = row_ok ? buf[t + B * j] : make_float2(0.f, 0.f);
      __syncthreads();  // the landing rows are read
      mix::fwd_step1<N, Cfg::P, 1, true, Cfg::P>(y, buf, t, tws);
      __syncthreads();
      if (t < A) {
        mix::fwd_step2<N, Cfg::P, 1, true>(z, buf, t);
#pragma unroll
        for (int k = 0; k < B; ++k) {
          z[k] = cscale(z[k], a.inv_n);
          pool[l * N + t + A * k] = cabs2(z[k]);
        }
      }
      __syncthreads();
      // pooled values of this unit's rows: (lines / ds) x lw blocks, contiguous in the output
      for (int q = tid; q < nb; q += blockDim.x) {
        const int py = q / lw, px = q - py * lw;
        float sum = 0.f;
        for (int yy = 0; yy < ds; ++yy) {
          const float* row = pool + (py * ds + yy) * N + px * ds;
          if (ds % 4 == 0) {  // rows and blocks then start on 16 bytes
            for (int xx = 0; xx < ds; xx += 4) {
              const float4 v = *reinterpret_cast<const float4*>(row + xx);
              sum = ((sum + v.x) + v.y + v.z) + v.w;
            }
          } else if (ds % 2 == 0) {
            for (int xx = 0; xx < ds; xx += 2) {
              const float2 v = *reinterpret_cast<const float2*>(row + xx);
              sum = (sum + v.x) + v.y;
            }
          } else {
            for (int xx = 0; xx < ds; ++xx) sum += row[xx];
          }
        }
        const float am = sqrtf(fmaxf(sum / static_cast<float>(ds * ds), 0.f));
        const size_t oidx = block0 + q;
        if (MODE == kMixColForward) {
          a.amplitude[oidx] = am;
        } else {
          const float d = am - sqrtf(static_cast<float>(q == tid ? first : __ldg(a.measured + oidx)) * a.scale);
          acc += static_cast<double>(d) * static_cast<double>(d);
          // the factor gA / (A ds^2) of the block
          factor[q] = a.grad_scale * d / (fmaxf(am, kAmpFloor) * static_cast<float>(ds * ds));
        }
      }
      __syncthreads();
    }
    if (MODE == kMixColForward) {
      it.next();
      if (it.more() && it.group * lines + l < N) {
        land_frame_row<N>(buf, a.scratch, it.frame, it.group * lines + l, t, pol_first);
      }
      if (t < A && row_ok) {
        float2* srow = a.sensor + (g * N + r) * N;
#pragma unroll
        for (int k = 0; k < B; ++k) srow[t + A * k] = z[k];
      }
      continue;
    }
    if (t < A) {
      if (MODE == kMixColSweep) {
#pragma unroll
        for (int k = 0; k < B; ++k) {
          z[k] = row_ok ? cscale(z[k], factor[(l / ds) * lw + block_of(t + A * k)]) : make_float2(0.f, 0.f);
        }
      }
      mix::inv_step1<N, Cfg::P, 1, false, Cfg::P>(z, buf, t, tws);
    }
    __syncthreads();
    float2 y[A];
    mix::inv_step2<N, Cfg::P, 1, false>(y, buf, t);
    __syncthreads();  // the exchange rows are read
    it.next();
    if (MODE != kMixColBackward && it.more() && it.group * lines + l < N) {
      land_frame_row<N>(buf, a.scratch, it.frame, it.group * lines + l, t, pol_first);
    }
    if (row_ok) {
#pragma unroll
      for (int j = 0; j < A; ++j) a.scratch[frame_elem<N>(f, r, t + B * j)] = y[j];
    }
  }
  if (MODE == kMixColSweep) block_add_double(acc, a.inv_numel, a.loss);
}

// Pass 6: inverse row DFT (g_a), grad_M += g_a conj(x), g_a conj(M), forward DFT.  The mask
// gradient accumulates in registers over a row group's frames (thread u < A holds B columns of its
// row) and leaves with one float2 atomic per element when the CTA leaves the group: an atomic per
// element and frame was most of the pass's 434 us.  (The spectrum gradient of pass 7 gained
// nothing from the same, 144 us either way: its accumulators cost it half its warps.)
template <int N>
__global__ void __launch_bounds__(CodedRows<N>::LINES * CodedRows<N>::B, 2)
    mix_coded_rows_grad_mask(MixCodedArgs a, int lines) {
  pdl_wait();
  using Cfg = RowCfg<N>;
  using R = CodedRows<N>;
  constexpr int A = Cfg::A, B = Cfg::B;
  extern __shared__ __align__(16) float2 sm[];
  const int tid = threadIdx.x;
  const int l = tid / B;
  const int t0 = tid - l * B;
  float2* buf = sm + l * R::BUF;
  float2* mbuf = sm + lines * R::BUF + l * R::ROW;
  float2* xbuf = sm + lines * (R::BUF + R::ROW) + l * R::ROW;
  float2* tws = sm + lines * (R::BUF + 2 * R::ROW);
  Units it((N + lines - 1) / lines, a.nframes);
  if (!it.more()) return;
  Twiddles<N>::load(tws, a.twt);
  const uint64_t pol_first = policy_evict_first();
  float2 acc[B];
#pragma unroll
  for (int k = 0; k < B; ++k) acc[k] = make_float2(0.f, 0.f);
  int group = -1;
  auto land = [&](int t) {
    const int r = it.group * lines + l;
    if (r < N) {
      land_frame_row<N>(buf, a.scratch, it.frame, r, t, pol_first);
      land_row<N>(xbuf, a.xstore + ((size_t)it.frame * N + r) * N, t, pol_first);  // the stored x row
    }
  };
  land(t0);
  while (it.more()) {
    const int t = this_unit(t0);
    const int f = it.frame, r = it.group * lines + l;
    const bool row_ok = r < N;
    if (it.group != group) {
      group = it.group;
      if (row_ok) {
        for (int c = t; c < N; c += B) mbuf[c] = __ldg(&a.mask[(size_t)r * N + c]);
      }
    }
    cp_async_wait_all();
    __syncthreads();
    float2 y[A];
#pragma unroll
    for (int j = 0; j < A; ++j) y[j] = row_ok ? buf[t + B * j] : make_float2(0.f, 0.f);
    __syncthreads();  // the landing rows are read
    mix::fwd_step1<N, Cfg::P, 1, true, Cfg::P>(y, buf, t, tws);
    __syncthreads();
    if (t < A) {
      float2 z[B];
      mix::fwd_step2<N, Cfg::P, 1, true>(z, buf, t);
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const int c = t + A * k;
        if (row_ok) acc[k] = cadd(acc[k], cmulc(z[k], xbuf[c]));
        z[k] = cmulc(z[k], mbuf[c]);
      }
      mix::inv_step1<N, Cfg::P, 1, false, Cfg::P>(z, buf, t, tws);
    }
    __syncthreads();
    mix::inv_step2<N, Cfg::P, 1, false>(y, buf, t);
    __syncthreads();  // the exchange rows are read
    it.next();
    if (it.more()) land(t);
    if (row_ok) {
#pragma unroll
      for (int j = 0; j < A; ++j) a.scratch[frame_elem<N>(f, r, t + B * j)] = y[j];
    }
    if (!it.more() || it.group != group) {
      if (row_ok && t < A) {
        float2* grow = a.grad_mask + (size_t)r * N;
#pragma unroll
        for (int k = 0; k < B; ++k) {
          atomicAdd(&grow[t + A * k], acc[k]);
          acc[k] = make_float2(0.f, 0.f);
        }
      }
    }
  }
}

// ---- launchers --------------------------------------------------------------------------

template <int N>
struct Ops {
  using RC = RowCfg<N>;
  using R = CodedRows<N>;
  using Strip = StripCfg<N>;
  static int row_lines() { return std::min(R::LINES, N); }
  // rows per CTA of pass 4: a multiple of ds, 0 when ds rows of B threads exceed the
  // kernel's 512-thread bound
  static int pool_lines(int ds) {
    if (ds < 1 || N % ds != 0 || ds * RC::B > 512) return 0;
    return ds * std::max(1, RC::LINES / ds);
  }
  static int pool_smem(int lines, int ds) {
    return R::smem(lines, 0) + (lines * N + (lines / ds) * (N / ds)) * (int)sizeof(float);
  }
  static int prepare(int ds) {
    const int pl = pool_lines(ds);
    if (pl == 0) return set_error(PTX_ERR_UNSUPPORTED_SIZE, "downsample %d too large for field side %d", ds, N);
    int st = ensure_smem((const void*)mix_coded_cols<1, false, false, N>, Strip::smem(false));
    if (!st) st = ensure_smem((const void*)mix_coded_cols<1, false, true, N>, Strip::smem(true));
    if (!st) st = ensure_smem((const void*)mix_coded_cols<3, false, false, N>, Strip::smem(false));
    if (!st) st = ensure_smem((const void*)mix_coded_cols<3, true, false, N>, Strip::smem(false));
    if (!st) st = ensure_smem((const void*)mix_coded_cols<7, false, false, N>, Strip::smem(false));
    if (!st) st = ensure_smem((const void*)mix_coded_cols<7, false, true, N>, Strip::smem(true));
    if (!st) st = ensure_smem((const void*)mix_coded_rows_mask<N>, R::smem(row_lines(), 1));
    if (!st) st = ensure_smem((const void*)mix_coded_rows_grad_mask<N>, R::smem(row_lines(), 2));
    if (!st) st = ensure_smem((const void*)mix_coded_rows_pool<kMixColSweep, N>, pool_smem(pl, ds));
    if (!st) st = ensure_smem((const void*)mix_coded_rows_pool<kMixColForward, N>, pool_smem(pl, ds));
    if (!st) st = ensure_smem((const void*)mix_coded_rows_pool<kMixColBackward, N>, pool_smem(pl, ds));
    return st;
  }
  static void cols(int stage, bool conj, const MixCodedArgs& a, cudaStream_t s) {
    if (a.nframes <= 0) return;
    auto run = [&](auto kern, bool table) {
      const int smem = Strip::smem(table);
      const int grid = persistent_grid((const void*)kern, Strip::THREADS, smem, (long long)Strip::STRIPS * a.nframes);
      launch_pdl(kern, grid, Strip::THREADS, smem, s, a);
    };
    if (stage == 1) {
      if (a.ramps) run(mix_coded_cols<1, false, true, N>, true);
      else run(mix_coded_cols<1, false, false, N>, false);
    } else if (stage == 3) {
      if (conj) run(mix_coded_cols<3, true, false, N>, false);
      else run(mix_coded_cols<3, false, false, N>, false);
    } else {
      if (a.ramps) run(mix_coded_cols<7, false, true, N>, true);
      else run(mix_coded_cols<7, false, false, N>, false);
    }
  }
  template <typename K>
  static void run_rows(K kern, int lines, int smem, const MixCodedArgs& a, cudaStream_t s) {
    if (a.nframes <= 0) return;
    const int threads = lines * RC::B;
    const int grid = persistent_grid((const void*)kern, threads, smem, (long long)((N + lines - 1) / lines) * a.nframes);
    launch_pdl(kern, grid, threads, smem, s, a, lines);
  }
  static void rows_mask(const MixCodedArgs& a, cudaStream_t s) {
    run_rows(mix_coded_rows_mask<N>, row_lines(), R::smem(row_lines(), 1), a, s);
  }
  static void rows_grad_mask(const MixCodedArgs& a, cudaStream_t s) {
    run_rows(mix_coded_rows_grad_mask<N>, row_lines(), R::smem(row_lines(), 2), a, s);
  }
  static void rows_pool(int mode, const MixCodedArgs& a, cudaStream_t s) {
    const int lines = pool_lines(a.ds), smem = pool_smem(lines, a.ds);
    if (mode == kMixColSweep) {
      run_rows(mix_coded_rows_pool<kMixColSweep, N>, lines, smem, a, s);
    } else if (mode == kMixColForward) {
      run_rows(mix_coded_rows_pool<kMixColForward, N>, lines, smem, a, s);
    } else {
      run_rows(mix_coded_rows_pool<kMixColBackward, N>, lines, smem, a, s);
    }
  }
  static const MixCodedOps* table() {
    static const MixCodedOps ops{&prepare, &cols, &rows_mask, &rows_pool, &rows_grad_mask};
    return &ops;
  }
};

}  // namespace mixcoded
}  // namespace ptx
