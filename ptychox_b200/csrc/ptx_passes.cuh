// Pieces shared by the modality kernels built on the register FFT: launch shapes, the
// FP64 block reduction of loss partials, and generic 2-D transform passes between a
// natural row-major array and the tiled frame layout [tile][row][16].
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <stdint.h>

#include "ptx_counts.cuh"
#include "ptx_internal.h"
#include "ptx_pairfft.cuh"
#include "ptx_pipering.h"
#include "ptx_regfft.cuh"

namespace ptx {

constexpr float kEpsF32 = 1.1920928955078125e-07f;  // torch.finfo(float32).eps
constexpr int kColsPerCta = 8;                        // columns per column-pass CTA

// Copy the N-element row `src` (float2, 8-byte aligned) into `dst` with 16-byte cp.async
// that bypasses L1, element c landing at dst[c + s], s = 1 when src sits 8 bytes past a
// 16-byte boundary (dst must be 16-byte aligned and hold N + 2 elements).  A shifted row
// copies its first and last elements singly so no access leaves the row.  Thread t of the
// T threads of a line copies chunks t + T i; the caller commits, waits and then meets the
// other lanes at a barrier before reading.
template <int N>
__device__ __forceinline__ void copy_row_shifted(float2* dst, const float2* src, int s, int t, uint64_t pol) {
  using S = RegShape<N>;
  if (s == 0) {
#pragma unroll
    for (int i = 0; i < S::N1 / 2; ++i) {
      const int c = 2 * (t + S::T * i);
      cp_async16_hint(dst + c, src + c, pol);
    }
  } else {
#pragma unroll
    for (int i = 0; i < S::N1 / 2; ++i) {
      const int c = 1 + 2 * (t + S::T * i);
      if (c + 1 < N) cp_async16_hint(dst + c + 1, src + c, pol);
    }
    if (t == 0) cp_async8_hint(dst + 1, src, pol);
    if (t == S::T - 1) cp_async8_hint(dst + N, src + N - 1, pol);
  }
}
// 8-byte offset of p from a 16-byte boundary, in float2 elements (0 or 1)
__device__ __forceinline__ int half_shift(const float2* p) {
  return static_cast<int>((reinterpret_cast<uintptr_t>(p) >> 3) & 1);
}

template <int N>
struct RowPass {
  static constexpr int T = RegShape<N>::T;
  static constexpr int LP = row_line_pitch<N>();
  // rows per CTA (a whole number of warps)
  __host__ static int lines(int threads, int rows) {
    int l = threads / T;
    if (l < 1) l = 1;
    const int quantum = T >= 32 ? 1 : 32 / T;
    const int need = ((rows + quantum - 1) / quantum) * quantum;
    return l < need ? l : need;
  }
  __host__ static int smem(int lines) { return lines * LP * (int)sizeof(float2); }
  // exchange buffers plus one prefetched row of N complex values per line
  __host__ static int smem_with_row(int lines) { return lines * (LP + N) * (int)sizeof(float2); }
};

template <int N>
struct ColPass {
  static constexpr int T = RegShape<N>::T;
  static constexpr int LP = col_line_pitch<N>();
  static constexpr int kThreads = kColsPerCta * T;
  static constexpr int kSmemBytes = kColsPerCta * LP * (int)sizeof(float2);
};

// Bytes behind a workspace's error word that the sweeps leave unused: workspaces are sized with
// them (a count-decode table stood there), and callers hold such sizes.
constexpr size_t kReservedBytes = 65536 * sizeof(float);

// One launch for everything a sweep (or an adjoint: no loss) resets before its passes: two
// gradient arrays (n_a and n_b complex elements), n_c doubles, the FP64 loss and the error word.
// Grid-stride; any grid size works.
static __global__ void sweep_prologue_kernel(float2* __restrict__ zero_a, size_t n_a, float2* __restrict__ zero_b,
                                             size_t n_b, double* __restrict__ loss, unsigned* __restrict__ err,
                                             double* __restrict__ zero_c, size_t n_c) {
  pdl_wait();
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const float2 z = make_float2(0.f, 0.f);
  for (size_t i = i0; i < n_a; i += stride) zero_a[i] = z;
  for (size_t i = i0; i < n_b; i += stride) zero_b[i] = z;
  for (size_t i = i0; i < n_c; i += stride) zero_c[i] = 0.0;
  if (i0 == 0) {
    if (loss) *loss = 0.0;
    if (err) *err = 0u;
  }
}

// Grid of sweep_prologue_kernel: about 8 elements per thread, at most 4 waves of 256-thread CTAs.
inline unsigned prologue_blocks(size_t elements, int sms) {
  const size_t want = (elements / 8 + 255) / 256;
  return static_cast<unsigned>(std::max<size_t>(1, std::min<size_t>(want, (size_t)sms * 8 * 4)));
}

inline void launch_prologue(cudaStream_t s, float2* zero_a, size_t n_a, float2* zero_b, size_t n_b, double* loss,
                            unsigned* err, double* zero_c = nullptr, size_t n_c = 0) {
  prof_begin(kMiscKernel, s);
  launch_pdl(sweep_prologue_kernel, prologue_blocks(std::max(n_a, n_b), sm_count()), 256, 0, s, zero_a, n_a, zero_b, n_b,
             loss, err, zero_c, n_c);
  prof_end(kMiscKernel, s);
}

// 1/sqrt(s), s > 0: the rsqrtf estimate refined by one Newton-Raphson step for the
// reciprocal square root, y <- y (3 - s y^2) / 2.
__device__ __forceinline__ float rsqrt_nr(float s) {
  const float y = rsqrtf(s);
  return y * fmaf(-0.5f * s, y * y, 1.5f);
}

// |z| and 1 / max(|z|, eps) from one reciprocal square root.
__device__ __forceinline__ void abs_and_inv(float2 z, float eps, float& a, float& inv) {
  const float s2 = cabs2(z);
  const float r = rsqrt_nr(fmaxf(s2, 1e-37f));
  a = s2 * r;
  inv = (a >= eps) ? r : 1.0f / eps;
}

// Sum a per-thread FP64 partial over the block and add it (times `scale`) to *out.
// Every thread of the block must call it; blocks that are not whole warps take the
// shared-memory atomic route (a full-mask shuffle needs all 32 lanes).  Calls may follow one
// another (the staging array is free again when a call returns).
__device__ __forceinline__ void block_add_double(double v, double scale, double* out) {
  __shared__ double red[32];
  const int tid = threadIdx.x;
  if ((blockDim.x & 31) == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    if (tid < 32) {
      const int nw = blockDim.x >> 5;
      double w = (tid < nw) ? red[tid] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
      if (tid == 0) atomicAdd(out, w * scale);
    }
    __syncthreads();  // red is read: a following call may write it
  } else {
    if (tid == 0) red[0] = 0.0;
    __syncthreads();
    atomicAdd(&red[0], v);
    __syncthreads();
    if (tid == 0) atomicAdd(out, red[0] * scale);
  }
}

// ---------------------------------------------------------------------------------------
// Generic 2-D transform passes (unnormalised; INV selects the sign)
// ---------------------------------------------------------------------------------------

// Row pass: in [H][N] natural (times conj(factor), when given) -> row DFT -> tiled [N/16][H][16].
template <int N, bool INV>
__global__ void __launch_bounds__(256, 2) fft2_rows_kernel(const float2* __restrict__ in, int H,
                                                            float2* __restrict__ tiled,
                                                            const float2* __restrict__ tw, int lines,
                                                            const float2* __restrict__ factor) {
  pdl_wait();
  using S = RegShape<N>;
  extern __shared__ float2 sm[];
  const int tid = threadIdx.x;
  const int l = tid / S::T;
  const int t = tid - l * S::T;
  const int r = blockIdx.x * lines + l;
  const bool row_ok = r < H;
  float2 v[S::N1];
#pragma unroll
  for (int j = 0; j < S::N1; ++j) v[j] = row_ok ? in[(size_t)r * N + t + S::T * j] : make_float2(0.f, 0.f);
  if (factor && row_ok) {
#pragma unroll
    for (int j = 0; j < S::N1; ++j) v[j] = cmulc(v[j], __ldg(&factor[(size_t)r * N + t + S::T * j]));
  }
  reg_fft<N, INV, false>(v, sm + l * RowPass<N>::LP, t, tw);
  if (row_ok) {
#pragma unroll
    for (int m = 0; m < S::N1; ++m) {
      const int kc = t + S::T * m;
      tiled[((size_t)(kc / kTile) * H + r) * kTile + (kc % kTile)] = v[m];
    }
  }
}

// Column pass: tiled [tiles][N][16] -> column DFT -> out [N][W] natural, times `scale` (and
// `factor`, when given).
template <int N, bool INV>
__global__ void __launch_bounds__(256, 2) fft2_cols_kernel(const float2* __restrict__ tiled, int W,
                                                            float2* __restrict__ out, float scale,
                                                            const float2* __restrict__ tw,
                                                            const float2* __restrict__ factor) {
  pdl_wait();
  using S = RegShape<N>;
  extern __shared__ float2 sm[];
  const int tid = threadIdx.x;
  const int c = tid % kColsPerCta;
  const int t = tid / kColsPerCta;
  constexpr int kSubs = kTile / kColsPerCta;
  const int ct = blockIdx.x / kSubs;
  const int c0 = ct * kTile + (blockIdx.x - ct * kSubs) * kColsPerCta;
  const int kc = c0 + c;
  const bool col_ok = kc < W;
  const float2* tile = tiled + (size_t)ct * N * kTile + (c0 - ct * kTile);
  float2 v[S::N1];
#pragma unroll
  for (int j = 0; j < S::N1; ++j) v[j] = col_ok ? tile[(t + S::T * j) * kTile + c] : make_float2(0.f, 0.f);
  reg_fft<N, INV, true>(v, sm + c * ColPass<N>::LP, t, tw);
  if (col_ok) {
#pragma unroll
    for (int m = 0; m < S::N1; ++m) {
      const size_t at = (size_t)(t + S::T * m) * W + kc;
      const float2 z = cscale(v[m], scale);
      out[at] = factor ? cmul(z, __ldg(&factor[at])) : z;
    }
  }
}

// ---- column pass of a fused sweep on the two-line packed-FP32x2 FFT ------------------
// A CTA owns one 16-column tile of one frame of the tiled scratch [frame][tile][row][16];
// thread (p, t) transforms the column pair (2p, 2p+1) of the tile, both columns in
// lock-step (ptx_pairfft.cuh), so every butterfly, twiddle product and epilogue operation is
// one packed instruction for two columns.  A column pair is one 16-byte load / store per
// row (a warp covers four whole 128-byte tile rows).  The sequence per column: DFT in the
// FIRST_INV direction, scale by `norm`, amplitude-loss epilogue against the counts
// (decoded with their scale; SHIFTED: the counts are stored fftshifted in both axes), the
// DFT in the other direction, store in place.  The tile's counts arrive by cp.async while
// the first transform runs; the twiddle table sits in shared memory as broadcast pairs.
template <int N>
struct ColPairCfg {
  static constexpr int kPairs = kTile / 2;
  static constexpr int LP4 = RegShape<N>::BUF + 1;  // odd float4 pitch: quarter-warps conflict-free
  static constexpr int kThreads = kPairs * RegShape<N>::T;
  static constexpr int kExchBytes = kPairs * LP4 * (int)sizeof(float4);
  static constexpr int kTwBytes = N * (int)sizeof(float4);
  static constexpr int kMeasBytes = N * kTile * (int)sizeof(uint16_t);
  static constexpr int kSmemBytes = kExchBytes + kTwBytes + kMeasBytes;
};

// UNIT_NORM: `norm` is 1 (the epilogue drops the scaling); FULL: `width` is a multiple of
// the tile, so every column pair exists and the per-column masks go.
// Up to 256-point columns a CTA fits 128 registers per thread and 47 KB of shared memory, so
// four CTAs share an SM (16 warps); longer columns keep two (512) or one (1024).
template <int N>
constexpr int col_pair_min_blocks() {
  return ColPairCfg<N>::kThreads > 128 ? 1 : (N <= 256 ? 4 : 2);
}

template <int N, bool FIRST_INV, bool SHIFTED, bool UNIT_NORM, bool FULL, bool PLAIN>
__global__ void __launch_bounds__(ColPairCfg<N>::kThreads, col_pair_min_blocks<N>()) cols_sweep_pair(
    float2* __restrict__ scratch, int width, int frame0, const float2* __restrict__ tw,
    const uint16_t* __restrict__ measured, float scale, float norm, float grad_scale, double inv_numel,
    double* __restrict__ loss) {
  pdl_wait();
  using S = RegShape<N>;
  using Cfg = ColPairCfg<N>;
  extern __shared__ float4 sm4[];
  float4* tw4 = sm4 + Cfg::kPairs * Cfg::LP4;
  uint16_t* meas_s = reinterpret_cast<uint16_t*>(tw4 + N);
  const int tid = threadIdx.x;
  const int p = tid % Cfg::kPairs;
  const int t = tid / Cfg::kPairs;
  const int ct = blockIdx.x;
  const int f = blockIdx.y;
  const int c0 = ct * kTile;
  const bool okA = FULL || c0 + 2 * p < width;
  const bool okB = FULL || c0 + 2 * p + 1 < width;
  float2* tile = scratch + ((size_t)f * num_tiles(width) + ct) * N * kTile + 2 * p;
  const size_t g = (size_t)frame0 + f;
  float4* buf = sm4 + p * Cfg::LP4;
  constexpr int kRowOff = SHIFTED ? N / 2 : 0;
  const int col_off = SHIFTED ? width / 2 : 0;

  // counts of rows kr of the tile -> meas_s[kr][16]
  int ic0 = c0 + col_off;
  if (ic0 >= width) ic0 -= width;
  const bool fast = (width % (2 * kTile) == 0) && ((reinterpret_cast<uintptr_t>(measured) & 15) == 0);
  if (fast) {
    for (int i = tid; i < 2 * N; i += blockDim.x) {
      const int kr = i >> 1, h = (i & 1) * 8;
      const int ir = (kr + kRowOff) & (N - 1);
      cp_async16(meas_s + kr * kTile + h, measured + (g * N + ir) * width + ic0 + h);
    }
    cp_async_commit();
  } else {
    for (int i = tid; i < N * kTile; i += blockDim.x) {
      const int kr = i / kTile, cc = i - kr * kTile;
      const int ir = (kr + kRowOff) & (N - 1);
      int icc = c0 + cc + col_off;
      if (icc >= width) icc -= width;
      meas_s[i] = (c0 + cc < width) ? measured[(g * N + ir) * width + icc] : 0;
    }
  }
  for (int i = tid; i < N; i += blockDim.x) {
    const float2 w = __ldg(&tw[i]);
    tw4[i] = make_float4(w.x, w.x, w.y, w.y);
  }
  const uint64_t pol = policy_evict_first();
  CPair v[S::N1];
#pragma unroll
  for (int j = 0; j < S::N1; ++j) {
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    if (okA) q = ld_stream4(tile + (t + S::T * j) * kTile, pol);
    if (!okB) q.z = q.w = 0.f;
    v[j] = {make_float2(q.x, q.z), make_float2(q.y, q.w)};
  }
  __syncthreads();  // twiddle table
  pair_fft<N, FIRST_INV, true>(v, buf, t, tw4);
  cp_async_wait_all();
  __syncthreads();
  float2 part = make_float2(0.f, 0.f);  // squared residuals of the two columns
  const float2 gs = f2(grad_scale), nrm = f2(norm);
#pragma unroll
  for (int m = 0; m < S::N1; ++m) {
    const int kr = t + S::T * m;
    const CPair F = UNIT_NORM ? v[m] : CPair{mul2(v[m].re, nrm), mul2(v[m].im, nrm)};
    const float2 s2 = fma2(F.re, F.re, mul2(F.im, F.im));
    // rsqrt_nr on both lanes, its Newton-Raphson step in packed form (the same IEEE operations)
    const float2 sc2 = make_float2(fmaxf(s2.x, 1e-37f), fmaxf(s2.y, 1e-37f));
    const float2 y0 = make_float2(rsqrt_floor(sc2.x), rsqrt_floor(sc2.y));
    const float2 r = mul2(y0, fma2(mul2(f2(-0.5f), sc2), mul2(y0, y0), f2(1.5f)));
    const float2 a = mul2(s2, r);
    const float2 inv =
        make_float2(a.x >= kEpsF32 ? r.x : 1.0f / kEpsF32, a.y >= kEpsF32 ? r.y : 1.0f / kEpsF32);
    float2 rr = minus_amplitudes<PLAIN>(a, *reinterpret_cast<const uint32_t*>(meas_s + kr * kTile + 2 * p), scale);
    rr = make_float2(okA ? rr.x : 0.f, okB ? rr.y : 0.f);
    part = fma2(rr, rr, part);
    const float2 sc = mul2(mul2(gs, rr), inv);
    v[m] = {mul2(F.re, sc), mul2(F.im, sc)};
  }
  pair_fft<N, !FIRST_INV, true>(v, buf, t, tw4);
  if (okA) {
#pragma unroll
    for (int m = 0; m < S::N1; ++m) {
      *reinterpret_cast<float4*>(tile + (t + S::T * m) * kTile) =
          make_float4(v[m].re.x, v[m].im.x, v[m].re.y, v[m].im.y);
    }
  }
  block_add_double(static_cast<double>(part.x) + static_cast<double>(part.y), inv_numel, loss);
}

// ---- the same pass as a pipeline over tiles ------------------------------------------------
// One wave of CTAs, each walking tiles with two groups of threads (one tile each, alternating)
// over three tile buffers.  A whole tile is one contiguous block, so it arrives by one bulk copy
// (cp.async.bulk, no registers, no load instructions) while both groups transform earlier tiles;
// the exchanges of a tile's two transforms happen in the same buffer: thread (c, t) of column c
// writes exactly where it has read (rows t + T j), and a half-warp always covers one 128-byte row.
// The buffer takes the next tile as soon as the second exchange has been read, before that
// transform's last step and the stores.
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
// Bulk copy of `bytes` (a multiple of 16, both ends 16-byte aligned) that completes on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t pol) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(pol)
      : "memory");
}
// Wait for the phase of `parity`; false if it has not completed after a bounded number of tries
// (tens of milliseconds at least, where a copy takes microseconds): the caller then stops, waits
// once more for the copies it still has under way, and reports kStatusTimeout and NaN results.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (int i = 0; i < (1 << 20); ++i) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void group_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}
// group_sync that tells every thread whether `flag` holds for any of them.
__device__ __forceinline__ bool group_sync_any(int id, int threads, bool flag) {
  uint32_t any;
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.u32 q, %3, 0;\nbar.red.or.pred p, %1, %2, q;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(any)
      : "r"(id), "r"(threads), "r"(static_cast<uint32_t>(flag))
      : "memory");
  return any != 0;
}

template <int N>
struct ColPipeCfg {
  static constexpr int kPairs = kTile / 2;
  static constexpr int kGroup = kPairs * RegShape<N>::T;  // threads per tile
  static constexpr int kBufs = PipeRing::kBufs;
  static constexpr int kTileBytes = N * kTile * (int)sizeof(float2);
  static constexpr int kMeasBytes = N * kTile * (int)sizeof(uint16_t);
  static constexpr int kTwBytes = N / 2 * (int)sizeof(float2);
  static constexpr int kSmemBytes = kBufs * kTileBytes + 2 * kMeasBytes + kTwBytes + PipeRing::kBars * (int)sizeof(uint64_t);
  static constexpr int kBlocks = N <= 256 ? 2 : 1;  // CTAs per SM
};

// First step of the pair transform for thread t: DFT-N1, twiddles from the half table
// tw[m] = exp(-2 pi i m / N), m < N / 2 (the other half is its negative), to rows t + T k1.
template <int N, bool INV>
__device__ __forceinline__ void pipe_step1(CPair (&v)[RegShape<N>::N1], float4* rows, int t, const float2* tw) {
  using S = RegShape<N>;
  constexpr int P = kTile / 2;
  PRegDft<S::N1, INV>::run(v);
  rows[t * P] = pack4(v[0]);
#pragma unroll
  for (int k1 = 1; k1 < S::N1; ++k1) {
    const int m = t * k1;
    float2 w = tw[m & (N / 2 - 1)];
    const uint32_t flip = static_cast<uint32_t>(m & (N / 2)) << (31 - (S::LOG - 1));
    w.x = __uint_as_float(__float_as_uint(w.x) ^ flip);
    w.y = __uint_as_float(__float_as_uint(w.y) ^ (INV ? flip ^ 0x80000000u : flip));
    const float2 wx = f2(w.x), wy = f2(w.y), wn = f2(-w.y);
    const CPair z = v[k1];
    rows[(t + S::T * k1) * P] = pack4({fma2(z.im, wn, mul2(z.re, wx)), fma2(z.im, wx, mul2(z.re, wy))});
  }
}
// Second step: the C rows of T values k1 = q T + t, then their DFT-T.
template <int N>
__device__ __forceinline__ void pipe_load2(CPair (&v)[RegShape<N>::N1], const float4* rows, int t) {
  using S = RegShape<N>;
  constexpr int P = kTile / 2;
#pragma unroll
  for (int q = 0; q < S::C; ++q)
#pragma unroll
    for (int j = 0; j < S::T; ++j) v[q * S::T + j] = unpack4(rows[((q * S::T + t) * S::T + j) * P]);
}
template <int N, bool INV>
__device__ __forceinline__ void pipe_step2(CPair (&v)[RegShape<N>::N1]) {
  using S = RegShape<N>;
#pragma unroll
  for (int q = 0; q < S::C; ++q) PRegDft<S::T, INV>::run(v + q * S::T);
}
// after pipe_step2: element t + T m of the line (m = q + C k2) is v[pipe_index(m)]
template <int N>
__device__ __forceinline__ constexpr int pipe_index(int m) {
  return (m % RegShape<N>::C) * RegShape<N>::T + m / RegShape<N>::C;
}

// Whole tiles only (`width` a multiple of 2 kTile) and counts on a 16-byte boundary.  Bound: at 8
// warps per SM the transforms, the exchanges and the epilogue overlap only in part, no pipe is above
// 47% (900 frames of 512^2: 1023 us, cols_sweep_pair 1135; 825 without the DFT arithmetic, 780 with
// the frames in L2 as well).
template <int N, bool FIRST_INV, bool SHIFTED, bool UNIT_NORM>
__global__ void __launch_bounds__(2 * ColPipeCfg<N>::kGroup, ColPipeCfg<N>::kBlocks) cols_sweep_pipe(
    float2* __restrict__ scratch, int width, int nframes, int frame0, const float2* __restrict__ tw,
    const uint16_t* __restrict__ measured, float scale, float norm, float grad_scale, double inv_numel,
    double* __restrict__ loss, unsigned* __restrict__ err) {
  using S = RegShape<N>;
  using Cfg = ColPipeCfg<N>;
  constexpr int P = Cfg::kPairs;
  extern __shared__ __align__(128) unsigned char pipe_smem[];
  const int tid = threadIdx.x;
  const int grp = tid / Cfg::kGroup, gt = tid - grp * Cfg::kGroup;
  const int p = gt % P, t = gt / P;
  uint16_t* meas_s = reinterpret_cast<uint16_t*>(pipe_smem + Cfg::kBufs * Cfg::kTileBytes + grp * Cfg::kMeasBytes);
  float2* tws = reinterpret_cast<float2*>(pipe_smem + Cfg::kBufs * Cfg::kTileBytes + 2 * Cfg::kMeasBytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(tws + N / 2);
  for (int i = tid; i < N / 2; i += blockDim.x) tws[i] = __ldg(&tw[i]);
  if (tid == 0) {
    for (int b = 0; b < PipeRing::kBars; ++b) mbar_init(full + b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  pdl_wait();
  const int tiles = width / kTile;
  const long long total = (long long)tiles * nframes;
  const int n = static_cast<int>((total - blockIdx.x + gridDim.x - 1) / gridDim.x);
  const uint64_t pol = policy_evict_first();
  auto tile_at = [&](int i) { return blockIdx.x + (long long)i * gridDim.x; };
  auto issue = [&](int i) {
    bulk_load(pipe_smem + PipeRing::buffer(i) * Cfg::kTileBytes, scratch + tile_at(i) * N * kTile, Cfg::kTileBytes,
              full + PipeRing::barrier(i), pol);
  };
  if (tid == 0) {
    for (int i = 0; i < Cfg::kBufs && i < n; ++i) issue(i);
  }
  constexpr int kRowOff = SHIFTED ? N / 2 : 0;
  const int col_off = SHIFTED ? width / 2 : 0;
  const float2 gs = f2(grad_scale), nrm = f2(norm);
  double acc = 0.0;
  int i = grp;
  for (; i < n; i += PipeRing::kGroups) {
    const long long tile = tile_at(i);
    const int f = static_cast<int>(tile / tiles), c0 = static_cast<int>(tile - (long long)f * tiles) * kTile;
    // the tile's counts, by rows of the spectrum; the previous tile's were read before a barrier
    {
      int ic0 = c0 + col_off;
      if (ic0 >= width) ic0 -= width;
      const uint16_t* src = measured + ((size_t)frame0 + f) * N * width + ic0;
#pragma unroll 4
      for (int e = gt; e < 2 * N; e += Cfg::kGroup) {
        const int kr = e >> 1, h = (e & 1) * 8;
        cp_async16(meas_s + kr * kTile + h, src + (size_t)((kr + kRowOff) & (N - 1)) * width + h);
      }
      cp_async_commit();
    }
    float4* rows = reinterpret_cast<float4*>(pipe_smem + PipeRing::buffer(i) * Cfg::kTileBytes) + p;
    const bool late = !mbar_wait(full + PipeRing::barrier(i), PipeRing::parity(i));
    CPair v[S::N1];
#pragma unroll
    for (int j = 0; j < S::N1; ++j) {
      const float4 q = rows[(t + S::T * j) * P];
      v[j] = {make_float2(q.x, q.z), make_float2(q.y, q.w)};
    }
    pipe_step1<N, FIRST_INV>(v, rows, t, tws);
    if (group_sync_any(1 + grp, Cfg::kGroup, late)) break;
    pipe_load2<N>(v, rows, t);
    pipe_step2<N, FIRST_INV>(v);
    cp_async_wait_all();
    group_sync(1 + grp, Cfg::kGroup);  // the exchange is read, the counts are complete
    float2 part = make_float2(0.f, 0.f);  // squared residuals of the two columns
    CPair g[S::N1];
#pragma unroll
    for (int m = 0; m < S::N1; ++m) {
      const int kr = t + S::T * m;
      const CPair z = v[pipe_index<N>(m)];
      const CPair F = UNIT_NORM ? z : CPair{mul2(z.re, nrm), mul2(z.im, nrm)};
      const float2 s2 = fma2(F.re, F.re, mul2(F.im, F.im));
      // the reciprocal square root and its Newton-Raphson step as in cols_sweep_pair
      const float2 sc2 = make_float2(fmaxf(s2.x, 1e-37f), fmaxf(s2.y, 1e-37f));
      const float2 y0 = make_float2(rsqrt_floor(sc2.x), rsqrt_floor(sc2.y));
      const float2 r = mul2(y0, fma2(mul2(f2(-0.5f), sc2), mul2(y0, y0), f2(1.5f)));
      const float2 a = mul2(s2, r);
      const float2 inv =
          make_float2(a.x >= kEpsF32 ? r.x : 1.0f / kEpsF32, a.y >= kEpsF32 ? r.y : 1.0f / kEpsF32);
      const float2 rr = minus_amplitudes<true>(a, *reinterpret_cast<const uint32_t*>(meas_s + kr * kTile + 2 * p), scale);
      part = fma2(rr, rr, part);
      const float2 sc = mul2(mul2(gs, rr), inv);
      g[m] = {mul2(F.re, sc), mul2(F.im, sc)};
    }
    acc += static_cast<double>(part.x) + static_cast<double>(part.y);
    pipe_step1<N, !FIRST_INV>(g, rows, t, tws);
    group_sync(1 + grp, Cfg::kGroup);
    pipe_load2<N>(g, rows, t);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    group_sync(1 + grp, Cfg::kGroup);  // the buffer is free
    if (gt == 0 && i + Cfg::kBufs < n) issue(i + Cfg::kBufs);
    pipe_step2<N, !FIRST_INV>(g);
    float4* out = reinterpret_cast<float4*>(scratch + tile * N * kTile) + p;
#pragma unroll
    for (int m = 0; m < S::N1; ++m) {
      const CPair z = g[pipe_index<N>(m)];
      out[(t + S::T * m) * P] = make_float4(z.re.x, z.im.x, z.re.y, z.im.y);
    }
  }
  // a copy that did not come: the tiles from there on are NaN, and so are the loss and gradients
  const bool stopped = i < n;
  if (__syncthreads_or(stopped)) {
    const float nan = __int_as_float(0x7fc00000);
    if (stopped) {
      if (gt == 0 && err) atomicOr(err, kStatusTimeout);
      cp_async_wait_all();
      for (int k = i; k < n; k += PipeRing::kGroups) {
        float4* out = reinterpret_cast<float4*>(scratch + tile_at(k) * N * kTile) + p;
        for (int m = 0; m < S::N1; ++m) out[(t + S::T * m) * P] = make_float4(nan, nan, nan, nan);
      }
      acc = nan;
    }
    // the copies issued and not waited for: they write to this CTA's shared memory
    int* next = reinterpret_cast<int*>(tws);
    if (gt == 0) next[grp] = i;
    __syncthreads();
    if (tid == 0) {
      for (int k = 0; k < n; ++k) {
        if (PipeRing::left_open(k, next)) mbar_wait(full + PipeRing::barrier(k), PipeRing::parity(k));
      }
    }
    __syncthreads();
  }
  block_add_double(acc, inv_numel, loss);
}

// Column lengths the pipeline is used for, and the frames it takes: whole pairs of tiles (the
// counts' 16-byte pieces stay inside a tile), counts on a 16-byte boundary and of a plain scale, and
// five tiles or more per CTA.  At 512 points a CTA of cols_sweep_pair leaves no room for the next tile's loads beside it
// (14400 tiles 1135 us against 1023 here); at 256 several of its CTAs share an SM and it is the faster
// one (225 frames: 60.5 us against 69.8).  With few tiles per CTA the pipeline's start and end
// weigh more (whole sweeps, us, pipeline and pair: 180 tiles of 512 x 96 33.3 and 32.5, 600 tiles 81.6 and
// 79.5, 640 tiles of 512^2 75.1 and 73.2; equal within 1% from 740 to 1200 tiles).
template <int N>
constexpr bool col_pipe_length() {
  return N == 512;
}
inline bool col_pipe_takes(int width, int nframes, const uint16_t* measured, float scale) {
  return width % (2 * kTile) == 0 && (reinterpret_cast<uintptr_t>(measured) & 15) == 0 && plain_scale(scale) &&
         (long long)(width / kTile) * nframes >= 5LL * sm_count();
}

// The column pass of a sweep (every power-of-two length), once prepared: the pipeline, or the paired
// pass in the compilation for whole tiles (UNIT_NORM: a `norm` of 1 is then not applied) or any width,
// and for the scale.
template <int N, bool FIRST_INV, bool SHIFTED, bool UNIT_NORM>
int prepare_cols_sweep() {
  int st = PTX_OK;
  if constexpr (col_pipe_length<N>()) {
    st = ensure_smem((const void*)cols_sweep_pipe<N, FIRST_INV, SHIFTED, UNIT_NORM>, ColPipeCfg<N>::kSmemBytes);
  }
  auto pair = [&](auto kern) {
    if (!st) st = ensure_smem((const void*)kern, ColPairCfg<N>::kSmemBytes);
  };
  pair(cols_sweep_pair<N, FIRST_INV, SHIFTED, UNIT_NORM, true, true>);
  pair(cols_sweep_pair<N, FIRST_INV, SHIFTED, UNIT_NORM, true, false>);
  pair(cols_sweep_pair<N, FIRST_INV, SHIFTED, false, false, true>);
  pair(cols_sweep_pair<N, FIRST_INV, SHIFTED, false, false, false>);
  return st;
}
template <int N, bool FIRST_INV, bool SHIFTED, bool UNIT_NORM>
void launch_cols_sweep(float2* frames, int width, int nframes, int frame0, const float2* tw, const uint16_t* measured,
                       float scale, float norm, float grad_scale, double inv_numel, double* loss, unsigned* err,
                       cudaStream_t s) {
  if constexpr (col_pipe_length<N>()) {
    if (col_pipe_takes(width, nframes, measured, scale)) {
      using C = ColPipeCfg<N>;
      auto kern = cols_sweep_pipe<N, FIRST_INV, SHIFTED, UNIT_NORM>;
      const int grid =
          persistent_grid((const void*)kern, 2 * C::kGroup, C::kSmemBytes, (long long)num_tiles(width) * nframes);
      launch_pdl(kern, grid, 2 * C::kGroup, C::kSmemBytes, s, frames, width, nframes, frame0, tw, measured, scale, norm,
                 grad_scale, inv_numel, loss, err);
      return;
    }
  }
  auto pair = [&](auto kern) {
    launch_pdl(kern, dim3(num_tiles(width), nframes), ColPairCfg<N>::kThreads, ColPairCfg<N>::kSmemBytes, s, frames,
               width, frame0, tw, measured, scale, norm, grad_scale, inv_numel, loss);
  };
  const bool full = width % kTile == 0;
  if (plain_scale(scale)) {
    full ? pair(cols_sweep_pair<N, FIRST_INV, SHIFTED, UNIT_NORM, true, true>)
         : pair(cols_sweep_pair<N, FIRST_INV, SHIFTED, false, false, true>);
  } else {
    full ? pair(cols_sweep_pair<N, FIRST_INV, SHIFTED, UNIT_NORM, true, false>)
         : pair(cols_sweep_pair<N, FIRST_INV, SHIFTED, false, false, false>);
  }
}

}  // namespace ptx
