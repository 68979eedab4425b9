// Line transforms of length N = R p, p a prime of 37 to 127 and R small and {2,3,5}-smooth: the
// plain 2-D transforms and the twice-upsampled correlation of the registration at image sides such
// as 472 (a 512-pixel crop less a 20-pixel border on each side) = 8 x 59.
//
// With n = p i + j and k = k1 + R k2 (i, k1 < R; j, k2 < p)
//   X[k] = sum_j exp(-+2 pi i j k2 / p) y_k1[j],
//   y_k1[j] = exp(-+2 pi i j k1 / N) sum_i x[p i + j] exp(-+2 pi i i k1 / R)
// A thread takes the two R-point transforms of j and p - j in registers, applies the twiddles and
// leaves s = y[j] + y[p - j] and d = y[j] - y[p - j] in shared memory, [j][column], a column being
// one (line, k1).  The p-point transforms are then a real matrix product over j = 1 .. (p - 1) / 2,
//   X[k2], X[p - k2] = y[0] + sum_j s_j cos(2 pi j k2 / p) -+ i sum_j d_j sin(2 pi j k2 / p)
// (p FMA per point instead of 4 p), a warp computing 8 outputs k2 of 64 columns, 2 per lane: 64
// FMA against 12 shared-memory wavefronts a step.  Each output is a plain FP32 sum, as accurate as a
// library's direct prime factor; a chirp transform would take three times the rounding error.
// Lines run along contiguous memory; the output can be written transposed, 8 to 16 lines (64 to
// 128 bytes) at a time, so that the second dimension is again contiguous and nothing is
// transposed in a pass of its own.
//
// Bound: FP32 issue and shared memory about equally in the product (57 FMA a point), and step 1, whose
// loads only the other CTA of the SM hides where they are not staged; HBM alone would take a third
// of the time.  200 images of 472^2 (us; cuFFT with its padding and transposing passes before): their
// spectra 1420 -> 470 (first pass 232, second 240), the correlation on 944^2 2900 -> 1260 (431 and
// 828; 551 and 1165 with loads on demand and the padding tested element by element).  At 60 images
// 70 to 73% of the issue slots and half of the FMA pipe are busy.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/ptychox.h"
#include "ptx_internal.h"
#include "ptx_fft.cuh"
#include "ptx_mixfft.cuh"

namespace ptx {
namespace {

constexpr int kThreads = 256;
constexpr int kColumns = 128;  // columns (line, k1) of a CTA
constexpr int kOut = 8;        // outputs k2 of a warp's step
constexpr int kStagedSmem = 113 << 10;  // lines are staged where two CTAs still fit an SM

int padded_outputs(int p) { return ((p - 1) / 2 + 1 + kOut - 1) / kOut * kOut; }

// p of n = R p where these kernels take n, else 0.  Both sides, 2-D transforms of 64 images of
// n^2 (us): cuFFT needs 8 to 12 ps per point up to the factor 31 (bar 17, 19 and 23: 20) and 29 to 48
// from 37 on; 222 = 6 x 37 163 against 64 here, 246 = 6 x 41 202/70, 472 = 8 x 59 473/210,
// 492 = 12 x 41 543/242, 508 = 4 x 127 450/373.  The relative error against FP64 is the smaller
// one throughout (472: 3.3e-7 against 3.6e-7, 492: 3.0e-7 against 4.6e-7), but for n = p, which also
// gains nothing (113: 62 against 58 us, 4.0e-7 against 3.9e-7) and stays with the library.
// R = 7 and 11 have no register transform.  An image is taken where both its sides are (layout): of
// the sides 60 to 984 that are 17.5%, where 59% have a prime factor of 37 or more.
int prime_part(int n) {
  if (n < 74 || n > 127 * 12) return 0;
  int p = 1, m = n;
  for (int q = 2; q * q <= m; ++q) {
    while (m % q == 0) {
      p = std::max(p, q);
      m /= q;
    }
  }
  p = std::max(p, m);
  const int r = n / p;
  if (p < 37 || p > 127 || r == 1 || r > 12 || r == 7 || r == 11) return 0;
  return p;
}

// Tables of a line length N = R p: the twiddles [k1][j], then (cos, sin)(2 pi j k / p) as
// [j - 1][k], k < padded_outputs(p).
size_t table_entries(int n, int p) { return (size_t)n + (size_t)((p - 1) / 2) * padded_outputs(p); }

__global__ void __launch_bounds__(256) prime_tables_kernel(int n, int p, int kpad, float2* __restrict__ out) {
  const int total = n + (p - 1) / 2 * kpad;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    double s, c;
    if (i < n) {
      const int k1 = i / p, j = i - k1 * p;
      sincospi(-2.0 * (j * k1) / n, &s, &c);  // j k1 < n
    } else {
      const int q = i - n, j = q / kpad + 1, k = q % kpad;
      sincospi(2.0 * (j * k % p) / p, &s, &c);
    }
    out[i] = make_float2(static_cast<float>(c), static_cast<float>(s));
  }
}

struct PrimeArgs {
  const float2* in;      // [image][line][valid] complex, or null
  const float* real;     // real images: element (image, line, i) at image * real_image + line * real_line + i
  long long real_image, real_line;
  float sign;            // -1: the input's conjugate
  int lines, images;     // lines per image
  int p;
  const float2* tables;
  float2* out;
};

// STAGE: a unit's lines (one contiguous block) land in shared memory by cp.async while the previous
// unit's product runs.  PAD = false: element n of the line; PAD = true: the line holds
// R p / 2 bins, zero-padded to twice as many around the highest frequency (FTpad,
// dftregistration.m:189-224).
template <int R, bool PLUS, bool PAD, bool REAL, bool TRANSPOSE, bool STAGE>
__global__ void __launch_bounds__(kThreads, R <= 16 ? 2 : 1) prime_lines_kernel(PrimeArgs a) {
  constexpr int LINES = kColumns / R, COLS = LINES * R;
  constexpr int PITCH = kColumns + 1;  // float4 of a row j: consecutive j fall in consecutive banks
  extern __shared__ __align__(16) float4 sd[];  // [h][PITCH], then coefficients, then y[0]
  const int p = a.p, h = (p - 1) / 2, n = R * p;
  const int kpad = (h + 1 + kOut - 1) / kOut * kOut;
  float2* coef = reinterpret_cast<float2*>(sd + (size_t)h * PITCH);
  float2* y0 = coef + (size_t)h * kpad;
  const float2* tw = a.tables;
  float2* raw = coef + (size_t)h * kpad + kColumns;  // STAGE: [LINES][valid]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < h * kpad; i += kThreads) coef[i] = __ldg(a.tables + n + i);
  const int per_image = (a.lines + LINES - 1) / LINES;
  const long long units = (long long)per_image * a.images;
  const int valid = PAD ? n / 2 : n, low = valid - valid / 2;
  auto request = [&](long long u) {
    const long long image = u / per_image, line0 = (u - image * per_image) * LINES;
    const float2* src = a.in + (image * a.lines + line0) * valid;
    const int count = static_cast<int>(min((long long)LINES, a.lines - line0)) * valid;
    for (int i = tid; i < count; i += kThreads) cp_async8(raw + i, src + i);
    cp_async_commit();
  };
  if (STAGE && blockIdx.x < units) request(blockIdx.x);
  for (long long u = blockIdx.x; u < units; u += gridDim.x) {
    if (STAGE) {
      cp_async_wait_all();
      __syncthreads();
    }
    const int image = static_cast<int>(u / per_image);
    const int line0 = static_cast<int>(u - (long long)image * per_image) * LINES;
    // step 1: item (line, j) takes the elements j and p - j of every stretch of p
    for (int item = tid; item < LINES * (h + 1); item += kThreads) {
      const int l = item / (h + 1), j = item - l * (h + 1);
      const int line = min(line0 + l, a.lines - 1);  // columns past the last line are not stored
      const float* real = REAL ? a.real + image * a.real_image + line * a.real_line : nullptr;
      const float2* src = STAGE ? raw + (line - line0) * valid : a.in + ((size_t)image * a.lines + line) * valid;
      auto load = [&](int at) {
        if constexpr (REAL) return make_float2(__ldg(real + at), 0.f);
        const float2 v = STAGE ? src[at] : __ldg(src + at);
        return make_float2(v.x, a.sign * v.y);
      };
      auto element = [&](int i, int j) {  // element p i + j of the (padded) line
        const int at = p * i + j;
        if constexpr (!PAD) {
          return load(at);
        } else if constexpr (R % 4 == 0) {  // the padding is whole stretches of p
          return i < R / 4 ? load(at) : i >= 3 * R / 4 ? load(at - valid) : make_float2(0.f, 0.f);
        } else {
          return at < low ? load(at) : at >= low + valid ? load(at - valid) : make_float2(0.f, 0.f);
        }
      };
      float2 ya[R], yb[R];
      const int jb = j ? p - j : 0;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        ya[i] = element(i, j);
        yb[i] = element(i, jb);
      }
      mix::Dft<R, PLUS>::run(ya);
      mix::Dft<R, PLUS>::run(yb);
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int c = TRANSPOSE ? k * LINES + l : l * R + k;
        const float2 wa = __ldg(tw + k * p + j), wb = __ldg(tw + k * p + jb);
        const float2 x = PLUS ? mix::mulc(ya[k], wa) : mix::mul(ya[k], wa);
        if (j) {
          const float2 z = PLUS ? mix::mulc(yb[k], wb) : mix::mul(yb[k], wb);
          sd[(j - 1) * PITCH + c] = make_float4(x.x + z.x, x.y + z.y, x.x - z.x, x.y - z.y);
        } else {
          y0[c] = x;
        }
      }
    }
    __syncthreads();
    if (STAGE && u + gridDim.x < units) request(u + gridDim.x);
    // step 2: kOut outputs of 64 columns per warp
    const int tiles = kpad / kOut;
    for (int task = warp; task < 2 * tiles; task += kThreads / 32) {
      const int k0 = (task >> 1) * kOut, c0 = (task & 1) * 64 + lane;
      float acc[2][kOut][4];
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int k = 0; k < kOut; ++k)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[q][k][e] = 0.f;
#pragma unroll 2
      for (int j = 0; j < h; ++j) {
        const float4 s0 = sd[j * PITCH + c0], s1 = sd[j * PITCH + c0 + 32];
        const float4* cf = reinterpret_cast<const float4*>(coef + j * kpad + k0);
#pragma unroll
        for (int k = 0; k < kOut; k += 2) {
          const float4 w = cf[k / 2];  // cos, sin of k and k + 1
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float c = e ? w.z : w.x, s = e ? w.w : w.y;
            acc[0][k + e][0] = fmaf(c, s0.x, acc[0][k + e][0]);
            acc[0][k + e][1] = fmaf(c, s0.y, acc[0][k + e][1]);
            acc[0][k + e][2] = fmaf(s, s0.z, acc[0][k + e][2]);
            acc[0][k + e][3] = fmaf(s, s0.w, acc[0][k + e][3]);
            acc[1][k + e][0] = fmaf(c, s1.x, acc[1][k + e][0]);
            acc[1][k + e][1] = fmaf(c, s1.y, acc[1][k + e][1]);
            acc[1][k + e][2] = fmaf(s, s1.z, acc[1][k + e][2]);
            acc[1][k + e][3] = fmaf(s, s1.w, acc[1][k + e][3]);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c = c0 + 32 * q;
        const int l = TRANSPOSE ? c % LINES : c / R, k1 = TRANSPOSE ? c / LINES : c % R;
        const int line = line0 + l;
        if (c >= COLS || line >= a.lines) continue;
        const float2 b = y0[c];
        float2* out = TRANSPOSE ? a.out + (size_t)image * n * a.lines + line : a.out + ((size_t)image * a.lines + line) * n;
        auto at = [&](int k2) { return (size_t)(k1 + R * k2) * (TRANSPOSE ? a.lines : 1); };
#pragma unroll
        for (int k = 0; k < kOut; ++k) {
          const int k2 = k0 + k;
          if (k2 > h) continue;
          const float re = b.x + acc[q][k][0], im = b.y + acc[q][k][1];
          // -i D = (D.im, -D.re) in the forward transform, its negative in the inverse
          const float dr = PLUS ? -acc[q][k][3] : acc[q][k][3], di = PLUS ? acc[q][k][2] : -acc[q][k][2];
          out[at(k2)] = make_float2(re + dr, im + di);
          if (k2) out[at(p - k2)] = make_float2(re - dr, im - di);
        }
      }
    }
    __syncthreads();  // the columns are read
  }
}

template <int R, bool PLUS, bool PAD, bool REAL, bool TRANSPOSE, bool STAGE = PAD>
int launch_lines(const PrimeArgs& a, cudaStream_t s) {
  constexpr int LINES = kColumns / R;
  auto kern = prime_lines_kernel<R, PLUS, PAD, REAL, TRANSPOSE, STAGE>;
  const int h = (a.p - 1) / 2, kpad = padded_outputs(a.p);
  const int smem = h * (kColumns + 1) * (int)sizeof(float4) + (h * kpad + kColumns + (STAGE ? LINES * R * a.p / 2 : 0)) * (int)sizeof(float2);
  if constexpr (STAGE) {
    if (smem > kStagedSmem) return launch_lines<R, PLUS, PAD, REAL, TRANSPOSE, false>(a, s);
  }
  if (int st = ensure_smem((const void*)kern, smem)) return st;
  const long long units = (long long)((a.lines + LINES - 1) / LINES) * a.images;
  const int grid = persistent_grid((const void*)kern, kThreads, smem, units);
  kern<<<grid, kThreads, smem, s>>>(a);
  return PTX_OK;
}

// Lines of R p points; pad: R counts the padded line's.
template <bool PAD, bool REAL, bool TRANSPOSE>
int dispatch_lines(int r, const PrimeArgs& a, cudaStream_t s) {
#define PTX_PRIME_CASE(N) \
  case N:                 \
    return launch_lines<(PAD ? 2 : 1) * N, PAD, PAD, REAL, TRANSPOSE>(a, s);
  switch (r) {
    PTX_PRIME_CASE(2)
    PTX_PRIME_CASE(3)
    PTX_PRIME_CASE(4)
    PTX_PRIME_CASE(5)
    PTX_PRIME_CASE(6)
    PTX_PRIME_CASE(8)
    PTX_PRIME_CASE(9)
    PTX_PRIME_CASE(10)
    PTX_PRIME_CASE(12)
    default:
      return set_error(PTX_ERR_UNSUPPORTED_SIZE, "no prime-factor line transform of %d p points", r);
  }
#undef PTX_PRIME_CASE
}

void make_tables(int n, int p, float2* out, cudaStream_t s) {
  const int total = static_cast<int>(table_entries(n, p));
  prime_tables_kernel<<<(total + 255) / 256, 256, 0, s>>>(n, p, padded_outputs(p), out);
}

// tables of both directions, 256-byte aligned, then the half-transformed images
struct Layout {
  int pr, pc;
  size_t tab_c, tab_r, total;
};
bool layout(int batch, int rows, int cols, int up, Layout* l) {
  l->pr = prime_part(rows);
  l->pc = prime_part(cols);
  if (!l->pr || !l->pc || batch < 0) return false;
  auto round = [](size_t b) { return (b + 255) / 256 * 256; };
  l->tab_c = 0;
  l->tab_r = round(table_entries(up * cols, l->pc) * sizeof(float2));
  l->total = l->tab_r + round(table_entries(up * rows, l->pr) * sizeof(float2));
  return true;
}

int check(int batch, int rows, int cols, int up, const void* in, const void* mid, const void* out, const void* ws,
          size_t bytes, Layout* l) {
  if (!layout(batch, rows, cols, up, l)) {
    return set_error(PTX_ERR_UNSUPPORTED_SIZE, "%d x %d images: a side is no small multiple of a prime of 37 to 127", rows,
                     cols);
  }
  if (batch == 0) return PTX_OK;
  if (!in || !mid || !out || !ws) return set_error(PTX_ERR_INVALID_ARGUMENT, "null pointer argument");
  if (bytes < l->total) {
    return set_error(PTX_ERR_WORKSPACE, "workspace of %zu bytes is smaller than %zu", bytes, l->total);
  }
  return PTX_OK;
}

}  // namespace
}  // namespace ptx

using namespace ptx;

extern "C" {

size_t ptx_reg_prime_fft_workspace_bytes(int rows, int cols) {
  Layout l;
  return layout(1, rows, cols, 2, &l) ? l.total : 0;
}

int ptx_reg_prime_fft2(const float* images, long long image_stride, long long row_stride, int batch, int rows, int cols,
                       float* half, float* out, void* workspace, size_t workspace_bytes, void* stream) {
  Layout l;
  if (int st = check(batch, rows, cols, 1, images, half, out, workspace, workspace_bytes, &l)) return st;
  if (batch == 0) return PTX_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  float2* tc = reinterpret_cast<float2*>(static_cast<char*>(workspace) + l.tab_c);
  float2* tr = reinterpret_cast<float2*>(static_cast<char*>(workspace) + l.tab_r);
  prof_begin(kMiscKernel, s);
  make_tables(cols, l.pc, tc, s);
  make_tables(rows, l.pr, tr, s);
  prof_end(kMiscKernel, s);
  prof_begin(kMiscKernel, s);
  const PrimeArgs first{nullptr, images, image_stride, row_stride, 1.f,
                        rows, batch, l.pc, tc, reinterpret_cast<float2*>(half)};
  int st = dispatch_lines<false, true, true>(cols / l.pc, first, s);
  const PrimeArgs second{reinterpret_cast<const float2*>(half), nullptr, 0, 0, 1.f,
                         cols, batch, l.pr, tr, reinterpret_cast<float2*>(out)};
  if (!st) st = dispatch_lines<false, false, true>(rows / l.pr, second, s);
  prof_end(kMiscKernel, s);
  return st ? st : cuda_status(cudaGetLastError(), "ptx_reg_prime_fft2 launch");
}

int ptx_reg_prime_correlation(const float* cross_power, int batch, int rows, int cols, float* half, float* correlation,
                              void* workspace, size_t workspace_bytes, void* stream) {
  Layout l;
  if (int st = check(batch, rows, cols, 2, cross_power, half, correlation, workspace, workspace_bytes, &l)) return st;
  if (batch == 0) return PTX_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  float2* tc = reinterpret_cast<float2*>(static_cast<char*>(workspace) + l.tab_c);
  float2* tr = reinterpret_cast<float2*>(static_cast<char*>(workspace) + l.tab_r);
  prof_begin(kMiscKernel, s);
  make_tables(2 * cols, l.pc, tc, s);
  make_tables(2 * rows, l.pr, tr, s);
  prof_end(kMiscKernel, s);
  prof_begin(kMiscKernel, s);
  const PrimeArgs first{reinterpret_cast<const float2*>(cross_power), nullptr, 0, 0, -1.f,
                        rows, batch, l.pc, tc, reinterpret_cast<float2*>(half)};
  int st = dispatch_lines<true, false, true>(cols / l.pc, first, s);
  const PrimeArgs second{reinterpret_cast<const float2*>(half), nullptr, 0, 0, 1.f,
                         2 * cols, batch, l.pr, tr, reinterpret_cast<float2*>(correlation)};
  if (!st) st = dispatch_lines<true, false, false>(rows / l.pr, second, s);
  prof_end(kMiscKernel, s);
  return st ? st : cuda_status(cudaGetLastError(), "ptx_reg_prime_correlation launch");
}

}  // extern "C"
