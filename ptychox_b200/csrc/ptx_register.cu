// Sub-pixel registration: the matrix-multiply DFT refinement of dftregistration.
//
// Reference: matlab/Examples/Near-field Ptychography/+misc/dftregistration.m:102-121 (the
// usfac > 2 branch) with its helper dftups (:150-185): around an initial estimate
// (R_row, R_col) / usfac of the shift, the cross-power spectrum Q = buf2ft .* conj(buf1ft)
// (rows x cols) is inverse-transformed onto an n_out x n_out patch of the grid upsampled by
// usfac (n_out = ceil(1.5 usfac)), the patch's origin at dftshift = fix(n_out / 2):
//
//   out[r][c] = sum_m sum_n kr[r][m] Q[m][n] kc[n][c]
//   kc[n][c]  = exp(-2 pi i fc(n) (c - coff) / (cols usfac)),  coff = dftshift - R_col
//   kr[r][m]  = exp(-2 pi i (r - roff) fr(m) / (rows usfac)),  roff = dftshift - R_row
//
// fr, fc the centred frequencies (k for k < ceil(L/2), else k - L).  CC = conj(out); its
// peak |CC| (the first maximum in column-major order, as MATLAB's find(..., 1, 'first'))
// gives the refined shift.
//
// The dense products cost rows * cols * n_out complex FP64 terms per image (n_out = 900 at
// usfac = 600).  They are not needed: the patch is at most 1.6 pixels wide, so each phase factor
// is a smooth function of the patch coordinate.  With h = dftshift, x = (c - dftshift) / h in
// [-1, 1] and z = 2 pi fc h / (cols usfac), |z| <= 2.52, the Jacobi-Anger expansion
//
//   exp(-i z x) = sum_p eps_p (-i)^p J_p(z) T_p(x),   eps_0 = 1, eps_p = 2
//
// (Abramowitz and Stegun 9.1.44-47; J_p Bessel functions, T_p Chebyshev polynomials)
// separates the frequency from the coordinate.  Its tail after kRank = 24 terms is below
// 2 (z/2)^24 / 24! < 1e-21, under FP64 rounding, so the patch has numerical rank 24:
//
//   Y[m][q] = sum_n Q[m][n] exp(-2 pi i fc(n) R_col / (cols usfac)) eps_q J_q(z_n)
//   M[p][q] = (-i)^(p+q) sum_m exp(-2 pi i fr(m) R_row / (rows usfac)) eps_p J_p(z_m) Y[m][q]
//   out[r][c] = sum_pq T_p(x_r) M[p][q] T_q(x_c)
//
// all in FP64 (the input spectrum stays FP32): at usfac = 600 neighbouring grid points of a
// smooth correlation peak differ in |CC| by parts in 1e5 and less, below what FP32 sums over
// thousands of terms resolve.  The phases exp(-2 pi i f R / (L usfac)) come from the exact
// integer f R mod (L usfac).  Bound: FP64 issue (Y: 48 FMA per spectrum element against 8
// bytes read; patch: 48 FMA per point, nothing written but each CTA's peak).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "ptx_internal.h"

namespace ptx {
namespace {

constexpr int kRank = 24;        // terms of the expansion
constexpr int kProjRows = 64;    // spectrum rows per CTA of the projection
constexpr int kProjK = 32;       // columns per shared-memory stage
constexpr int kProjThreads = 128;
constexpr int kPatchTile = 64;   // patch rows and columns per tile
constexpr int kPatchThreads = 256;
constexpr int kMaxColSplits = 16;  // CTAs that may share a patch's row block

// |out|^2, its column-major index and value at a peak candidate
struct PeakCand {
  double m;
  long long at;
  double2 z;
};

__device__ __forceinline__ int centred_freq(int k, int len) { return k < (len + 1) / 2 ? k : k - len; }

// eps_p J_p(z) by the power series (z/2)^p sum_k (-z^2/4)^k / (k! (k+p)!) (Abramowitz and
// Stegun 9.1.10): at |z| <= 2.52 its terms fall below 1e-18 after 18.
__device__ __forceinline__ double bessel_coefficient(int p, double z) {
  const double half = 0.5 * z, q = -half * half;
  double lead = p ? 2.0 : 1.0;  // eps_p (z/2)^p / p!
  for (int k = 1; k <= p; ++k) lead *= half / k;
  double term = 1.0, sum = 1.0;
  for (int k = 1; k <= 18; ++k) {
    term *= q / (static_cast<double>(k) * (k + p));
    sum += term;
  }
  return lead * sum;
}

// The tables of one call: jr [rows][kRank], jc [cols][kRank] (expansion coefficients of each
// frequency), tt [kRank][n] (T_p at each patch coordinate), and per image the phases of its
// centre, pr [batch][rows] and pc [batch][cols].
__global__ void __launch_bounds__(128) reg_tables_kernel(int batch, int rows, int cols, int n, int usfac, int dftshift,
                                                         const int* __restrict__ row_center,
                                                         const int* __restrict__ col_center, double* __restrict__ jr,
                                                         double* __restrict__ jc, double* __restrict__ tt,
                                                         double2* __restrict__ pr, double2* __restrict__ pc) {
  constexpr double kTwoPi = 6.283185307179586476925286766559;
  const long long lines = rows + cols, coefficients = lines * kRank;
  const long long total = coefficients + n + batch * lines;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    if (i < coefficients) {
      const int l = static_cast<int>(i / kRank), p = static_cast<int>(i - (long long)l * kRank);
      const bool col = l >= rows;
      const int k = col ? l - rows : l, len = col ? cols : rows;
      const double z = kTwoPi * centred_freq(k, len) * dftshift / (static_cast<double>(len) * usfac);
      (col ? jc : jr)[(size_t)k * kRank + p] = bessel_coefficient(p, z);
    } else if (i < coefficients + n) {
      const int c = static_cast<int>(i - coefficients);
      const double x = static_cast<double>(c - dftshift) / dftshift;
      double a = 1.0, b = x;
      for (int p = 0; p < kRank; ++p) {
        tt[(size_t)p * n + c] = a;
        const double next = 2.0 * x * b - a;
        a = b;
        b = next;
      }
    } else {
      const long long j = i - coefficients - n;
      const int b = static_cast<int>(j / lines), l = static_cast<int>(j - b * lines);
      const bool col = l >= rows;
      const int k = col ? l - rows : l, len = col ? cols : rows;
      const long long period = (long long)len * usfac;
      long long ph = (long long)centred_freq(k, len) * (col ? col_center[b] : row_center[b]) % period;
      if (ph < 0) ph += period;
      double sn, cs;
      sincospi(2.0 * static_cast<double>(ph) / static_cast<double>(period), &sn, &cs);
      (col ? pc + (size_t)b * cols : pr + (size_t)b * rows)[k] = make_double2(cs, -sn);
    }
  }
}

// D += A B on the FP64 tensor unit, A 8 x 4 (row-major fragment), B 4 x 8 (column-major
// fragment), D 8 x 8: lane l holds A[l / 4][l % 4], B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// Y for a block of kProjRows rows of one image, and the block's share of M, written to
// part [b][row block][kRank][kRank].  Both products run on the FP64 tensor unit, real and
// imaginary parts apart.  Y: warp w owns rows 16 w .. 16 w + 15 (2 x 3 fragments, 12 products
// per 4 columns against 7 shared loads); the next kProjK columns travel from global memory to
// registers meanwhile.  The share: warp w < 3 owns terms p in [8 w, 8 w + 8).
__global__ void __launch_bounds__(kProjThreads, 4) reg_project_kernel(const float2* __restrict__ q, int rows, int cols,
                                                                      const double* __restrict__ jr,
                                                                      const double* __restrict__ jc,
                                                                      const double2* __restrict__ pr,
                                                                      const double2* __restrict__ pc,
                                                                      double2* __restrict__ part) {
  // pitches = 4 and 12 (mod 16): the 4 x 4 lanes of half a fragment hit distinct banks
  constexpr int QP = kProjRows + 4, JP = kRank + 4;
  constexpr int kLoads = kProjRows * kProjK / kProjThreads;
  constexpr int kStage = kProjK * (2 * QP + JP), kShare = kProjRows * 3 * JP;
  __shared__ double buf[kStage > kShare ? kStage : kShare];
  double* qr = buf;                    // [kProjK][QP]: rotated spectrum, real
  double* qi = qr + kProjK * QP;       // imaginary
  double* js = qi + kProjK * QP;       // [kProjK][JP]: column coefficients
  const int b = blockIdx.y, m0 = blockIdx.x * kProjRows;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int i = lane >> 2, j = lane & 3;
  const float2* qb = q + (size_t)b * rows * cols;
  const double2* ph = pc + (size_t)b * cols;
  double yr[2][3][2], yi[2][3][2];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 3; ++v) yr[u][v][0] = yr[u][v][1] = yi[u][v][0] = yi[u][v][1] = 0.0;
  // lanes run along a row (256-byte reads): thread (kk, mm) loads rows mm + 4 l of column k0 + kk
  const int kk = tid % kProjK, mm = tid / kProjK;
  float2 x[kLoads];
  auto load = [&](int k0) {
    const int k = k0 + kk;
#pragma unroll
    for (int l = 0; l < kLoads; ++l) {
      const int m = m0 + mm + (kProjThreads / kProjK) * l;
      x[l] = k < cols && m < rows ? qb[(size_t)m * cols + k] : make_float2(0.f, 0.f);
    }
  };
  load(0);
  for (int k0 = 0; k0 < cols; k0 += kProjK) {
    const double2 f = k0 + kk < cols ? ph[k0 + kk] : make_double2(0.0, 0.0);
#pragma unroll
    for (int l = 0; l < kLoads; ++l) {
      const double xr = x[l].x, xi = x[l].y;
      const int at = kk * QP + mm + (kProjThreads / kProjK) * l;
      qr[at] = fma(xr, f.x, -xi * f.y);
      qi[at] = fma(xr, f.y, xi * f.x);
    }
    for (int e = tid; e < kProjK * kRank; e += kProjThreads) {
      const int k = e / kRank;
      js[k * JP + e - k * kRank] = k0 + k < cols ? jc[(size_t)k0 * kRank + e] : 0.0;
    }
    __syncthreads();
    if (k0 + kProjK < cols) load(k0 + kProjK);
#pragma unroll 2
    for (int k = 0; k < kProjK; k += 4) {
      double c[3];
#pragma unroll
      for (int v = 0; v < 3; ++v) c[v] = js[(k + j) * JP + 8 * v + i];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int at = (k + j) * QP + 16 * w + 8 * u + i;
        const double ar = qr[at], ai = qi[at];
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          mma_f64(yr[u][v], ar, c[v]);
          mma_f64(yi[u][v], ai, c[v]);
        }
      }
    }
    __syncthreads();
  }
  // Y times the row phases, and the rows' coefficients (zero for rows past the last)
  double* ysr = buf;                       // [kProjRows][JP]
  double* ysi = ysr + kProjRows * JP;
  double* rs = ysi + kProjRows * JP;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int r = 16 * w + 8 * u + i;
    const double2 f = m0 + r < rows ? pr[(size_t)b * rows + m0 + r] : make_double2(0.0, 0.0);
#pragma unroll
    for (int v = 0; v < 3; ++v)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int at = r * JP + 8 * v + 2 * j + k;
        ysr[at] = fma(yr[u][v][k], f.x, -yi[u][v][k] * f.y);
        ysi[at] = fma(yr[u][v][k], f.y, yi[u][v][k] * f.x);
      }
  }
  for (int e = tid; e < kProjRows * kRank; e += kProjThreads) {
    const int r = e / kRank;
    rs[r * JP + e - r * kRank] = m0 + r < rows ? jr[(size_t)m0 * kRank + e] : 0.0;
  }
  __syncthreads();
  if (w >= 3) return;
  double sr[3][2], si[3][2];
#pragma unroll
  for (int v = 0; v < 3; ++v) sr[v][0] = sr[v][1] = si[v][0] = si[v][1] = 0.0;
#pragma unroll 4
  for (int m = 0; m < kProjRows; m += 4) {
    const double a = rs[(m + j) * JP + 8 * w + i];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      mma_f64(sr[v], a, ysr[(m + j) * JP + 8 * v + i]);
      mma_f64(si[v], a, ysi[(m + j) * JP + 8 * v + i]);
    }
  }
  double2* out = part + ((size_t)b * gridDim.x + blockIdx.x) * kRank * kRank;
#pragma unroll
  for (int v = 0; v < 3; ++v)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int p = 8 * w + i, qq = 8 * v + 2 * j + k;
      const double re = sr[v][k], im = si[v][k];
      double2 o;  // times (-i)^(p+q)
      switch ((p + qq) & 3) {
        case 0: o = make_double2(re, im); break;
        case 1: o = make_double2(im, -re); break;
        case 2: o = make_double2(-re, -im); break;
        default: o = make_double2(-im, re); break;
      }
      out[p * kRank + qq] = o;
    }
}

__device__ __forceinline__ bool better(const PeakCand& a, const PeakCand& b) {
  return a.m > b.m || (a.m == b.m && a.at < b.at);
}

__device__ __forceinline__ PeakCand warp_best(PeakCand c) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    PeakCand x;
    x.m = __shfl_xor_sync(0xffffffffu, c.m, o);
    x.at = __shfl_xor_sync(0xffffffffu, c.at, o);
    x.z.x = __shfl_xor_sync(0xffffffffu, c.z.x, o);
    x.z.y = __shfl_xor_sync(0xffffffffu, c.z.y, o);
    if (better(x, c)) c = x;
  }
  return c;
}

// no candidate yet: any |out|^2 >= 0 is better, a NaN is not
__device__ __forceinline__ PeakCand no_peak() {
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  return {-1.0, 0x7fffffffffffffffll, make_double2(nan, nan)};
}

// The patch of one image on a block of kPatchTile rows and every gridDim.y-th column tile, its
// points evaluated and compared without being stored.  M is the sum of its row blocks' shares.
// Warp (wr, wc) owns a 32 x 16 piece of a 64 x 64 tile as 4 x 2 matrix fragments, real and
// imaginary parts apart: 16 products per 4 terms against 10 shared loads (a scalar form, 32 FMA
// against 8 loads, was bound by its loads: 0.51 ms on average per call of the tracking of 200
// crops of 472^2 at usfac 600 and 100, against 0.37).
__global__ void __launch_bounds__(kPatchThreads, 2) reg_patch_kernel(const double2* __restrict__ part, int shares,
                                                                     const double* __restrict__ tt, int n,
                                                                     PeakCand* __restrict__ cand) {
  constexpr int ZP = kPatchTile + 4;  // pitch = 4 (mod 16): the 4 x 8 lanes of a fragment hit distinct banks
  __shared__ double zr[kRank][ZP], zi[kRank][ZP];  // sum_p T_p(x_r) M[p][q]
  __shared__ double cs[kRank][ZP];                 // T_q(x_c)
  __shared__ PeakCand best_s[kPatchThreads / 32];
  const int b = blockIdx.z, r0 = blockIdx.x * kPatchTile;
  const int tid = threadIdx.x, lane = tid & 31;
  const int wr = (tid >> 5) & 1, wc = tid >> 6;
  const int i = lane >> 2, j = lane & 3;
  {
    // M in the space of the column table, T_p(x_r) of the row block in zr's rows until zi is formed
    double2* ms = reinterpret_cast<double2*>(&cs[0][0]);
    static_assert(sizeof(double2) * kRank * kRank <= sizeof(cs), "M fits the column table");
    const double2* mb = part + (size_t)b * shares * kRank * kRank;
    for (int e = tid; e < kRank * kRank; e += kPatchThreads) {
      double2 s = mb[e];
      for (int k = 1; k < shares; ++k) {
        const double2 x = mb[(size_t)k * kRank * kRank + e];
        s.x += x.x;
        s.y += x.y;
      }
      ms[e] = s;
    }
    const int rr = tid % kPatchTile, r = r0 + rr;
    double t[kRank];
#pragma unroll
    for (int p = 0; p < kRank; ++p) t[p] = r < n ? tt[(size_t)p * n + r] : 0.0;
    __syncthreads();
    for (int q = tid / kPatchTile; q < kRank; q += kPatchThreads / kPatchTile) {
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int p = 0; p < kRank; ++p) {
        const double2 m = ms[p * kRank + q];
        s.x = fma(m.x, t[p], s.x);
        s.y = fma(m.y, t[p], s.y);
      }
      zr[q][rr] = s.x;
      zi[q][rr] = s.y;
    }
  }
  PeakCand best = no_peak();
  for (long long c0 = (long long)blockIdx.y * kPatchTile; c0 < n; c0 += (long long)gridDim.y * kPatchTile) {
    __syncthreads();  // zr and zi are complete, and cs is free
    for (int e = tid; e < kRank * kPatchTile; e += kPatchThreads) {
      const long long c = c0 + e % kPatchTile;
      cs[e / kPatchTile][e % kPatchTile] = c < n ? tt[(size_t)(e / kPatchTile) * n + c] : 0.0;
    }
    __syncthreads();
    double re[4][2][2], im[4][2][2];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 2; ++v) re[u][v][0] = re[u][v][1] = im[u][v][0] = im[u][v][1] = 0.0;
#pragma unroll
    for (int q = 0; q < kRank; q += 4) {
      double w[2];
#pragma unroll
      for (int v = 0; v < 2; ++v) w[v] = cs[q + j][wc * 16 + 8 * v + i];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double ar = zr[q + j][wr * 32 + 8 * u + i], ai = zi[q + j][wr * 32 + 8 * u + i];
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          mma_f64(re[u][v], ar, w[v]);
          mma_f64(im[u][v], ai, w[v]);
        }
      }
    }
#pragma unroll
    for (int v = 0; v < 2; ++v)
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const long long r = r0 + wr * 32 + 8 * u + i, c = c0 + wc * 16 + 8 * v + 2 * j + k;
          if (r < n && c < n) {
            const double2 z = make_double2(re[u][v][k], im[u][v][k]);
            const PeakCand x{z.x * z.x + z.y * z.y, c * n + r, z};
            if (better(x, best)) best = x;
          }
        }
  }
  best = warp_best(best);
  if (lane == 0) best_s[tid >> 5] = best;
  __syncthreads();
  if (tid < 32) {
    best = warp_best(tid < kPatchThreads / 32 ? best_s[tid] : no_peak());
    if (tid == 0) cand[((size_t)b * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = best;
  }
}

// Peak of |out[b]| over its candidates, the first in column-major order on ties (MATLAB's
// find(..., 1, 'first')); writes (r, c) and conj(out[r][c]) (= CC at the peak).
__global__ void __launch_bounds__(32) reg_peak_kernel(const PeakCand* __restrict__ cand, int count, int n,
                                                      int* __restrict__ peak_rc, double2* __restrict__ peak_cc) {
  const int b = blockIdx.x;
  PeakCand best = no_peak();
  for (int i = threadIdx.x; i < count; i += 32) {
    const PeakCand x = cand[(size_t)b * count + i];
    if (better(x, best)) best = x;
  }
  best = warp_best(best);
  if (threadIdx.x == 0) {
    const long long at = best.m >= 0.0 ? best.at : 0;  // every point a NaN: the first one
    peak_rc[2 * b] = static_cast<int>(at % n);
    peak_rc[2 * b + 1] = static_cast<int>(at / n);
    peak_cc[b] = make_double2(best.z.x, -best.z.y);
  }
}

// ---- the initial estimate: peak of the twice-upsampled cross-correlation -----------------------
// Frequency k of a line of n bins in the line zero-padded to 2 n (FTpad,
// dftregistration.m:189-224): the non-negative ones keep their bins, the negative ones move to
// the end.
__device__ __forceinline__ int unpadded_bin(int c, int n) {
  const int half = n - n / 2;
  return c < half ? c : (c >= n + half ? c - n : -1);
}

// One pass from the two spectra to the product spec1 conj(spec2), rows zero-padded to 2 cols
// (what a library's row transform reads; null where the padding is the transform's own), and the
// cross-power conj(spec1) spec2 the refinement reads.
// HBM-bound: 8 B read (spec1 of a tracked stack is one image, resident in L2), 24 B written.
__global__ void __launch_bounds__(256) reg_cross_power_kernel(const float2* __restrict__ s1, bool one,
                                                              const float2* __restrict__ s2, int rows, int cols,
                                                              float2* __restrict__ padded, float2* __restrict__ q) {
  const long long row = (long long)blockIdx.y * rows + blockIdx.x;
  const float2* a = s1 + (one ? (long long)blockIdx.x : row) * cols;
  const float2* b = s2 + row * cols;
  for (int c = threadIdx.x; c < 2 * cols; c += blockDim.x) {
    const int k = unpadded_bin(c, cols);
    float2 v = make_float2(0.f, 0.f);
    if (k >= 0) {
      const float2 z = cmulc(b[k], a[k]);
      q[row * cols + k] = z;
      v = cconj(z);
    }
    if (padded) padded[row * 2 * cols + c] = v;
  }
}

// [batch][rows][2 cols] -> [batch][2 cols][2 rows]: transposed, the rows zero-padded, so that
// the second transform again runs along contiguous lines (and the transform along the rows is
// taken over the rows that are not zero only).  32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256) reg_pad_transpose_kernel(const float2* __restrict__ in, int rows, int cols,
                                                                float2* __restrict__ out) {
  __shared__ float2 tile[32][33];
  const int xtiles = (2 * cols + 31) / 32;
  const int x0 = static_cast<int>(blockIdx.x % xtiles) * 32, y0 = static_cast<int>(blockIdx.x / xtiles) * 32;
  const int lx = threadIdx.x % 32, ly = threadIdx.x / 32;
  const float2* ib = in + (size_t)blockIdx.y * rows * 2 * cols;
  float2* ob = out + (size_t)blockIdx.y * 4 * rows * cols;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int y = y0 + ly + 8 * i, x = x0 + lx;
    const int r = y < 2 * rows ? unpadded_bin(y, rows) : -1;
    tile[ly + 8 * i][lx] = r >= 0 && x < 2 * cols ? ib[(size_t)r * 2 * cols + x] : make_float2(0.f, 0.f);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int x = x0 + ly + 8 * i, y = y0 + lx;
    if (x < 2 * cols && y < 2 * rows) ob[(size_t)x * 2 * rows + y] = tile[lx][ly + 8 * i];
  }
}

constexpr int kCorrThreads = 256;
constexpr int kCorrChunk = 1 << 15;  // correlation values per CTA

// Peak candidates of chunks of |corr[b]|, `count` values in column-major order.  A value with
// an infinite part has magnitude infinity, and a NaN beats every number (as a maximum over the
// magnitudes would have it); |.|^2 of FP32 values cannot reach the two stand-ins in FP64.
__global__ void __launch_bounds__(kCorrThreads) reg_corr_peak_kernel(const float2* __restrict__ corr, long long count,
                                                                     PeakCand* __restrict__ cand) {
  constexpr double kInfinite = 1e300, kNan = 1e301;
  __shared__ PeakCand best_s[kCorrThreads / 32];
  const float2* cb = corr + (size_t)blockIdx.y * count;
  const long long l1 = min(count, ((long long)blockIdx.x + 1) * kCorrChunk);
  PeakCand best = no_peak();
#pragma unroll 4
  for (long long l = (long long)blockIdx.x * kCorrChunk + threadIdx.x; l < l1; l += kCorrThreads) {
    const float2 z = cb[l];
    const double x = z.x, y = z.y;
    double m = x * x + y * y;
    if (!(m < kInfinite)) m = isinf(z.x) || isinf(z.y) ? kInfinite : kNan;
    if (m > best.m) {  // l increases per thread, so the thread's first maximum is kept
      best.m = m;
      best.at = l;
      best.z = make_double2(x, y);
    }
  }
  best = warp_best(best);
  if ((threadIdx.x & 31) == 0) best_s[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x < 32) {
    best = warp_best(threadIdx.x < kCorrThreads / 32 ? best_s[threadIdx.x] : no_peak());
    if (threadIdx.x == 0) cand[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = best;
  }
}

// From an image's candidates: the peak in half pixels (signed), the refinement's centres
// round(shift usfac) (halves away from zero, MATLAB's round) and the correlation there.
__global__ void __launch_bounds__(32) reg_estimate_kernel(const PeakCand* __restrict__ cand, int count, int rows,
                                                          int cols, int usfac, int* __restrict__ half_rc,
                                                          int* __restrict__ row_center, int* __restrict__ col_center,
                                                          double2* __restrict__ peak_cc) {
  const int b = blockIdx.x;
  PeakCand best = no_peak();
  for (int i = threadIdx.x; i < count; i += 32) {
    const PeakCand x = cand[(size_t)b * count + i];
    if (better(x, best)) best = x;
  }
  best = warp_best(best);
  if (threadIdx.x == 0) {
    int r = static_cast<int>(best.at % (2 * rows)), c = static_cast<int>(best.at / (2 * rows));
    if (r >= rows) r -= 2 * rows;
    if (c >= cols) c -= 2 * cols;
    half_rc[2 * b] = r;
    half_rc[2 * b + 1] = c;
    auto centre = [&](int half) {
      const double v = 0.5 * half * usfac, a = floor(fabs(v) + 0.5);
      return static_cast<int>(v < 0.0 ? -a : a);
    };
    row_center[b] = centre(r);
    col_center[b] = centre(c);
    peak_cc[b] = best.z;
  }
}

// sum |spec[b]|^2 in FP64 over `parts` pieces of each image, one CTA per piece (the same order of
// summation on every call).  A CTA alone reads 60 GB/s, bound by the latency of its loads, so that few
// and large images are shared out (us, with the sum over the pieces, in one piece -> as
// ptx_reg_energy_parts has it): one of 4096^2 2290 -> 31 (4.3 TB/s), one of 512^2 27 -> 10, 64 of
// 512^2 48 -> 29; 200 of 472^2 keep one piece (60; 68 in three).
__global__ void __launch_bounds__(1024) reg_energy_kernel(const float2* __restrict__ spec, long long count, int parts,
                                                          double* __restrict__ out) {
  __shared__ double sums[32];
  const long long image = blockIdx.x / parts, p = blockIdx.x - image * parts;
  const float2* sb = spec + image * count;
  const long long end = count * (p + 1) / parts;
  double s = 0.0;
#pragma unroll 4
  for (long long i = count * p / parts + threadIdx.x; i < end; i += 1024) {
    const double x = sb[i].x, y = sb[i].y;
    s = fma(x, x, fma(y, y, s));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = sums[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
  }
}

int corr_chunks(int rows, int cols) {
  return static_cast<int>((4LL * rows * cols + kCorrChunk - 1) / kCorrChunk);
}

// Shape checks shared by the entry points of the initial estimate.
int reg_check_stack(int batch, int rows, int cols) {
  if (batch < 0 || rows <= 0 || cols <= 0) return set_error(PTX_ERR_INVALID_ARGUMENT, "non-positive shape");
  if (rows > (1 << 29) || cols > (1 << 29)) return set_error(PTX_ERR_UNSUPPORTED_SIZE, "image side above 2^29");
  return PTX_OK;
}

// f(first image, images) over slabs of a batch that fit a grid dimension
template <typename F>
void for_slabs(int batch, F&& f) {
  for (int b0 = 0; b0 < batch; b0 += 65535) f((size_t)b0, std::min(65535, batch - b0));
}

int reg_out_size(int usfac) { return (3 * usfac + 1) / 2; }  // ceil(1.5 usfac)

// Workspace of a call: the shared tables, then per image the phases, its row blocks' shares of M
// and the peak candidates of its CTAs.
struct RegLayout {
  size_t jr, jc, tt, pr, pc, part, cand, bytes;
  int shares, rblocks, max_splits;
};
RegLayout reg_layout(int batch, int rows, int cols, int usfac) {
  const size_t n = static_cast<size_t>(reg_out_size(usfac)), b = static_cast<size_t>(batch);
  RegLayout l{};
  l.rblocks = static_cast<int>((n + kPatchTile - 1) / kPatchTile);
  l.max_splits = std::min(l.rblocks, kMaxColSplits);
  l.shares = (rows + kProjRows - 1) / kProjRows;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at = align_up(at + bytes, 256);
    return here;
  };
  l.jr = take(sizeof(double) * rows * kRank);
  l.jc = take(sizeof(double) * cols * kRank);
  l.tt = take(sizeof(double) * n * kRank);
  l.pr = take(sizeof(double2) * b * rows);
  l.pc = take(sizeof(double2) * b * cols);
  l.part = take(sizeof(double2) * b * l.shares * kRank * kRank);
  l.cand = take(sizeof(PeakCand) * b * l.rblocks * l.max_splits);
  l.bytes = at;
  return l;
}

}  // namespace
}  // namespace ptx

using namespace ptx;

extern "C" {

size_t ptx_reg_workspace_bytes(int batch, int rows, int cols, int usfac) {
  if (batch <= 0 || rows <= 0 || cols <= 0 || usfac <= 2) return 0;
  // the size of the patch and the half-transformed spectrum, which callers allot; the tables of
  // a patch of a few points need more than that
  const size_t n = static_cast<size_t>(reg_out_size(usfac));
  const size_t patch = sizeof(double2) * (size_t)batch * n * ((size_t)rows + n);
  return std::max(patch, reg_layout(batch, rows, cols, usfac).bytes);
}

int ptx_reg_upsampled_peak(const float* cross_power, int batch, int rows, int cols, int usfac,
                           const int* row_center, const int* col_center, int* peak_rc, double* peak_cc,
                           void* workspace, size_t workspace_bytes, void* stream) {
  if (batch < 0 || rows <= 0 || cols <= 0) return set_error(PTX_ERR_INVALID_ARGUMENT, "non-positive shape");
  if (usfac <= 2 || usfac > 100000) {
    return set_error(PTX_ERR_INVALID_ARGUMENT, "usfac must lie in [3, 100000] for the upsampled refinement");
  }
  if (batch == 0) return PTX_OK;
  if (!cross_power || !row_center || !col_center || !peak_rc || !peak_cc || !workspace) {
    return set_error(PTX_ERR_INVALID_ARGUMENT, "null pointer argument");
  }
  if ((long long)rows * usfac > (1ll << 30) || (long long)cols * usfac > (1ll << 30)) {
    return set_error(PTX_ERR_UNSUPPORTED_SIZE, "rows or cols times usfac exceeds 2^30");
  }
  const size_t need = ptx_reg_workspace_bytes(batch, rows, cols, usfac);
  if (workspace_bytes < need) {
    return set_error(PTX_ERR_WORKSPACE, "workspace of %zu bytes is smaller than %zu", workspace_bytes, need);
  }
  if (batch > 65535) return set_error(PTX_ERR_UNSUPPORTED_SIZE, "at most 65535 images per call");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int n = reg_out_size(usfac);
  const int dftshift = n / 2;
  const RegLayout l = reg_layout(batch, rows, cols, usfac);
  char* ws = static_cast<char*>(workspace);
  double* jr = reinterpret_cast<double*>(ws + l.jr);
  double* jc = reinterpret_cast<double*>(ws + l.jc);
  double* tt = reinterpret_cast<double*>(ws + l.tt);
  double2* pr = reinterpret_cast<double2*>(ws + l.pr);
  double2* pc = reinterpret_cast<double2*>(ws + l.pc);
  double2* part = reinterpret_cast<double2*>(ws + l.part);
  PeakCand* cand = reinterpret_cast<PeakCand*>(ws + l.cand);
  const long long entries = (long long)(batch + kRank) * (rows + cols) + n;
  const unsigned tblocks = static_cast<unsigned>(std::min<long long>((entries + 127) / 128, (long long)sm_count() * 16));
  prof_begin(kMiscKernel, s);
  reg_tables_kernel<<<tblocks, 128, 0, s>>>(batch, rows, cols, n, usfac, dftshift, row_center, col_center, jr, jc, tt,
                                            pr, pc);
  prof_end(kMiscKernel, s);
  prof_begin(kMiscKernel, s);
  reg_project_kernel<<<dim3(l.shares, batch), kProjThreads, 0, s>>>(reinterpret_cast<const float2*>(cross_power), rows,
                                                                    cols, jr, jc, pr, pc, part);
  prof_end(kMiscKernel, s);
  // few images: several CTAs share a row block of the patch, so that the SMs are covered
  const long long blocks = (long long)l.rblocks * batch;
  const int splits = static_cast<int>(std::min<long long>(l.max_splits, std::max<long long>(1, 4LL * sm_count() / blocks)));
  prof_begin(kMiscKernel, s);
  reg_patch_kernel<<<dim3(l.rblocks, splits, batch), kPatchThreads, 0, s>>>(part, l.shares, tt, n, cand);
  prof_end(kMiscKernel, s);
  prof_begin(kMiscKernel, s);
  reg_peak_kernel<<<batch, 32, 0, s>>>(cand, l.rblocks * splits, n, peak_rc, reinterpret_cast<double2*>(peak_cc));
  prof_end(kMiscKernel, s);
  return cuda_status(cudaGetLastError(), "ptx_reg_upsampled_peak launch");
}

int ptx_reg_cross_power(const float* spec1, int batch1, const float* spec2, int batch, int rows, int cols,
                        float* padded, float* cross_power, void* stream) {
  if (int st = reg_check_stack(batch, rows, cols)) return st;
  if (batch1 != 1 && batch1 != batch) return set_error(PTX_ERR_INVALID_ARGUMENT, "spec1 holds 1 or %d images", batch);
  if (batch == 0) return PTX_OK;
  if (!spec1 || !spec2 || !cross_power) return set_error(PTX_ERR_INVALID_ARGUMENT, "null pointer argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  prof_begin(kMiscKernel, s);
  const size_t image = (size_t)rows * cols;
  for_slabs(batch, [&](size_t b0, int nb) {
    reg_cross_power_kernel<<<dim3(rows, nb), 256, 0, s>>>(
        reinterpret_cast<const float2*>(spec1) + (batch1 == 1 ? 0 : b0 * image), batch1 == 1,
        reinterpret_cast<const float2*>(spec2) + b0 * image, rows, cols,
        padded ? reinterpret_cast<float2*>(padded) + 2 * b0 * image : nullptr,
        reinterpret_cast<float2*>(cross_power) + b0 * image);
  });
  prof_end(kMiscKernel, s);
  return cuda_status(cudaGetLastError(), "ptx_reg_cross_power launch");
}

int ptx_reg_pad_transpose(const float* in, int batch, int rows, int cols, float* out, void* stream) {
  if (int st = reg_check_stack(batch, rows, cols)) return st;
  if (batch == 0) return PTX_OK;
  if (!in || !out) return set_error(PTX_ERR_INVALID_ARGUMENT, "null pointer argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  prof_begin(kMiscKernel, s);
  const size_t image = (size_t)rows * cols;
  const unsigned tiles = static_cast<unsigned>((2LL * cols + 31) / 32 * ((2LL * rows + 31) / 32));
  for_slabs(batch, [&](size_t b0, int nb) {
    reg_pad_transpose_kernel<<<dim3(tiles, nb), 256, 0, s>>>(reinterpret_cast<const float2*>(in) + 2 * b0 * image, rows,
                                                             cols, reinterpret_cast<float2*>(out) + 4 * b0 * image);
  });
  prof_end(kMiscKernel, s);
  return cuda_status(cudaGetLastError(), "ptx_reg_pad_transpose launch");
}

size_t ptx_reg_estimate_workspace_bytes(int batch, int rows, int cols) {
  if (batch <= 0 || rows <= 0 || cols <= 0) return 0;
  return sizeof(PeakCand) * (size_t)batch * corr_chunks(rows, cols);
}

int ptx_reg_estimate(const float* correlation, int batch, int rows, int cols, int usfac, int* half_rc, int* row_center,
                     int* col_center, double* peak_cc, void* workspace, size_t workspace_bytes, void* stream) {
  if (int st = reg_check_stack(batch, rows, cols)) return st;
  if (usfac < 2 || (long long)std::max(rows, cols) * usfac > (1ll << 30)) {
    return set_error(PTX_ERR_INVALID_ARGUMENT, "usfac must be at least 2 and usfac times a side at most 2^30");
  }
  if (batch == 0) return PTX_OK;
  if (!correlation || !half_rc || !row_center || !col_center || !peak_cc || !workspace) {
    return set_error(PTX_ERR_INVALID_ARGUMENT, "null pointer argument");
  }
  if (workspace_bytes < ptx_reg_estimate_workspace_bytes(batch, rows, cols)) {
    return set_error(PTX_ERR_WORKSPACE, "workspace of %zu bytes is smaller than %zu", workspace_bytes,
                     ptx_reg_estimate_workspace_bytes(batch, rows, cols));
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  PeakCand* cand = static_cast<PeakCand*>(workspace);
  const int chunks = corr_chunks(rows, cols);
  prof_begin(kMiscKernel, s);
  for_slabs(batch, [&](size_t b0, int nb) {
    reg_corr_peak_kernel<<<dim3(chunks, nb), kCorrThreads, 0, s>>>(
        reinterpret_cast<const float2*>(correlation) + 4 * b0 * rows * cols, 4LL * rows * cols, cand + b0 * chunks);
  });
  prof_end(kMiscKernel, s);
  prof_begin(kMiscKernel, s);
  reg_estimate_kernel<<<batch, 32, 0, s>>>(cand, chunks, rows, cols, usfac, half_rc, row_center, col_center,
                                           reinterpret_cast<double2*>(peak_cc));
  prof_end(kMiscKernel, s);
  return cuda_status(cudaGetLastError(), "ptx_reg_estimate launch");
}

int ptx_reg_energy_parts(int batch, int rows, int cols) {
  if (batch <= 0 || rows <= 0 || cols <= 0) return 1;
  // at most one wave of CTAs (two of 1024 threads per SM), of at least 2^15 values each: below that
  // the sum over the pieces costs what they gain
  const long long resident = 2LL * sm_count() / batch, most = (long long)rows * cols >> 15;
  return static_cast<int>(std::max(1LL, std::min(resident, most)));
}

int ptx_reg_partial_energy(const float* spec, int batch, int rows, int cols, int parts, double* energy, void* stream) {
  if (int st = reg_check_stack(batch, rows, cols)) return st;
  if (parts < 1 || (long long)parts * batch > 0x7fffffff) return set_error(PTX_ERR_INVALID_ARGUMENT, "parts out of range");
  if (batch == 0) return PTX_OK;
  if (!spec || !energy) return set_error(PTX_ERR_INVALID_ARGUMENT, "null pointer argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  prof_begin(kMiscKernel, s);
  reg_energy_kernel<<<batch * parts, 1024, 0, s>>>(reinterpret_cast<const float2*>(spec), (long long)rows * cols, parts,
                                                   energy);
  prof_end(kMiscKernel, s);
  return cuda_status(cudaGetLastError(), "ptx_reg_energy launch");
}

int ptx_reg_energy(const float* spec, int batch, int rows, int cols, double* energy, void* stream) {
  return ptx_reg_partial_energy(spec, batch, rows, cols, 1, energy, stream);
}

}  // extern "C"
