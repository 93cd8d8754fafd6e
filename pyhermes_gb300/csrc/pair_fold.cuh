// Pair products on the symmetry-folded spectrum.
//
// The image set of a mode (x, y, z) is {x, L-x} x {y, L-y} x {z, L-z} (and
// the same shifted by multiples of L at a larger bandwidth), so a
// window that is even in every component and symmetric in x and y (every
// isotropic window, and the cylindrical ones with the line of sight on z)
// has the same FFT kernel on the up to eight columns (+-x, +-y), (+-y, +-x).
// pp_fold_kernel adds the pair products T = w_z Re(F_i conj F_j) of those
// columns into one, for x >= y in [0, L/2]: the passes over bins then walk
// (L/2+1)(L/2+2)/2 columns instead of L^2.
//
// An isotropic window is a function of n2 = |k L|^2 alone, so at bandwidth 1
// its pair product is a sum over n2:
//   sum_k T(k) K_b(k) = sum_n2 W_b(n2) Hist(n2),
//   Hist(n2) = sum over modes and images with |image|^2 = n2 of P P P T.
// Hist does not depend on the bin: pp_hist_kernel builds it once (8 adds per
// folded mode, which is what bounds it: scattered 64-bit atomics on an array
// that stays in L2; P P P W is also symmetric in z, so the modes are folded once
// more, onto x >= y >= z) and pp_radial_bins_kernel evaluates each bin's window
// once per n2, 3 L^2 + 1 values, instead of 8 times per mode.  The histogram
// is in 64-bit fixed point (exponent from the largest |T|), so its sums are
// exact and do not depend on the order of the atomics.  It has two levels: a
// contribution that is a whole number of quanta, 2^-46 of the largest |T|, goes
// to the first, any other to the second, whose quanta are 2^-26 of those.  All 24
// bits of a float32 contribution therefore count down to 2^-48 of the largest |T|
// (one level lost them from 2^-18 on, and a mode below 2^-43 altogether: a window
// that does not weigh the large modes, over a mean or a steep spectrum, then
// had no more than its strongest few bits).
#pragma once

#include "pair_products.cuh"

namespace hermes {

constexpr int kHistThreads = 256;
// max |T| < 2^46 quanta.  pp_hist_kernel adds sums of up to three T, and an n2
// has at most 3234 images (L = 1024): below 2^60.  Values below 2^24 quanta, of the
// second level's below 2^50, stay below 2^62 there.
constexpr int kHistBits = 46;
constexpr int kFineBits = 26;
constexpr int kLevels = 2;
constexpr int kRadialPerBlock = 4096;
constexpr int kRadialBins = 4;      // bins per block of pp_radial_bins_kernel

__host__ __device__ __forceinline__ long long fold_columns(int L) {
  const long long H = L / 2 + 1;
  return H * (H + 1) / 2;
}

// (x, y), x >= y, of folded column c = x (x + 1) / 2 + y.
__device__ __forceinline__ void fold_xy(int c, int& x, int& y) {
  x = (int)((sqrtf(8.f * (float)c + 1.f) - 1.f) * 0.5f);
  while (x * (x + 1) / 2 > c) --x;
  while ((x + 1) * (x + 2) / 2 <= c) ++x;
  y = c - x * (x + 1) / 2;
}

// T[column][z] of the folded columns of one pair (si, sj), one warp per
// column; the largest |T| (as float bits; a NaN has the largest) in maxbits.
// The up to eight products are added with their rounding errors kept (the pass is
// bound by its reads), so that T is rounded once however they cancel.
// One launch per pair: 0.098 ms for an auto pair at J = 9 (0.54 GB, 5.5 TB/s);
// two pairs of different spectra in one launch took 0.57 ms.
__global__ void __launch_bounds__(kHistThreads)
pp_fold_kernel(const float2* __restrict__ si, const float2* __restrict__ sj, int L, int exclude_k0, float* __restrict__ T,
               unsigned* __restrict__ maxbits) {
  const int H = L / 2 + 1, Lm = L - 1;
  const int ncol = (int)fold_columns(L);
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * (kHistThreads / 32);
  const bool same = si == sj;
  unsigned mx = 0u;
  for (int c = blockIdx.x * (kHistThreads / 32) + (threadIdx.x >> 5); c < ncol; c += nw) {
    int x, y;
    fold_xy(c, x, y);
    const bool rx = x != 0 && 2 * x != L, ry = y != 0 && 2 * y != L, sw = x != y;
    // rows (x, y), (-x, y), (x, -y), (-x, -y), then the same with x and y exchanged
    const int xs[2] = {x, (L - x) & Lm}, ys[2] = {y, (L - y) & Lm};
    for (int z = lane; z < H; z += 32) {
      float t = 0.f, lost = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int i = r & 1, j = (r >> 1) & 1, s = r >> 2;
        if ((i && !rx) || (j && !ry) || (s && !sw)) continue;
        const long long row = s ? (long long)ys[j] * L + xs[i] : (long long)xs[i] * L + ys[j];
        const long long m = row * H + z;
        const float2 u = si[m];
        const float2 v = same ? u : sj[m];
        float e;
        two_sum(t, u.x * v.x + u.y * v.y, t, e);
        lost += e;
      }
      const float wgt = (z == 0 || 2 * z == L) ? 1.f : 2.f;
      const float v = (exclude_k0 && c == 0 && z == 0) ? 0.f : wgt * (isfinite(t) ? t + lost : t);
      T[(size_t)c * H + z] = v;
      mx = max(mx, __float_as_uint(fabsf(v)));
    }
  }
  const unsigned m = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0 && m) atomicMax(maxbits, m);
}

// Exponent shift of the fixed point: quanta = v * 2^shift, |v| <= the largest |T|.
__device__ __forceinline__ int hist_shift(unsigned maxbits) { return kHistBits + 126 - max((int)(maxbits >> 23), 1); }

// hist[level][n2] += v in the level's quanta (exact in the first level; in the
// second rounded to the nearest integer, ties away from zero), with integer
// operations only.
__device__ __forceinline__ void hist_add(unsigned long long* __restrict__ hist, int nh, int n2, float v, int shift) {
  const int b = __float_as_int(v);
  const int e = (b >> 23) & 0xFF;
  const long long m = e ? (b & 0x7FFFFF) | 0x800000 : b & 0x7FFFFF;  // v = m 2^(max(e, 1) - 150)
  int up = max(e, 1) + shift - 150;
  if (up < 0) {
    up += kFineBits;
    hist += nh;
  }
  const long long q = up >= 0 ? m << up : (up <= -25 ? 0 : ((m + (1LL << (-up - 1))) >> -up));
  if (q) atomicAdd(hist + n2, (unsigned long long)(b < 0 ? -q : q));
}

// hist[p][level][n2] += P(a) P(b) P(c) T over the images (a, b, c) of every mode with
// x >= y >= z, T the sum over the places that z can take among the three (each
// once, their rounding errors kept); one warp per column (x, y), lanes along z.
// J = 9: 0.13 ms a pair (0.12 with one level), 0.33 folded over x and y alone.
template <int NP>
__global__ void __launch_bounds__(kHistThreads)
pp_hist_kernel(const float* __restrict__ T, int L, const double* __restrict__ pd, const unsigned* __restrict__ maxbits,
               unsigned long long* __restrict__ hist, int nh) {
  extern __shared__ float P[];
  for (int i = threadIdx.x; i <= L; i += kHistThreads) P[i] = (float)pd[i];
  __syncthreads();
  const int H = L / 2 + 1, ncol = (int)fold_columns(L);
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * (kHistThreads / 32);
  int shift[NP];
  bool finite[NP];  // a pair that is not finite is left out: its bins report NaN
  float unit[NP];   // 1/4 where three T could overflow
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const unsigned mb = maxbits[p];
    finite[p] = mb < 0x7F800000u;
    shift[p] = hist_shift(mb) + (mb >= 0x7E000000u ? 2 : 0);
    unit[p] = mb >= 0x7E000000u ? 0.25f : 1.f;
  }
  for (int c = blockIdx.x * (kHistThreads / 32) + (threadIdx.x >> 5); c < ncol; c += nw) {
    int x, y;
    fold_xy(c, x, y);
    float w[4];
    int s[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int pa = (i & 1) ? L - x : x, pb = (i & 2) ? L - y : y;
      w[i] = P[pa] * P[pb];
      s[i] = pa * pa + pb * pb;
    }
    const int cx = x * (x + 1) / 2, cy = y * (y + 1) / 2;
    for (int z = lane; z <= y; z += 32) {
      const int z2 = z * z, m2 = (L - z) * (L - z);
      const float p1 = P[z], p2 = P[L - z];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        if (!finite[p]) continue;
        const float* Tp = T + (size_t)p * ncol * H;
        float t, e1, e2;
        two_sum(unit[p] * Tp[(size_t)c * H + z], y != z ? unit[p] * Tp[(size_t)(cx + z) * H + y] : 0.f, t, e1);
        two_sum(t, x != y ? unit[p] * Tp[(size_t)(cy + z) * H + x] : 0.f, t, e2);
        t += e1 + e2;
        unsigned long long* h = hist + (size_t)p * kLevels * nh;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          hist_add(h, nh, s[i] + z2, w[i] * p1 * t, shift[p]);
          hist_add(h, nh, s[i] + m2, w[i] * p2 * t, shift[p]);
        }
      }
    }
  }
}

// partial[block][bin][pair] = sum over the block's n2 of W_bin(n2) hist(n2)
// (window values in float32, products and sums in float64).
template <int NP>
__global__ void __launch_bounds__(kHistThreads)
pp_radial_bins_kernel(const WinDev* __restrict__ wins, int n_bins, int L, const double* __restrict__ pd,
                      const unsigned* __restrict__ maxbits, const unsigned long long* __restrict__ hist, int nh,
                      double* __restrict__ partial, double* __restrict__ k0) {
  extern __shared__ float P[];
  __shared__ double red[kHistThreads / 32][kRadialBins * NP];
  const int b0 = blockIdx.y * kRadialBins, nb = min(kRadialBins, n_bins - b0);
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i <= L; i += kHistThreads) P[i] = (float)pd[i];
    __syncthreads();
    if (threadIdx.x < nb)
      k0[b0 + threadIdx.x] = (double)kernel_value(wins[b0 + threadIdx.x], 0, 0, 0, L, P, 1).x;
  }
  double acc[kRadialBins][NP];
#pragma unroll
  for (int b = 0; b < kRadialBins; ++b)
#pragma unroll
    for (int p = 0; p < NP; ++p) acc[b][p] = 0.0;
  const int end = min(nh, (int)(blockIdx.x + 1) * kRadialPerBlock);
  for (int n2 = blockIdx.x * kRadialPerBlock + threadIdx.x; n2 < end; n2 += kHistThreads) {
    double h[NP];
    bool any = false;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const unsigned long long* hp = hist + (size_t)p * kLevels * nh + n2;
      const long long q = (long long)hp[0], f = (long long)hp[nh];
      any = any || (q | f) != 0;
      h[p] = fma((double)f, 1.0 / (1 << kFineBits), (double)q);
    }
    if (!any) continue;
#pragma unroll
    for (int b = 0; b < kRadialBins; ++b) {
      if (b < nb) {
        bool ok;
        const double w = (double)window_radial_n2(wins[b0 + b], n2, &ok);
#pragma unroll
        for (int p = 0; p < NP; ++p) acc[b][p] = fma(w, h[p], acc[b][p]);
      }
    }
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int b = 0; b < kRadialBins; ++b)
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      double v = acc[b][p];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[wid][b * NP + p] = v;
    }
  __syncthreads();
  if (threadIdx.x < nb * NP) {
    const int b = threadIdx.x / NP, p = threadIdx.x % NP;
    double s = 0.0;
    for (int w = 0; w < kHistThreads / 32; ++w) s += red[w][b * NP + p];
    const unsigned mb = maxbits[p];
    s = mb >= 0x7F800000u ? __longlong_as_double(0x7ff8000000000000LL)
                          : ldexp(s * (double)wins[b0 + b].scale, -hist_shift(mb));
    partial[((long long)blockIdx.x * n_bins + b0 + b) * NP + p] = s;
  }
}

}  // namespace hermes
