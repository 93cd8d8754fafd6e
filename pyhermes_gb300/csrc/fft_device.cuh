// Device pieces of the hand-written inverse FFTs: 8-, 4- and 2-point
// transforms, twiddle tables, and one contiguous line of L = 8 * 8 * R points
// (R = 2, 4, 8) held eight points a thread.
#pragma once

#include "hermes_common.cuh"

namespace hermes {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// a[k] <- sum_n a[n] e^{+2 pi i n k / 8}: two 4-point transforms of the
// even and odd inputs, combined with e^{+i pi k / 4}.
__device__ __forceinline__ void idft8(float2 (&a)[8]) {
  constexpr float r = 0.70710678118654752f;  // 1/sqrt(2)
  const float2 b0 = make_float2(a[0].x + a[4].x, a[0].y + a[4].y), b1 = make_float2(a[0].x - a[4].x, a[0].y - a[4].y);
  const float2 b2 = make_float2(a[2].x + a[6].x, a[2].y + a[6].y), b3 = make_float2(a[2].x - a[6].x, a[2].y - a[6].y);
  const float2 b4 = make_float2(a[1].x + a[5].x, a[1].y + a[5].y), b5 = make_float2(a[1].x - a[5].x, a[1].y - a[5].y);
  const float2 b6 = make_float2(a[3].x + a[7].x, a[3].y + a[7].y), b7 = make_float2(a[3].x - a[7].x, a[3].y - a[7].y);
  // even part E[k] and odd part O[k], k = 0..3 (i b = (-b.y, b.x))
  const float2 e0 = make_float2(b0.x + b2.x, b0.y + b2.y), e2 = make_float2(b0.x - b2.x, b0.y - b2.y);
  const float2 e1 = make_float2(b1.x - b3.y, b1.y + b3.x), e3 = make_float2(b1.x + b3.y, b1.y - b3.x);
  const float2 o0 = make_float2(b4.x + b6.x, b4.y + b6.y), o2 = make_float2(b4.x - b6.x, b4.y - b6.y);
  const float2 o1 = make_float2(b5.x - b7.y, b5.y + b7.x), o3 = make_float2(b5.x + b7.y, b5.y - b7.x);
  // w^k O[k], w = e^{+i pi / 4}
  const float2 t1 = make_float2((o1.x - o1.y) * r, (o1.x + o1.y) * r);
  const float2 t2 = make_float2(-o2.y, o2.x);
  const float2 t3 = make_float2(-(o3.x + o3.y) * r, (o3.x - o3.y) * r);
  a[0] = make_float2(e0.x + o0.x, e0.y + o0.y);
  a[4] = make_float2(e0.x - o0.x, e0.y - o0.y);
  a[1] = make_float2(e1.x + t1.x, e1.y + t1.y);
  a[5] = make_float2(e1.x - t1.x, e1.y - t1.y);
  a[2] = make_float2(e2.x + t2.x, e2.y + t2.y);
  a[6] = make_float2(e2.x - t2.x, e2.y - t2.y);
  a[3] = make_float2(e3.x + t3.x, e3.y + t3.y);
  a[7] = make_float2(e3.x - t3.x, e3.y - t3.y);
}

// The same for 4 and 2 points.
__device__ __forceinline__ void idft4(float2 (&a)[4]) {
  const float2 b0 = make_float2(a[0].x + a[2].x, a[0].y + a[2].y), b1 = make_float2(a[0].x - a[2].x, a[0].y - a[2].y);
  const float2 b2 = make_float2(a[1].x + a[3].x, a[1].y + a[3].y), b3 = make_float2(a[1].x - a[3].x, a[1].y - a[3].y);
  a[0] = make_float2(b0.x + b2.x, b0.y + b2.y);
  a[2] = make_float2(b0.x - b2.x, b0.y - b2.y);
  a[1] = make_float2(b1.x - b3.y, b1.y + b3.x);
  a[3] = make_float2(b1.x + b3.y, b1.y - b3.x);
}
__device__ __forceinline__ void idft2(float2 (&a)[2]) {
  const float2 t = a[0];
  a[0] = make_float2(t.x + a[1].x, t.y + a[1].y);
  a[1] = make_float2(t.x - a[1].x, t.y - a[1].y);
}

// tw[j] = e^{2 pi i j / L}, j < L, by `threads` threads: the first octant in
// float64 (slow on this part: 512 evaluations cost as much as two tiles of the
// strided pass), the others are its reflections.  The caller synchronises.
template <int L>
__device__ __forceinline__ void fill_twiddles(float2* tw, int threads) {
  for (int j = threadIdx.x; j <= L / 8; j += threads) {
    double sd, cd;
    sincospi((double)j / (L / 2), &sd, &cd);
    const float sn = (float)sd, cs = (float)cd;
    constexpr int q = L / 4;  // a quarter turn
    tw[j] = make_float2(cs, sn);
    tw[q - j] = make_float2(sn, cs);
    tw[q + j] = make_float2(-sn, cs);
    tw[2 * q - j] = make_float2(-cs, sn);
    tw[2 * q + j] = make_float2(-cs, -sn);
    tw[3 * q - j] = make_float2(-sn, -cs);
    tw[3 * q + j] = make_float2(sn, -cs);
    if (j > 0) tw[4 * q - j] = make_float2(cs, -sn);
  }
}

// One line of L points by P = L / 8 threads (t = 0 .. P - 1; whole warps or, for
// L = 128, halves of one), unnormalised inverse transform:
//   in   v[n2] = x[t + P n2]
//   out  v[R i + q1] = X[j + 64 q1], j = t + P i, i < 8 / R, q1 < R
// with n = n1 + P n2, k = k2 + 8 q2 + 64 q1.  buf: 9 P float2 of the line's own
// (rows of 8 padded to 9: the strided reads and writes do not conflict).
// `sync` synchronises the line's threads; buf may be written again after one
// more of it.
template <int L, class Sync>
__device__ __forceinline__ void line_ifft(float2 (&v)[8], float2* buf, const float2* tw, int t, Sync sync) {
  constexpr int P = L / 8, R = L / 64;
  idft8(v);
  buf[9 * t] = v[0];
#pragma unroll
  for (int k2 = 1; k2 < 8; ++k2) buf[9 * t + k2] = cmul(v[k2], tw[t * k2]);
  sync();
  const int k2 = t & 7, m1 = t >> 3;  // R-strided inputs m1 + R m2 of the P-point transform k2
#pragma unroll
  for (int m2 = 0; m2 < 8; ++m2) v[m2] = buf[9 * (m1 + R * m2) + k2];
  sync();
  idft8(v);
  buf[9 * t] = v[0];
#pragma unroll
  for (int q2 = 1; q2 < 8; ++q2) buf[9 * t + q2] = cmul(v[q2], tw[8 * m1 * q2]);
  sync();
#pragma unroll
  for (int i = 0; i < 8 / R; ++i) {
    const int j = t + P * i, kk = j & 7, q2 = j >> 3;
    float2 a[R];
#pragma unroll
    for (int m = 0; m < R; ++m) a[m] = buf[9 * (8 * m + kk) + q2];
    if constexpr (R == 8)
      idft8(a);
    else if constexpr (R == 4)
      idft4(a);
    else
      idft2(a);
#pragma unroll
    for (int m = 0; m < R; ++m) v[R * i + m] = a[m];
  }
}

}  // namespace hermes
