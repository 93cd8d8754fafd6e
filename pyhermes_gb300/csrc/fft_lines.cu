// 512-point FFTs along the strided axes of complex64 fields [nf][512][512][..]
// (x, y, z; z contiguous), in place, unnormalised: full fields of 512 columns
// (the multipole fields) and half spectra of 257 columns of a real field.
//
// cuFFT's strided passes move their bytes at about half of HBM bandwidth.
// Here a CTA owns 16 adjacent z columns of one (field, other-axis) slab and
// the 512 elements of the transformed axis: every row it reads or writes is
// 128 contiguous bytes, each element is read and written once, and the
// transform runs in shared memory as three radix-8 stages
// (512 = 8 * 8 * 8; n = n1 + 64 n2, k = k2 + 8 k1 with the 64-point part
// split the same way), twiddles from a float64 table per CTA.  Column 256 of a
// half spectrum is one column wide: 16 slabs share a tile.
//
// Measured: 5.0 / 5.1 ms per y / x pass of 15 full fields (30 GB, 6.2 TB/s;
// cuFFT 7.7 ms), 0.215 ms per y pass of a half spectrum (1.08 GB, 5 TB/s; cuFFT
// 0.254 ms), 0.35 ms for the fused x pass (three passes took 1.04 ms).
//
// The last pass of a convolution's forward transform, the window and the
// first pass of its inverse are one pass (kFused): a thread's eight outputs of
// the forward transform, x[n1 + 64 n2], n2 = 0..7, are its eight inputs of
// the inverse one.
#include "fft_device.cuh"
#include "fft_lines.cuh"
#include "hermes_common.cuh"

namespace hermes {
namespace {

enum { kInverse = 0, kForward = 1, kFused = 2, kCompact = 3 };
constexpr int kLen = 512;
constexpr int kPitch = kLen + 1;  // float2 per column in shared memory (odd: conflict-free columns)

// 16-byte asynchronous global -> shared copy (L2 only) and its group fences
__device__ __forceinline__ void cp_async16_cg(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// One CTA per SM, 512 threads, persistent over tiles (field f, other-axis
// index a, z block zb of C = 16 columns).  A ring of three shared buffers
// of 16 x 513 float2 keeps the two tiles after the current one in flight
// by cp.async (the tile loads overlap the transform: with direct loads the
// pass waited on memory and reached about half of HBM bandwidth).  A tile
// lands row-major ([row][16], 128 B rows in the order of its global rows);
// stage 1 reads it into registers and, after a barrier, writes its output
// column-major (odd pitch: conflict-free columns) into the same buffer.
// Each thread runs R = 2 eight-point transforms per stage; task i = tid +
// 512 r has column c = i % 16, so a half warp covers the 16 columns of one
// row (coalesced global rows, one bank pair per lane in shared memory).
//   stage 1 (c, n1):      x[n1 + 64 n2], n2 = 0..7 -> Y[n1][k2] e^{2 pi i n1 k2 / 512}
//   stage 2 (c, k2, m1):  Y[m1 + 8 m2][k2], m2 = 0..7 -> W[k2][m1][q2] e^{2 pi i m1 q2 / 64}
//   stage 3 (c, k2, q2):  W[k2][m1][q2], m1 = 0..7 -> X[k2 + 8 q2 + 64 q1]
// The forward transform is the inverse one on exchanged parts:
// F(a) = swap(I(swap(a))), swap(re, im) = (im, re).
constexpr int kCols = 16, kThreads = 512, kR = kCols * kLen / 8 / kThreads;
constexpr int kBuf = kCols * kPitch;

__device__ __forceinline__ float2 swapped(float2 a) { return make_float2(a.y, a.x); }

// From registers x[n1 + 64 n2] (task (c, n1)) to the inputs of the last eight
// point transforms (task (c, k2 + 8 q2), which idft8 turns into
// X[k2 + 8 q2 + 64 q1]) through the tile buffer, whose other readers are past
// the barrier at entry.  The caller's next barrier frees the buffer; the last
// transforms come after it, so that they overlap the stores of other warps.
__device__ __forceinline__ void fft512_registers(float2 (&v)[kR][8], float2* buf, const float2* tw) {
  constexpr int C = kCols, T = kThreads;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int i = threadIdx.x + T * r, c = i % C, n1 = i / C;
    idft8(v[r]);
    float2* s = buf + c * kPitch + n1 * 8;
    s[0] = v[r][0];
#pragma unroll
    for (int k2 = 1; k2 < 8; ++k2) s[k2] = cmul(v[r][k2], tw[n1 * k2]);
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int i = threadIdx.x + T * r, c = i % C, rest = i / C, k2 = rest & 7, m1 = rest >> 3;
    const float2* s = buf + c * kPitch + m1 * 8 + k2;
#pragma unroll
    for (int m2 = 0; m2 < 8; ++m2) v[r][m2] = s[64 * m2];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int i = threadIdx.x + T * r, c = i % C, rest = i / C, k2 = rest & 7, m1 = rest >> 3;
    idft8(v[r]);
    float2* s = buf + c * kPitch + k2 * 64 + m1 * 8;
    s[0] = v[r][0];
#pragma unroll
    for (int q2 = 1; q2 < 8; ++q2) s[q2] = cmul(v[r][q2], tw[8 * m1 * q2]);
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int i = threadIdx.x + T * r, c = i % C, rest = i / C, k2 = rest & 7, q2 = rest >> 3;
    const float2* s = buf + c * kPitch + k2 * 64 + q2;
#pragma unroll
    for (int m1 = 0; m1 < 8; ++m1) v[r][m1] = s[8 * m1];
  }
}

// kHalf: half spectra of 257 columns with rows of kHalfPitch values, else full
// fields of 512 columns.  kCompact: the forward x pass from such rows to `out`,
// [512][512][257]; its 128-byte rows start on any 8 bytes, which the stores do
// not mind (0.236 ms; cuFFT's compact passes 0.255 ms each).
template <int kMode, bool kHalf>
__global__ void __launch_bounds__(kThreads, 1)
fft512_cols_kernel(float2* __restrict__ data, int nf, int axis, FftWindow win, float2* __restrict__ out) {
  constexpr int C = kCols, T = kThreads, R = kR;
  constexpr int kRow = kHalf ? kFft512HalfPitch : kLen;
  extern __shared__ __align__(16) float2 sm[];
  float2* tw = sm + 3 * kBuf;
  float* G = reinterpret_cast<float*>(tw + kLen);  // gaussian window factors (kFused)
  fill_twiddles<kLen>(tw, T);
  if (kMode == kFused && win.axis_factor)
    for (int j = threadIdx.x; j < kLen; j += T) G[j] = win.axis_factor[j];
  const long long L = kLen, L2 = L * kRow, L3 = L2 * L;
  const long long astride = axis == 1 ? L2 : kRow;
  const long long rstride = axis == 1 ? kRow : L2;
  // tiles of 16 columns per slab, then (kHalf) tiles of column 256 over 16 slabs
  constexpr int kFull = (kHalf ? kLen / 2 : kLen) / C;
  const long long nfull = (long long)nf * L * kFull, ntiles = nfull + (kHalf ? nf * (L / C) : 0);
  // slab index, first column and column stride of tile t of a half spectrum
  auto half_tile = [&](long long t, int& a, int& z, long long& cs) {
    const bool tail = t >= nfull;
    a = (int)(tail ? (t - nfull) * C : t / kFull);
    z = tail ? kLen / 2 : (int)(t % kFull) * C;
    cs = tail ? astride : 1;
  };
  auto tile_ptr = [&](long long t) {
    if constexpr (kHalf) {
      int a, z;
      long long cs;
      half_tile(t, a, z, cs);
      return data + a * astride + z;
    } else {
      const int zb = (int)(t % kFull);
      const long long fa = t / kFull;
      return data + (fa / L) * L3 + (fa % L) * astride + (long long)zb * C;
    }
  };
  // tile t -> buffer (row-major), 4096 16-byte pieces, 8 per 128-byte row
  auto prefetch = [&](long long t, float2* buf) {
    if (t < ntiles) {
      const float2* g = tile_ptr(t);
      if (!kHalf || t < nfull) {
#pragma unroll
        for (int q = 0; q < 4096 / T; ++q) {
          const int j = threadIdx.x + T * q, row = j >> 3, part = j & 7;
          cp_async16_cg(buf + row * C + 2 * part, g + (long long)row * rstride + 2 * part);
        }
      } else {
#pragma unroll 4
        for (int q = 0; q < 8192 / T; ++q) {
          const int j = threadIdx.x + T * q, row = j >> 4, c = j & 15;
          cp_async8(buf + row * C + c, g + row * rstride + c * astride);
        }
      }
    }
    cp_async_commit();  // an empty group past the end keeps the group count uniform
  };
  long long t = blockIdx.x;
  prefetch(t, sm);
  prefetch(t + gridDim.x, sm + kBuf);
  for (int k = 0; t < ntiles; t += gridDim.x, ++k) {
    float2* buf = sm + (k % 3) * kBuf;
    cp_async_wait_group<1>();  // this tile's group is complete (the next one may be in flight)
    __syncthreads();
    float2 v[R][8];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = threadIdx.x + T * r, c = i % C, n1 = i / C;
#pragma unroll
      for (int n2 = 0; n2 < 8; ++n2) {
        const float2 e = buf[(n1 + 64 * n2) * C + c];
        v[r][n2] = kMode == kInverse ? e : swapped(e);
      }
    }
    prefetch(t + 2LL * gridDim.x, sm + ((k + 2) % 3) * kBuf);
    fft512_registers(v, buf, tw);
    if (kMode == kFused) {
      int a, z;  // axis 0: the slab index a is y
      long long cs;
      half_tile(t, a, z, cs);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = threadIdx.x + T * r, c = i % C, k0 = i / C;  // k0 = k2 + 8 q2
        const int y = a + (cs == 1 ? 0 : c), zc = z + (cs == 1 ? c : 0);
        const int yq = min(y, kLen - y);
        idft8(v[r]);
#pragma unroll
        for (int q1 = 0; q1 < 8; ++q1) {
          const int kx = k0 + 64 * q1;
          float K;
          if (win.axis_factor) {
            K = G[kx] * G[y] * G[zc] * win.scale;
          } else {
            const int xq = min(kx, kLen - kx), hi = max(xq, yq), lo = min(xq, yq);
            K = __ldg(win.folded + (long long)(hi * (hi + 1) / 2 + lo) * (kLen / 2 + 1) + zc);
          }
          if (win.zero_k0 && kx == 0 && y == 0 && zc == 0) K = 0.f;
          const float2 e = swapped(v[r][q1]);
          v[r][q1] = make_float2(e.x * K * win.factor, e.y * K * win.factor);
        }
      }
      fft512_registers(v, buf, tw);
    }
    __syncthreads();  // buffer free: the next iteration prefetches into it
    float2* g = tile_ptr(t);
    [[maybe_unused]] const long long cs = kHalf && t >= nfull ? astride : 1;
    if constexpr (kMode == kCompact) {
      int a, z;
      long long unused;
      half_tile(t, a, z, unused);
      g = out + (long long)a * (kLen / 2 + 1) + z;
    }
    constexpr long long kOutRow = (long long)kLen * (kLen / 2 + 1);
    auto store = [&](int r, int q1) {
      const int i = threadIdx.x + T * r, c = i % C, k0 = i / C;
      if constexpr (kMode == kCompact)
        g[(k0 + 64 * q1) * kOutRow + (cs == 1 ? c : c * (kLen / 2 + 1))] = swapped(v[r][q1]);
      else g[(long long)(k0 + 64 * q1) * rstride + (kHalf ? c * cs : c)] = kMode == kForward ? swapped(v[r][q1]) : v[r][q1];
    };
    // The order of the row stores decides the x pass (rows 2 MB apart): both
    // transforms' rows of one q1 together 5.1 ms for 15 fields, one
    // transform's eight rows after the other's 6.0 ms; the fused pass is
    // 3% better the other way round.
    if (kMode == kFused) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        idft8(v[r]);
#pragma unroll
        for (int q1 = 0; q1 < 8; ++q1) store(r, q1);
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) idft8(v[r]);
#pragma unroll
      for (int q1 = 0; q1 < 8; ++q1)
#pragma unroll
        for (int r = 0; r < R; ++r) store(r, q1);
    }
  }
  cp_async_wait_group<0>();  // no copy outlives the kernel
}

// ---- z lines of a real field ------------------------------------------------------
// Two rows of 512 real values are one complex line: z = a + i b, of which
// A[k] = (Z[k] + conj Z[-k]) / 2 and B[k] = -i (Z[k] - conj Z[-k]) / 2.  64
// threads a line pair, eight points a thread in registers (line_ifft), rows read
// and written once in whole 128-byte lines.  Bound by HBM: 211 and 210 us (1.08 GB:
// 5.1 TB/s) where cuFFT's 1-D real transforms on the same rows took 305 and 308.
constexpr int kRealGroups = 4, kLinePT = kLen / 8;

struct RealLineSync {
  int id;
  __device__ __forceinline__ void operator()() const {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id + 1), "n"(kLinePT) : "memory");
  }
};

// rows [512 * 512][512] -> half spectra [512 * 512][kFft512HalfPitch] (257 values)
__global__ void __launch_bounds__(kRealGroups* kLinePT) real_to_half_kernel(const float* __restrict__ in,
                                                                            float2* __restrict__ out) {
  __shared__ float2 buf[kRealGroups][9 * kLinePT];
  __shared__ float2 tw[kLen];
  fill_twiddles<kLen>(tw, blockDim.x);
  __syncthreads();
  const int g = threadIdx.x / kLinePT, t = threadIdx.x % kLinePT;
  const RealLineSync sync{g};
  for (int p = blockIdx.x * kRealGroups + g; p < kLen * kLen / 2; p += gridDim.x * kRealGroups) {
    const float* a = in + (long long)p * 2 * kLen;
    float2 v[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) v[n] = make_float2(__ldcs(a + kLen + t + kLinePT * n), __ldcs(a + t + kLinePT * n));  // exchanged
    line_ifft<kLen>(v, buf[g], tw, t, sync);
    sync();
#pragma unroll
    for (int n = 0; n < 8; ++n) buf[g][t + kLinePT * n] = swapped(v[n]);
    sync();
    float2* o = out + (long long)p * 2 * kFft512HalfPitch;
#pragma unroll
    for (int n = 0; n < 5; ++n) {
      const int k = t + kLinePT * n;
      if (n == 4 && t != 0) break;
      const float2 z = buf[g][k], m = buf[g][(kLen - k) & (kLen - 1)];
      o[k] = make_float2(0.5f * (z.x + m.x), 0.5f * (z.y - m.y));
      o[k + kFft512HalfPitch] = make_float2(0.5f * (z.y + m.y), 0.5f * (m.x - z.x));
    }
    sync();  // buf free
  }
}

// the inverse, unnormalised; the imaginary parts at k = 0 and 256 count as zero
__global__ void __launch_bounds__(kRealGroups* kLinePT) half_to_real_kernel(const float2* __restrict__ in,
                                                                            float* __restrict__ out) {
  __shared__ float2 buf[kRealGroups][9 * kLinePT];
  __shared__ float2 tw[kLen];
  fill_twiddles<kLen>(tw, blockDim.x);
  __syncthreads();
  const int g = threadIdx.x / kLinePT, t = threadIdx.x % kLinePT;
  const RealLineSync sync{g};
  for (int p = blockIdx.x * kRealGroups + g; p < kLen * kLen / 2; p += gridDim.x * kRealGroups) {
    const float2* h = in + (long long)p * 2 * kFft512HalfPitch;
    float2 v[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int k = t + kLinePT * n;
      const bool low = n < 4 || (n == 4 && t == 0);
      const float2 a = h[low ? k : kLen - k], b = h[(low ? k : kLen - k) + kFft512HalfPitch];
      v[n] = low ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, b.x - a.y);
      if ((n == 0 || n == 4) && t == 0) v[n] = make_float2(a.x, b.x);
    }
    line_ifft<kLen>(v, buf[g], tw, t, sync);
    float* o = out + (long long)p * 2 * kLen;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      o[t + kLinePT * n] = v[n].x;
      o[kLen + t + kLinePT * n] = v[n].y;
    }
    sync();  // buf free
  }
}

// The strided pass of L = 128 and 256: tiles of 16 columns as above, one
// eight-point transform a thread (line_ifft's stages, its buffer per column
// with an odd pitch), two blocks an SM.
template <int L>
__global__ void __launch_bounds__(2 * L, 2)
fft_cols_kernel(float2* __restrict__ data, int nf, int axis) {
  constexpr int C = kCols, T = 2 * L, PT = L / 8, R = L / 64, kCol = 9 * PT + 1, kTile = C * kCol;
  extern __shared__ __align__(16) float2 sm[];
  float2* tw = sm + 3 * kTile;
  fill_twiddles<L>(tw, T);
  const int astride = axis == 1 ? L * L : L, rstride = axis == 1 ? L : L * L;
  const int ntiles = nf * L * (L / C);
  auto tile_ptr = [&](int t) {
    const int zb = t % (L / C), fa = t / (L / C);
    return data + (long long)(fa / L) * (L * L * L) + (fa % L) * astride + zb * C;
  };
  auto prefetch = [&](int t, float2* buf) {
    if (t < ntiles) {
      const float2* g = tile_ptr(t);
#pragma unroll
      for (int q = 0; q < 8 * L / T; ++q) {
        const int j = threadIdx.x + T * q, row = j >> 3, part = j & 7;
        cp_async16_cg(buf + row * C + 2 * part, g + row * rstride + 2 * part);
      }
    }
    cp_async_commit();
  };
  auto sync = [] { __syncthreads(); };
  const int c = threadIdx.x % C, n1 = threadIdx.x / C;
  int t = blockIdx.x;
  prefetch(t, sm);
  prefetch(t + gridDim.x, sm + kTile);
  for (int k = 0; t < ntiles; t += gridDim.x, ++k) {
    float2* buf = sm + (k % 3) * kTile;
    cp_async_wait_group<1>();
    __syncthreads();
    float2 v[8];
#pragma unroll
    for (int n2 = 0; n2 < 8; ++n2) v[n2] = buf[(n1 + PT * n2) * C + c];
    prefetch(t + 2 * gridDim.x, sm + ((k + 2) % 3) * kTile);
    __syncthreads();
    line_ifft<L>(v, buf + c * kCol, tw, n1, sync);
    float2* g = tile_ptr(t) + c;
#pragma unroll
    for (int i = 0; i < 8 / R; ++i)
#pragma unroll
      for (int q = 0; q < R; ++q) g[(n1 + PT * i + 64 * q) * rstride] = v[R * i + q];
    __syncthreads();  // buffer free: the next iteration prefetches into it
  }
  cp_async_wait_group<0>();
}

template <int L>
int launch_fft_cols(float2* data, int nf, int axis, cudaStream_t s) {
  constexpr size_t smem = sizeof(float2) * (3 * (size_t)kCols * (9 * L / 8 + 1) + L);
  static bool attr_set[64] = {false};
  int dev = 0;
  HERMES_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {  // once per device, before any stream capture
    HERMES_CUDA_TRY(cudaFuncSetAttribute(fft_cols_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  int nsm = 0;
  HERMES_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int ntiles = nf * L * (L / kCols), per_sm = L == 128 ? 4 : 2;
  fft_cols_kernel<L><<<ntiles < nsm * per_sm ? ntiles : nsm * per_sm, 2 * L, smem, s>>>(data, nf, axis);
  HERMES_LAUNCH_CHECK("fft_cols_kernel");
  return HERMES_OK;
}

template <int kMode, bool kHalf>
int launch_cols(float2* data, int nf, int axis, const FftWindow& win, cudaStream_t s, float2* out = nullptr) {
  constexpr size_t smem = sizeof(float2) * (3 * (size_t)kBuf + kLen) + (kMode == kFused ? sizeof(float) * kLen : 0);
  static bool attr_set[64] = {false};
  int dev = 0;
  HERMES_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {  // once per device, before any stream capture
    HERMES_CUDA_TRY(cudaFuncSetAttribute(fft512_cols_kernel<kMode, kHalf>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem));
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  int nsm = 0;
  HERMES_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  // one block per SM: every shape has more tiles (8224 at least) than SMs
  fft512_cols_kernel<kMode, kHalf><<<nsm, kThreads, smem, s>>>(data, nf, axis, win, out);
  HERMES_LAUNCH_CHECK("fft512_cols_kernel");
  return HERMES_OK;
}

}  // namespace

// axis 0: x, axis 1: y.
int fft512_strided_inverse(float2* data, int nf, int axis, cudaStream_t s) {
  return launch_cols<kInverse, false>(data, nf, axis, FftWindow{}, s);
}

int fft_strided_inverse(float2* data, int J, int nf, int axis, cudaStream_t s) {
  if (J == 9) return fft512_strided_inverse(data, nf, axis, s);
  if (J == 8) return launch_fft_cols<256>(data, nf, axis, s);
  if (J == 7) return launch_fft_cols<128>(data, nf, axis, s);
  return fail(HERMES_ERR_UNSUPPORTED, "fft_strided_inverse: J=%d", J);
}

static int real_grid(int* blocks) {
  int dev = 0, nsm = 0;
  HERMES_CUDA_TRY(cudaGetDevice(&dev));
  HERMES_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  *blocks = nsm * 8;
  return HERMES_OK;
}

int fft512_real_to_half(const float* in, float2* out, cudaStream_t s) {
  int blocks = 0, rc = real_grid(&blocks);
  if (rc) return rc;
  real_to_half_kernel<<<blocks, kRealGroups * kLinePT, 0, s>>>(in, out);
  HERMES_LAUNCH_CHECK("real_to_half_kernel");
  return HERMES_OK;
}

int fft512_half_to_real(const float2* in, float* out, cudaStream_t s) {
  int blocks = 0, rc = real_grid(&blocks);
  if (rc) return rc;
  half_to_real_kernel<<<blocks, kRealGroups * kLinePT, 0, s>>>(in, out);
  HERMES_LAUNCH_CHECK("half_to_real_kernel");
  return HERMES_OK;
}

int fft512_half_y(float2* data, bool forward, cudaStream_t s) {
  return forward ? launch_cols<kForward, true>(data, 1, 1, FftWindow{}, s)
                 : launch_cols<kInverse, true>(data, 1, 1, FftWindow{}, s);
}

int fft512_half_x_compact(float2* data, float2* out, cudaStream_t s) {
  return launch_cols<kCompact, true>(data, 1, 0, FftWindow{}, s, out);
}

int fft512_half_x_window_x(float2* data, const FftWindow& win, cudaStream_t s) {
  return launch_cols<kFused, true>(data, 1, 0, win, s);
}

}  // namespace hermes

extern "C" int hermes_fft512_strided_inverse(void* data, int nfields, int axis, void* stream) {
  if (!data) return hermes::fail(HERMES_ERR_INVALID, "fft512_strided_inverse: data is NULL");
  if (nfields < 1 || nfields > 64)
    return hermes::fail(HERMES_ERR_INVALID, "fft512_strided_inverse: nfields=%d outside [1, 64]", nfields);
  if (axis != 0 && axis != 1)
    return hermes::fail(HERMES_ERR_INVALID, "fft512_strided_inverse: axis=%d must be 0 (x) or 1 (y)", axis);
  return hermes::fft512_strided_inverse(static_cast<float2*>(data), nfields, axis, hermes::as_stream(stream));
}
