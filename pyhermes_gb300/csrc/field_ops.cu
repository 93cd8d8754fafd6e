// Passes over one float32 field that a task makes beside its kernels: the
// float64 sum of the coefficients (the k = 0 mode, the field integral) and
// the field minus a mean density.  Both are bound by HBM.  Written with
// float64 arithmetic they are bound by the float64 pipe (two lanes per SM
// and clock): a cast-and-sum takes 0.77 ms and a cast, subtract and cast back
// 1.3 ms for 512^3 cells.  Here the additions are float32 ones that keep their
// rounding errors (Knuth's two-sum), and float64 enters once per 64 values: the
// sum takes 0.091 ms (5.9 TB/s), 0.094 and 0.118 ms with float64 once per 32 and
// 16; the shift, with the bits of float64, 0.170 ms (6.3 TB/s).
#include <cmath>

#include "hermes_common.cuh"

namespace {

using hermes::fail;
using hermes::two_sum;

constexpr int kThreads = 256;
constexpr int kMaxBlocks = 2048;

// float64 sum of a block (fixed order).
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double sh[kThreads / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < kThreads / 32; ++i) s += sh[i];
  return s;
}

// s + c + d += x: s the float32 sum, c the sum of its rounding errors, d the sum of
// c's.  Up to 64 values then enter float64 with more digits than it has.  An
// infinity or a NaN in s makes d a NaN.
__device__ __forceinline__ void add3(float x, float& s, float& c, float& d) {
  float e;
  two_sum(s, x, s, e);
  two_sum(c, e, c, e);
  d += e;
}

// partial[block] = sum of x over the block's grid-stride share; kVec: x is
// 16-byte aligned and read as float4 (the n % 4 last values by block 0).
template <bool kVec>
__global__ void __launch_bounds__(kThreads) field_sum_kernel(const float* __restrict__ x, int64_t n,
                                                             double* __restrict__ partial) {
  double acc = 0.0;
  const int64_t t0 = (int64_t)blockIdx.x * kThreads + threadIdx.x, stride = (int64_t)gridDim.x * kThreads;
  if (kVec) {
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const int64_t n4 = n >> 2;
    for (int64_t i = t0; i < n4;) {
      const int64_t first = i;
      float s = 0.f, c = 0.f, d = 0.f;
      auto add = [&](const float4& v) {
        add3(v.x, s, c, d);
        add3(v.y, s, c, d);
        add3(v.z, s, c, d);
        add3(v.w, s, c, d);
      };
      for (int g = 0; g < 4 && i + 3 * stride < n4; ++g, i += 4 * stride) {
        float4 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = __ldcs(x4 + i + k * stride);
#pragma unroll
        for (int k = 0; k < 4; ++k) add(v[k]);
      }
      if (i == first)  // the last one to three
        for (; i < n4; i += stride) add(x4[i]);
      if (isfinite(d)) {
        acc += (double)s + ((double)c + (double)d);
      } else {  // an infinity, a NaN or a float32 overflow of s: as float64 gives it
        for (int64_t j = first; j < i; j += stride) {
          const float4 v = x4[j];
          acc += ((double)v.x + (double)v.y) + ((double)v.z + (double)v.w);
        }
      }
    }
    if (blockIdx.x == 0 && threadIdx.x < (n & 3)) acc += (double)x[(n4 << 2) + threadIdx.x];
  } else {
    for (int64_t i = t0; i < n; i += stride) acc += (double)x[i];
  }
  const double s = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

__global__ void __launch_bounds__(kThreads) field_sum_final_kernel(const double* __restrict__ partial, int n,
                                                                   double* __restrict__ out) {
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += kThreads) acc += partial[i];
  const double s = block_sum(acc);
  if (threadIdx.x == 0) *out = s;
}

struct Shift {
  double r;
  float hi, lo, rest;  // r = hi + lo + what |rest| bounds
};

// A call, so that the conversions (0.73 ms for 512^3 cells where the compiler makes
// them for every value) are made only where they decide.
__device__ __noinline__ float shifted_f64(float v, double r) { return __double2float_rn((double)v - r); }

// (float)((double)v - r), the same bits.  v - r = out + low + te + what r has
// beyond hi + lo, and the float64 difference is 2^-53 of it off: out is that float
// unless low comes within these of half a unit in the last place of out (a
// quarter below a power of two), or where out + low is exactly the difference
// and half a unit is a tie, which the addition has rounded to even.  Else, a few
// values in 10^6 or v beside r, and where anything is not finite, float64 decides
// (0.169 ms without the test, which hides behind the reads).
__device__ __forceinline__ float shifted(float v, const Shift& sh) {
  float s, e, t, te, out, low;
  two_sum(v, -sh.hi, s, e);
  two_sum(e, -sh.lo, t, te);
  two_sum(s, t, out, low);
  const int b = __float_as_int(out);
  const float half = __int_as_float(b & 0x7F800000) * ((b & 0x7FFFFF) ? 0x1p-24f : 0x1p-25f);
  const float beyond = fabsf(te) + sh.rest, err = 1.0001f * fmaf(0x1p-51f, fabsf(out), beyond);
  if (fabsf(low) + err < half || (beyond == 0.f && fabsf(low) == half && half > 0.f)) return out;
  return shifted_f64(v, sh.r);
}

template <bool kVec>
__global__ void __launch_bounds__(kThreads) field_shift_kernel(const float* __restrict__ x, int64_t n, Shift sh,
                                                               float* __restrict__ out) {
  const int64_t t0 = (int64_t)blockIdx.x * kThreads + threadIdx.x, stride = (int64_t)gridDim.x * kThreads;
  if (kVec) {
    const int64_t n4 = n >> 2;
    for (int64_t i = t0; i < n4; i += stride) {
      const float4 v = reinterpret_cast<const float4*>(x)[i];
      reinterpret_cast<float4*>(out)[i] =
          make_float4(shifted(v.x, sh), shifted(v.y, sh), shifted(v.z, sh), shifted(v.w, sh));
    }
    if (blockIdx.x == 0 && threadIdx.x < (n & 3)) out[(n4 << 2) + threadIdx.x] = shifted(x[(n4 << 2) + threadIdx.x], sh);
  } else {
    for (int64_t i = t0; i < n; i += stride) out[i] = shifted(x[i], sh);
  }
}

int blocks_for(int64_t n) {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int64_t want = (n + 4 * kThreads - 1) / (4 * kThreads), cap = (int64_t)nsm * 8 < kMaxBlocks ? nsm * 8 : kMaxBlocks;
  return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

extern "C" int hermes_field_sum(const float* x, int64_t n, double* dev_out, void* workspace, size_t workspace_bytes,
                                void* stream) {
  if (n < 0 || (n > 0 && !x) || !dev_out) return fail(HERMES_ERR_INVALID, "field_sum: bad argument");
  if (!workspace || workspace_bytes < sizeof(double) * kMaxBlocks)
    return fail(HERMES_ERR_WORKSPACE, "field_sum: workspace %zu < %zu", workspace_bytes, sizeof(double) * kMaxBlocks);
  cudaStream_t s = hermes::as_stream(stream);
  double* partial = static_cast<double*>(workspace);
  const int nblk = blocks_for(n);
  if (aligned16(x))
    field_sum_kernel<true><<<nblk, kThreads, 0, s>>>(x, n, partial);
  else
    field_sum_kernel<false><<<nblk, kThreads, 0, s>>>(x, n, partial);
  HERMES_LAUNCH_CHECK("field_sum_kernel");
  field_sum_final_kernel<<<1, kThreads, 0, s>>>(partial, nblk, dev_out);
  HERMES_LAUNCH_CHECK("field_sum_final_kernel");
  return HERMES_OK;
}

extern "C" int hermes_field_shift(const float* x, int64_t n, double r, float* out, void* stream) {
  if (n < 0 || (n > 0 && (!x || !out))) return fail(HERMES_ERR_INVALID, "field_shift: bad argument");
  if (n == 0) return HERMES_OK;
  cudaStream_t s = hermes::as_stream(stream);
  Shift sh;
  sh.r = r;
  sh.hi = (float)r;
  const double below = r - (double)sh.hi;
  sh.lo = (float)below;
  const double rest = std::fabs(below - (double)sh.lo);
  sh.rest = rest == 0.0 ? 0.f : std::nextafter((float)(1.001 * rest), INFINITY);  // not 0 by underflow
  const int nblk = blocks_for(n);
  if (aligned16(x) && aligned16(out))
    field_shift_kernel<true><<<nblk, kThreads, 0, s>>>(x, n, sh, out);
  else
    field_shift_kernel<false><<<nblk, kThreads, 0, s>>>(x, n, sh, out);
  HERMES_LAUNCH_CHECK("field_shift_kernel");
  return HERMES_OK;
}
