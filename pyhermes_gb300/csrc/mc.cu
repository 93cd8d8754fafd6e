// Monte Carlo 3PCF on the GPU: field interpolation at points and triplet
// products over (centre, rotation) pairs.
//
// Restates pyhermes/utils/wavelet_grid.py:143-186 (interpolate_grid_at_pos:
// the 27-point phi-weighted gather) and pyhermes/utils/corr3pcf_kernels.py:
// 66-140 (estimate_triplet_product_{particle,box_random}_centers).  The
// reference draws three uniforms per rotation from a re-seeded MT19937 and
// builds the two triangle offsets on the host (generate_triangle_offsets,
// :21-63); the offsets are tiny (n_rot x 6 doubles) and are passed in, so the
// GPU sums exactly the same (centre, offset) pairs.  One thread per centre
// loads the centre once, gathers n1 once and loops over the rotations;
// products are float32, sums float64 with a fixed-order block reduction.
#include <algorithm>

#include "hermes_common.cuh"

namespace {

using hermes::fail;

// Cell and fraction index of a scaled coordinate exactly as the reference:
// c = floor(s), f = int((s - c) * res) in float64.
__device__ __forceinline__ void mc_axis(double s, int res, int L, int& c, int& f) {
  const double fl = floor(s);
  c = ((int)fl) & (L - 1);
  int fi = (int)__dmul_rn(__dsub_rn(s, fl), (double)res);
  f = fi < 0 ? 0 : (fi >= res ? res - 1 : fi);
}

// Index of cell (x, y, z) of an L^3 field: C order (z fastest), or the brick
// layout of hermes_field_to_bricks: 2 x 2 x 2 bricks of 32 bytes (one DRAM
// sector) in C order of the brick coordinates, the 8 cells of a brick in
// (x, y, z) bit order.  A 3 x 3 x 3 stencil then touches exactly 8 sectors,
// against 9 rows of 1-2 sectors each in C order.
template <bool kBricks>
__device__ __forceinline__ size_t mc_cell(int x, int y, int z, int J) {
  if (!kBricks) return (((size_t)x << J) + y) << J | (size_t)z;
  const int h = J - 1;
  const size_t brick = ((((size_t)(x >> 1) << h) + (y >> 1)) << h) + (z >> 1);
  return brick << 3 | (size_t)((x & 1) << 2 | (y & 1) << 1 | (z & 1));
}

// phi samples of a block, one 16-byte read per axis (the table in global memory
// costs one 128-byte line per lane and read).
struct __align__(16) McPhi {
  float4 p[1024];  // phi at fraction f + 0, 1, 2 units
};

// The same from the table in global memory: one interpolation a thread does
// not pay for filling the block's copy (1e6 positions at J = 8: 68 us, 77 us with it).
struct McPhiGlobal {
  const float* phis;
  int res;
};

__device__ __forceinline__ float4 mc_weights(const McPhi* sp, int f) { return sp->p[f]; }
__device__ __forceinline__ float4 mc_weights(const McPhiGlobal* g, int f) {
  return make_float4(__ldg(g->phis + f), __ldg(g->phis + f + g->res), __ldg(g->phis + f + 2 * g->res), 0.f);
}

__device__ __forceinline__ void mc_load_phi(McPhi* sp, const float* __restrict__ phis, int res) {
  for (int i = threadIdx.x; i < res; i += blockDim.x) sp->p[i] = make_float4(phis[i], phis[i + res], phis[i + 2 * res], 0.f);
  __syncthreads();
}

// mc_axis for a power-of-two res = 2^rl and 0 <= s < 2^30, from the bits of s
// (the integer part and the next rl bits of the mantissa are exactly floor(s)
// and int((s - floor(s)) res)): float64 floor, subtract, multiply and
// conversions take 16 cycles of the SM per warp each.
__device__ __forceinline__ void mc_axis_bits(double s, int res, int rl, int L, int& c, int& f) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(s);
  const int ex = (int)(b >> 52);  // the sign bit makes it too large
  if (rl < 0 || ex >= 1023 + 30 || ex == 0) {
    mc_axis(s, res, L, c, f);
    return;
  }
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const int sh = 1075 - ex, t = sh - rl;  // s = m 2^-sh, sh >= 23
  c = sh >= 64 ? 0 : (int)(m >> sh) & (L - 1);
  f = t >= 64 ? 0 : (int)(m >> t) & (res - 1);
}

// One axis of the stencil: phi at fraction f + 0, 1, 2 units weights the cells
// c, c - 1, c - 2 (v2, v1, v0).  Every gather reduces z, then y, then x with
// this sum, so all layouts give the same bits.
__device__ __forceinline__ float mc_axis_sum(float v0, float v1, float v2, float p0, float p1, float p2) {
  return fmaf(p0, v2, fmaf(p1, v1, p2 * v0));
}

// The cells cz - 2, cz - 1, cz of a C-order row that starts on 16 bytes, from
// the one or two aligned quads that hold them (also across the wrap).
__device__ __forceinline__ void mc_row_quads(const float* __restrict__ row, int cz, int m, float (&v)[3]) {
  const int z = (cz - 2) & m, o = z & 3;
  const float4 a = __ldg(reinterpret_cast<const float4*>(row) + (z >> 2));
  float4 b = a;
  if (o > 1) b = __ldg(reinterpret_cast<const float4*>(row) + (cz >> 2));
  v[0] = o == 0 ? a.x : (o == 1 ? a.y : (o == 2 ? a.z : a.w));
  v[1] = o == 0 ? a.y : (o == 1 ? a.z : (o == 2 ? a.w : b.x));
  v[2] = o == 0 ? a.z : (o == 1 ? a.w : (o == 2 ? b.x : b.y));
}

// 27-point interpolation of a float32 field at scaled position (sx, sy, sz),
// row by row (kQuads: C order, 16-byte aligned) or cell by cell.
template <bool kBricks, bool kQuads, class Phi>
__device__ __forceinline__ float mc_interp(const float* __restrict__ grid, const Phi* sp, int res, int rl, int J,
                                           double sx, double sy, double sz) {
  const int L = 1 << J, m = L - 1;
  int cx, cy, cz, fx, fy, fz;
  mc_axis_bits(sx, res, rl, L, cx, fx);
  mc_axis_bits(sy, res, rl, L, cy, fy);
  mc_axis_bits(sz, res, rl, L, cz, fz);
  const float4 wx = mc_weights(sp, fx), wy = mc_weights(sp, fy), wz = mc_weights(sp, fz);
  float rx[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float ry[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      float v[3];
      if (kQuads) {
        mc_row_quads(grid + mc_cell<false>((cx - 2 + a) & m, (cy - 2 + b) & m, 0, J), cz, m, v);
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c)
          v[c] = __ldg(grid + mc_cell<kBricks>((cx - 2 + a) & m, (cy - 2 + b) & m, (cz - 2 + c) & m, J));
      }
      ry[b] = mc_axis_sum(v[0], v[1], v[2], wz.x, wz.y, wz.z);
    }
    rx[a] = mc_axis_sum(ry[0], ry[1], ry[2], wy.x, wy.y, wy.z);
  }
  return mc_axis_sum(rx[0], rx[1], rx[2], wx.x, wx.y, wx.z);
}

// ---- brick-layout gather --------------------------------------------------------
// A 3 x 3 x 3 stencil lies in exactly 8 bricks.  mc_interp above reads its 27
// cells one by one: 27 loads per lane, each of a warp's 32 addresses in another
// 128-byte line, which is what bounds it (about one line per SM and clock).
// Here a lane reads each brick with one 32-byte load and reduces z, y, x in
// turn.  Of the four cells per axis of the two bricks the stencil's three are
// picked by selects (a cell outside the stencil never enters a product).
// 2e5 centres x 100 rotations at J = 9: 2.75 ms (3.03 ms cell by cell), and
// 1.31 ms with the rotations of a centre side by side (mc_triplet_kernel).
__device__ __forceinline__ void mc_brick(const float* __restrict__ p, float (&v)[8]) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
      : "l"(p));
}

// the three of a0 .. a3 that start at a1 (odd) or a0
__device__ __forceinline__ float mc_reduce3(float a0, float a1, float a2, float a3, bool odd, float4 w) {
  return mc_axis_sum(odd ? a1 : a0, odd ? a2 : a1, odd ? a3 : a2, w.x, w.y, w.z);
}

__device__ __forceinline__ float mc_interp_bricks(const float* __restrict__ bricks, const McPhi* sp, int res, int rl, int J,
                                                  double sx, double sy, double sz) {
  const int L = 1 << J, h = J - 1, hm = (1 << h) - 1;
  int cx, cy, cz, fx, fy, fz;
  mc_axis_bits(sx, res, rl, L, cx, fx);
  mc_axis_bits(sy, res, rl, L, cy, fy);
  mc_axis_bits(sz, res, rl, L, cz, fz);
  const float4 wx = sp->p[fx], wy = sp->p[fy], wz = sp->p[fz];
  const bool ox = cx & 1, oy = cy & 1, oz = cz & 1;
  // brick coordinates: the lower one, then the one that holds the cell
  const int bx[2] = {((cx >> 1) - 1) & hm, cx >> 1}, by[2] = {((cy >> 1) - 1) & hm, cy >> 1};
  const int z0 = ((cz >> 1) - 1) & hm, z1 = cz >> 1;
  float rx[4];  // the four cells along x, reduced over y and z
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float ry[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const size_t row = (((size_t)bx[i] << h) + by[j]) << h;
      float lo[8], hi[8];
      mc_brick(bricks + ((row + z0) << 3), lo);
      mc_brick(bricks + ((row + z1) << 3), hi);
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const int k = 4 * x + 2 * y;
          ry[x][2 * j + y] = mc_reduce3(lo[k], lo[k + 1], hi[k], hi[k + 1], oz, wz);
        }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) rx[2 * i + x] = mc_reduce3(ry[x][0], ry[x][1], ry[x][2], ry[x][3], oy, wy);
  }
  return mc_reduce3(rx[0], rx[1], rx[2], rx[3], ox, wx);
}

// Interpolation in the layout of the kernel's fields: C order by quads or (a
// field that is not 16-byte aligned) by cells, bricks by whole bricks or (not
// 32-byte aligned) by cells.
enum { kCOrder = 0, kCells = 1, kBrickCells = 2, kBricks = 3 };
template <int kLayout>
__device__ __forceinline__ float mc_value(const float* __restrict__ grid, const McPhi* sp, int res, int rl, int J,
                                          double sx, double sy, double sz) {
  if constexpr (kLayout == kBricks)
    return mc_interp_bricks(grid, sp, res, rl, J, sx, sy, sz);
  else
    return mc_interp<kLayout == kBrickCells, kLayout == kCOrder>(grid, sp, res, rl, J, sx, sy, sz);
}

// Morton key (30 bits) of the cell of every centre (grid units).
__global__ void mc_morton_kernel(const double* __restrict__ centers, int64_t n, int L, int* __restrict__ keys) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    unsigned key = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      unsigned v = (unsigned)(long long)floor(centers[3 * i + a]) & (unsigned)(L - 1);  // 10 bits
      v = (v | (v << 16)) & 0x030000FFu;
      v = (v | (v << 8)) & 0x0300F00Fu;
      v = (v | (v << 4)) & 0x030C30C3u;
      v = (v | (v << 2)) & 0x09249249u;
      key |= v << a;
    }
    keys[i] = (int)key;
  }
}

__global__ void mc_phi_kernel(const double* __restrict__ phi, int n, float* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = (float)phi[i];
}

template <int kLayout>
__global__ void __launch_bounds__(256) mc_interp_kernel(const float* __restrict__ grid, int J, const double* __restrict__ pos, int64_t n,
                                 const float* __restrict__ phis, int res, int rl, double dx, double dy, double dz,
                                 double* __restrict__ out) {
  const McPhiGlobal g = {phis, res};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (double)mc_interp<false, kLayout == kCOrder>(grid, &g, res, rl, J, pos[3 * i] + dx, pos[3 * i + 1] + dy, pos[3 * i + 2] + dz);
}

// sum_i w_i n1_i sum_r n2(x_i + d2_r) n3(x_i + d3_r); n1 = eps1 interpolated
// (box-random centres) or rho1 (particle centres: eps1 == NULL).  When
// samples != NULL also writes the per-(centre, rotation) products f_ir.  A centre's rotations
// are shared by n_part threads (part p takes r = p, p + n_part, ...).  A warp
// holds 32 neighbouring centres of one part, and the parts of those centres
// are neighbouring warps: the threads in flight then cover a small part of the
// box (1/8 of it for 2e5 centres in 12 parts), whose bricks L2 holds, and not
// all centres with a few rotations each, whose bricks it does not.
template <int kLayout>
__global__ void __launch_bounds__(256)
mc_triplet_kernel(const float* __restrict__ eps1, const float* __restrict__ eps2, const float* __restrict__ eps3,
                  int J, const double* __restrict__ centers, const double* __restrict__ cw, int64_t nc,
                  const double* __restrict__ offsets, int n_rot, int n_part, const float* __restrict__ phis, int res,
                  int rl, double rho1, double* __restrict__ partial, float* __restrict__ samples) {
  __shared__ McPhi sphi;
  mc_load_phi(&sphi, phis, res);
  double acc = 0.0;
  const int64_t items = (nc + 31) / 32 * n_part * 32;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < items; k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t w32 = k >> 5;
    const int part = (int)(w32 % n_part);
    const int64_t i = w32 / n_part * 32 + (k & 31);
    if (i >= nc) continue;
    const double x = centers[3 * i], y = centers[3 * i + 1], z = centers[3 * i + 2];
    const float n1 = eps1 ? mc_value<kLayout>(eps1, &sphi, res, rl, J, x, y, z) : (float)rho1;
    const float w = cw ? (float)cw[i] : 1.f;
    float s = 0.f;
    for (int r = part; r < n_rot; r += n_part) {
      const double* o = offsets + 6 * r;
      const float n2 = mc_value<kLayout>(eps2, &sphi, res, rl, J, x + o[0], y + o[1], z + o[2]);
      const float n3 = mc_value<kLayout>(eps3, &sphi, res, rl, J, x + o[3], y + o[4], z + o[5]);
      const float f = w * n1 * n2 * n3;
      if (samples) samples[i * n_rot + r] = f;
      s += f;
    }
    acc += (double)s;
  }
  __shared__ double sh[256];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

__global__ void mc_sum_kernel(const double* __restrict__ partial, int n, double* __restrict__ out) {
  __shared__ double sh[256];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

// SplitMix64 (Steele, Lea and Flood, 2014): a counter-based generator, so a
// sample's draws depend only on (seed, sample index) and not on the launch.
__device__ __forceinline__ unsigned long long mc_splitmix(unsigned long long& s) {
  unsigned long long z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ double mc_u01(unsigned long long& s) {
  return (double)(mc_splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
}

// generate_triangle_offsets (corr3pcf_kernels.py:21-63) in float64 with the
// angles given as fractions of a turn: phi = 2 pi fp, alpha = 2 pi fa.
__device__ __forceinline__ void mc_triangle(double R1, double R2, double mu, double fp, double ct1, double fa,
                                            double o[6]) {
  const double st1 = sqrt(1.0 - ct1 * ct1);
  double sp, cp, sa, ca;
  sincospi(2.0 * fp, &sp, &cp);
  sincospi(2.0 * fa, &sa, &ca);
  const double dx1 = st1 * cp, dy1 = st1 * sp, dz1 = ct1;
  double ox1, oy1, oz1;
  if (fabs(dx1) > 1e-10 || fabs(dy1) > 1e-10) {
    ox1 = -dy1; oy1 = dx1; oz1 = 0.0;
  } else {
    ox1 = 0.0; oy1 = -dz1; oz1 = dy1;
  }
  const double nrm = sqrt(ox1 * ox1 + oy1 * oy1 + oz1 * oz1);
  ox1 /= nrm; oy1 /= nrm; oz1 /= nrm;
  const double ox2 = dy1 * oz1 - dz1 * oy1, oy2 = dz1 * ox1 - dx1 * oz1, oz2 = dx1 * oy1 - dy1 * ox1;
  double st2 = 1.0 - mu * mu;
  if (st2 < 0.0) st2 = 0.0;
  const double st = sqrt(st2);
  o[0] = R1 * dx1; o[1] = R1 * dy1; o[2] = R1 * dz1;
  o[3] = R2 * (mu * dx1 + st * (ca * ox1 + sa * ox2));
  o[4] = R2 * (mu * dy1 + st * (ca * oy1 + sa * oy2));
  o[5] = R2 * (mu * dz1 + st * (ca * oz1 + sa * oz2));
}

// One triplet per sample k: centre c = pool[i], i = idx[k] (clamped to
// [0, M)) or uniform in [0, M) when idx == NULL; offsets from `offsets`
// [n][6] or drawn (phi, cos theta1, alpha uniform, as the reference's three
// uniforms); value f_k = w_k n1(c) n2(c + o1) n3(c + o2) (w_k = 1 when w is
// NULL).  Block partial sums of f and f^2.
template <int kLayout>
__global__ void __launch_bounds__(256)
mc_sample_kernel(const float* __restrict__ eps1, const float* __restrict__ eps2, const float* __restrict__ eps3,
                 int J, const double* __restrict__ pool, long long M, const long long* __restrict__ idx,
                 const double* __restrict__ w, const double* __restrict__ offsets, long long n, double R1, double R2,
                 double mu, unsigned long long seed, const float* __restrict__ phis, int res, int rl,
                 double* __restrict__ partial) {
  __shared__ McPhi sphi;
  mc_load_phi(&sphi, phis, res);
  double acc = 0.0, acc2 = 0.0;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    unsigned long long st = seed ^ ((unsigned long long)k * 0xD1B54A32D192ED03ull);
    long long i;
    if (idx) {
      i = idx[k];
      i = i < 0 ? 0 : (i >= M ? M - 1 : i);  // indices outside the pool are clamped, never read past it
    } else {
      i = (long long)(mc_u01(st) * (double)M);
      if (i >= M) i = M - 1;
    }
    double o[6];
    if (offsets) {
#pragma unroll
      for (int q = 0; q < 6; ++q) o[q] = offsets[6 * k + q];
    } else {
      const double a = mc_u01(st), bb = mc_u01(st), c = mc_u01(st);
      mc_triangle(R1, R2, mu, a, 2.0 * bb - 1.0, c, o);
    }
    const double x = pool[3 * i], y = pool[3 * i + 1], z = pool[3 * i + 2];
    const float n1 = mc_value<kLayout>(eps1, &sphi, res, rl, J, x, y, z);
    const float n2 = mc_value<kLayout>(eps2, &sphi, res, rl, J, x + o[0], y + o[1], z + o[2]);
    const float n3 = mc_value<kLayout>(eps3, &sphi, res, rl, J, x + o[3], y + o[4], z + o[5]);
    double f = (double)(n1 * n2 * n3);
    if (w) f *= w[k];
    acc += f;
    acc2 += f * f;
  }
  __shared__ double sh[2][256];
  sh[0][threadIdx.x] = acc;
  sh[1][threadIdx.x] = acc2;
  __syncthreads();
  for (int s2 = blockDim.x / 2; s2 > 0; s2 >>= 1) {
    if (threadIdx.x < s2) {
      sh[0][threadIdx.x] += sh[0][threadIdx.x + s2];
      sh[1][threadIdx.x] += sh[1][threadIdx.x + s2];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = sh[0][0];
    partial[gridDim.x + blockIdx.x] = sh[1][0];
  }
}

// dst[mc_cell<true>(x, y, z)] = src[mc_cell<false>(x, y, z)], one thread per
// brick: the four 8-byte reads of a warp are 256 contiguous bytes each, its
// 32-byte writes 1 KB.  src 8-byte and dst 32-byte aligned.
__global__ void __launch_bounds__(256) mc_bricks_kernel(const float* __restrict__ src, int J, float* __restrict__ dst) {
  const int h = J - 1;
  const unsigned n = 1u << (3 * h), hm = (1u << h) - 1;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned x = i >> (2 * h), y = (i >> h) & hm, z = i & hm;
    const float2* row = reinterpret_cast<const float2*>(src) + ((((size_t)(2 * x) << J) + 2 * y) << h) + z;
    const size_t dy = (size_t)1 << h, dx = dy << J;
    const float2 a = __ldcs(row), b = __ldcs(row + dy), c = __ldcs(row + dx), d = __ldcs(row + dx + dy);
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + ((size_t)i << 3)), "f"(a.x), "f"(a.y),
                 "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y), "f"(d.x), "f"(d.y)
                 : "memory");
  }
}

// The same at any alignment, one thread per cell.
__global__ void mc_to_bricks_kernel(const float* __restrict__ src, int J, float* __restrict__ dst) {
  const size_t n = (size_t)1 << (3 * J);
  const int h = J - 1;
  const size_t hm = ((size_t)1 << h) - 1;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t brick = i >> 3;
    const int c = (int)(i & 7);
    const int x = (int)(((brick >> (2 * h)) & hm) << 1) | (c >> 2);
    const int y = (int)(((brick >> h) & hm) << 1) | ((c >> 1) & 1);
    const int z = (int)((brick & hm) << 1) | (c & 1);
    dst[i] = __ldg(src + mc_cell<false>(x, y, z, J));
  }
}

bool aligned(uintptr_t bytes, const float* a, const float* b = nullptr, const float* c = nullptr) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & (bytes - 1)) == 0;
}

int log2_or_negative(int v) { return (v & (v - 1)) == 0 ? __builtin_ctz((unsigned)v) : -1; }

int mc_grid() {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm * 8;
}

}  // namespace

extern "C" int hermes_mc_workspace_size(size_t* bytes) {
  if (!bytes) return fail(HERMES_ERR_INVALID, "bytes is NULL");
  hermes::Carver c(nullptr, 0);
  c.take<float>(4 * 1024);
  c.take<double>(2 * ((size_t)mc_grid() + 1));
  *bytes = c.used;
  return HERMES_OK;
}

static int mc_prepare(const double* phi, int n_phi, int res, void* workspace, size_t workspace_bytes, float** phis,
                      double** partial, cudaStream_t s) {
  if (!phi || res <= 0 || n_phi != 3 * res || res > 1024)
    return fail(HERMES_ERR_INVALID, "mc: phi must hold 3*res samples with res <= 1024 (n_phi=%d, res=%d)", n_phi, res);
  size_t need = 0;
  hermes_mc_workspace_size(&need);
  if (!workspace || workspace_bytes < need) return fail(HERMES_ERR_WORKSPACE, "mc: workspace %zu < %zu", workspace_bytes, need);
  hermes::Carver c(workspace, workspace_bytes);
  *phis = c.take<float>(4 * 1024);
  *partial = c.take<double>(2 * ((size_t)mc_grid() + 1));
  mc_phi_kernel<<<4, 256, 0, s>>>(phi, n_phi, *phis);
  HERMES_LAUNCH_CHECK("mc_phi_kernel");
  return HERMES_OK;
}

extern "C" int hermes_interp(const float* grid, int J, const double* scaled_pos, int64_t n, const double* phi,
                             int n_phi, int phi_res, double dx, double dy, double dz, double* out, void* workspace,
                             size_t workspace_bytes, void* stream) {
  if (!grid || (n > 0 && (!scaled_pos || !out))) return fail(HERMES_ERR_INVALID, "interp: NULL argument");
  if (J < 2 || J > 10) return fail(HERMES_ERR_INVALID, "interp: J=%d outside [2,10]", J);
  cudaStream_t s = hermes::as_stream(stream);
  float* phis;
  double* partial;
  int rc = mc_prepare(phi, n_phi, phi_res, workspace, workspace_bytes, &phis, &partial, s);
  if (rc) return rc;
  if (n == 0) return HERMES_OK;
  const auto kernel = aligned(16, grid) ? mc_interp_kernel<kCOrder> : mc_interp_kernel<kCells>;
  kernel<<<mc_grid(), 256, 0, s>>>(grid, J, scaled_pos, n, phis, phi_res, log2_or_negative(phi_res), dx, dy,
                                   dz, out);
  HERMES_LAUNCH_CHECK("mc_interp_kernel");
  return HERMES_OK;
}

static int mc_triplets(const float* eps1, const float* eps2, const float* eps3, int J, const double* centers,
                       const double* center_w, int64_t n_centers, const double* offsets, int n_rot, const double* phi,
                       int n_phi, int phi_res, double rho1, double* sum_out, float* samples_out, void* workspace,
                       size_t workspace_bytes, void* stream, bool bricks) {
  if (!eps2 || !eps3 || !sum_out || (n_centers > 0 && !centers) || (n_rot > 0 && !offsets))
    return fail(HERMES_ERR_INVALID, "mc_triplets: NULL argument");
  if (J < 2 || J > 10) return fail(HERMES_ERR_INVALID, "mc_triplets: J=%d outside [2,10]", J);
  if (n_rot < 0 || n_centers < 0) return fail(HERMES_ERR_INVALID, "mc_triplets: negative count");
  cudaStream_t s = hermes::as_stream(stream);
  float* phis;
  double* partial;
  int rc = mc_prepare(phi, n_phi, phi_res, workspace, workspace_bytes, &phis, &partial, s);
  if (rc) return rc;
  const int g = mc_grid();
  // about 8 rotations a thread: each part interpolates its centre's n1 again
  // (6% at 8); fewer parts leave the grid short of threads or spread the
  // threads in flight over the box
  const int n_part = std::max(1, n_rot / 8);
  const int rl = log2_or_negative(phi_res);
  const bool wide = aligned(bricks ? 32 : 16, eps1, eps2, eps3);
  const auto kernel = bricks ? (wide ? mc_triplet_kernel<kBricks> : mc_triplet_kernel<kBrickCells>)
                             : (wide ? mc_triplet_kernel<kCOrder> : mc_triplet_kernel<kCells>);
  kernel<<<g, 256, 0, s>>>(eps1, eps2, eps3, J, centers, center_w, n_centers, offsets, n_rot, n_part, phis, phi_res, rl,
                           rho1, partial, samples_out);
  HERMES_LAUNCH_CHECK("mc_triplet_kernel");
  mc_sum_kernel<<<1, 256, 0, s>>>(partial, g, partial + g);
  HERMES_LAUNCH_CHECK("mc_sum_kernel");
  HERMES_CUDA_TRY(cudaMemcpyAsync(sum_out, partial + g, sizeof(double), cudaMemcpyDeviceToHost, s));
  HERMES_CUDA_TRY(cudaStreamSynchronize(s));
  return HERMES_OK;
}

static int mc_sample(const float* eps1, const float* eps2, const float* eps3, int J, const double* pool, int64_t M,
                     const int64_t* idx, const double* weights, const double* offsets, int64_t n, double R1, double R2,
                     double mu, uint64_t seed, const double* phi, int n_phi, int phi_res, double* sums_out,
                     void* workspace, size_t workspace_bytes, void* stream, bool bricks) {
  if (!eps1 || !eps2 || !eps3 || !sums_out) return fail(HERMES_ERR_INVALID, "mc_sample: NULL argument");
  if (J < 2 || J > 10) return fail(HERMES_ERR_INVALID, "mc_sample: J=%d outside [2,10]", J);
  if (n < 0 || M < 0) return fail(HERMES_ERR_INVALID, "mc_sample: negative count");
  if (n > 0 && (!pool || M == 0)) return fail(HERMES_ERR_INVALID, "mc_sample: empty centre pool");
  cudaStream_t s = hermes::as_stream(stream);
  float* phis;
  double* partial;
  int rc = mc_prepare(phi, n_phi, phi_res, workspace, workspace_bytes, &phis, &partial, s);
  if (rc) return rc;
  const int g = mc_grid();
  const int rl = log2_or_negative(phi_res);
  const bool wide = aligned(bricks ? 32 : 16, eps1, eps2, eps3);
  const auto kernel = bricks ? (wide ? mc_sample_kernel<kBricks> : mc_sample_kernel<kBrickCells>)
                             : (wide ? mc_sample_kernel<kCOrder> : mc_sample_kernel<kCells>);
  kernel<<<g, 256, 0, s>>>(eps1, eps2, eps3, J, pool, (long long)M, reinterpret_cast<const long long*>(idx), weights,
                           offsets, (long long)n, R1, R2, mu, (unsigned long long)seed, phis, phi_res, rl, partial);
  HERMES_LAUNCH_CHECK("mc_sample_kernel");
  mc_sum_kernel<<<1, 256, 0, s>>>(partial, g, partial + 2 * g);
  HERMES_LAUNCH_CHECK("mc_sum_kernel");
  mc_sum_kernel<<<1, 256, 0, s>>>(partial + g, g, partial + 2 * g + 1);
  HERMES_LAUNCH_CHECK("mc_sum_kernel");
  HERMES_CUDA_TRY(cudaMemcpyAsync(sums_out, partial + 2 * g, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
  HERMES_CUDA_TRY(cudaStreamSynchronize(s));
  return HERMES_OK;
}

extern "C" int hermes_mc_triplets(const float* eps1, const float* eps2, const float* eps3, int J,
                                  const double* centers, const double* center_w, int64_t n_centers,
                                  const double* offsets, int n_rot, const double* phi, int n_phi, int phi_res,
                                  double rho1, double* sum_out, float* samples_out, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  return mc_triplets(eps1, eps2, eps3, J, centers, center_w, n_centers, offsets, n_rot, phi, n_phi, phi_res, rho1,
                     sum_out, samples_out, workspace, workspace_bytes, stream, false);
}

extern "C" int hermes_mc_triplets_bricks(const float* eps1, const float* eps2, const float* eps3, int J,
                                         const double* centers, const double* center_w, int64_t n_centers,
                                         const double* offsets, int n_rot, const double* phi, int n_phi, int phi_res,
                                         double rho1, double* sum_out, float* samples_out, void* workspace,
                                         size_t workspace_bytes, void* stream) {
  return mc_triplets(eps1, eps2, eps3, J, centers, center_w, n_centers, offsets, n_rot, phi, n_phi, phi_res, rho1,
                     sum_out, samples_out, workspace, workspace_bytes, stream, true);
}

extern "C" int hermes_mc_sample(const float* eps1, const float* eps2, const float* eps3, int J, const double* pool,
                                int64_t M, const int64_t* idx, const double* weights, const double* offsets,
                                int64_t n, double R1, double R2, double mu, uint64_t seed, const double* phi,
                                int n_phi, int phi_res, double* sums_out, void* workspace, size_t workspace_bytes,
                                void* stream) {
  return mc_sample(eps1, eps2, eps3, J, pool, M, idx, weights, offsets, n, R1, R2, mu, seed, phi, n_phi, phi_res,
                   sums_out, workspace, workspace_bytes, stream, false);
}

extern "C" int hermes_mc_sample_bricks(const float* eps1, const float* eps2, const float* eps3, int J,
                                       const double* pool, int64_t M, const int64_t* idx, const double* weights,
                                       const double* offsets, int64_t n, double R1, double R2, double mu,
                                       uint64_t seed, const double* phi, int n_phi, int phi_res, double* sums_out,
                                       void* workspace, size_t workspace_bytes, void* stream) {
  return mc_sample(eps1, eps2, eps3, J, pool, M, idx, weights, offsets, n, R1, R2, mu, seed, phi, n_phi, phi_res,
                   sums_out, workspace, workspace_bytes, stream, true);
}

extern "C" int hermes_mc_morton_keys(const double* centers, int64_t n, int J, int32_t* keys, void* stream) {
  if (n < 0 || (n > 0 && (!centers || !keys))) return fail(HERMES_ERR_INVALID, "mc_morton_keys: bad argument");
  if (J < 2 || J > 10) return fail(HERMES_ERR_INVALID, "mc_morton_keys: J=%d outside [2,10]", J);
  if (n == 0) return HERMES_OK;
  const int grid = (int)std::min<int64_t>((n + 255) / 256, mc_grid());
  mc_morton_kernel<<<grid, 256, 0, hermes::as_stream(stream)>>>(centers, n, 1 << J, keys);
  HERMES_LAUNCH_CHECK("mc_morton_kernel");
  return HERMES_OK;
}

extern "C" int hermes_field_to_bricks(const float* field, int J, float* bricks, void* stream) {
  if (!field || !bricks) return fail(HERMES_ERR_INVALID, "field_to_bricks: NULL argument");
  if (J < 2 || J > 10) return fail(HERMES_ERR_INVALID, "field_to_bricks: J=%d outside [2,10]", J);
  if (field == bricks) return fail(HERMES_ERR_INVALID, "field_to_bricks: the copy cannot be in place");
  const auto kernel = aligned(8, field) && aligned(32, bricks) ? mc_bricks_kernel : mc_to_bricks_kernel;
  kernel<<<mc_grid(), 256, 0, hermes::as_stream(stream)>>>(field, J, bricks);
  HERMES_LAUNCH_CHECK("mc_to_bricks_kernel");
  return HERMES_OK;
}
