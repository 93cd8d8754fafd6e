// 512-point FFT passes (fft_lines.cu) of a convolution's half spectrum.
#pragma once

#include "hermes_common.cuh"

namespace hermes {

// Row pitch (float2) of the half spectra [512][512][pitch] of these passes:
// 257 values and padding to whole 128-byte rows, which the 16-byte copies and
// the 16-column tiles want.  The buffer is 16-byte aligned.
constexpr int kFft512HalfPitch = 272;

// A real window on the half spectrum: G[x] G[y] G[z] scale (axis_factor), or
// folded[column][257] with column = hi (hi + 1) / 2 + lo of the sorted
// (min(x, 512 - x), min(y, 512 - y)).
struct FftWindow {
  const float* axis_factor;
  const float* folded;
  float scale, factor;  // factor: the transform's normalisation
  int zero_k0;
};

// z lines of a real field [512][512][512] to half spectra and back,
// unnormalised.
int fft512_real_to_half(const float* in, float2* out, cudaStream_t s);
int fft512_half_to_real(const float2* in, float* out, cudaStream_t s);
// y transform, in place, unnormalised.
int fft512_half_y(float2* data, bool forward, cudaStream_t s);
// Forward x transform into compact rows, out[512][512][257]; data is left as it is.
int fft512_half_x_compact(float2* data, float2* out, cudaStream_t s);
// Forward x transform, the window, inverse x transform, in place.
int fft512_half_x_window_x(float2* data, const FftWindow& win, cudaStream_t s);

}  // namespace hermes
