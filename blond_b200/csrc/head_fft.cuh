// The rfft -> x Z -> irfft chain of a long power-of-two profile in one
// cluster of 16 CTAs (see head_fft.cu); used by launch_spectral.
#pragma once

#include "spectral.cuh"

namespace bb {

// True when the parameters describe a transform this kernel takes.
bool head_fft_takes(const SpecParams& P);
int launch_head_fft(const SpecParams& P, cudaStream_t stream);
// Kernel attributes, set outside stream capture.
int prepare_head_fft();
// An n_fft that is no power of two, S profile bins: the outputs need the
// impulse response at lags |d| < S only, which a circular convolution of
// length P >= 2 S - 1 gives as well.  P when this kernel takes it, else 0
// (turns of 1e7 FP64 particles, 20000 slices: 116 us with the mixed-radix
// transform of 20000 points, 86 with this one of 65536).
int64_t head_fft_length(int64_t N, int S);
// The spectrum (cudaMalloc'd, P / 2 + 1 values) of that response from the
// impedance H, N / 2 + 1 values on the device.  Synchronous.
int make_head_response(const double2* H, int64_t N, int S, int64_t P, double2** out);

}  // namespace bb
