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

}  // namespace bb
