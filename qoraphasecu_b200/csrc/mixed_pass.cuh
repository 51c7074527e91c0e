// Mixed-radix line passes with in-register DFTs of up to 16 points
// (mixed_pass_kernel.cuh), for line lengths whose prime factors are at most 13.
#pragma once

#include "line_pass.cuh"

namespace qpb {

// True when the mixed-radix pass runs lines of p.L points with the storage of
// `p` (complex64 wave and iterate, amplitude in FFT order).
bool mixed_pass_supports(const PassParams& p);

void launch_mixed_pass(Mode mode, const PassParams& p, cudaStream_t stream);

// Sets the shared-memory attributes of the mixed-radix kernels on the current
// device (configure_line_passes).
void configure_mixed_passes();

// The same for one mode (mixed_pass_project.cu, _gradient, _update, _blur and _plain).
template <Mode M>
void launch_mixed_mode(const PassParams& p, cudaStream_t stream);
template <Mode M>
void configure_mixed_mode();

}  // namespace qpb
