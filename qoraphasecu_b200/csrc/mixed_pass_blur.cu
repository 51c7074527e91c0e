// The mixed-radix passes' blur modes.

#include "mixed_pass_kernel.cuh"

namespace qpb {

template void launch_mixed_mode<Mode::kBlur>(const PassParams&, cudaStream_t);
template void launch_mixed_mode<Mode::kBlurMag>(const PassParams&, cudaStream_t);
template void configure_mixed_mode<Mode::kBlur>();
template void configure_mixed_mode<Mode::kBlurMag>();

}  // namespace qpb
