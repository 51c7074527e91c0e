// The mixed-radix passes' modulus mode.

#include "mixed_pass_kernel.cuh"

namespace qpb {

template void launch_mixed_mode<Mode::kMod>(const PassParams&, cudaStream_t);
template void configure_mixed_mode<Mode::kMod>();

}  // namespace qpb
