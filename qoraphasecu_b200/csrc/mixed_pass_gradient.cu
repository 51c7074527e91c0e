// The mixed-radix passes' loss-gradient mode.

#include "mixed_pass_kernel.cuh"

namespace qpb {

template void launch_mixed_mode<Mode::kGrad>(const PassParams&, cudaStream_t);
template void configure_mixed_mode<Mode::kGrad>();

}  // namespace qpb
