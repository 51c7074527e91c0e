// The mixed-radix passes' single-transform modes.

#include "mixed_pass_kernel.cuh"

namespace qpb {

template void launch_mixed_mode<Mode::kFwd>(const PassParams&, cudaStream_t);
template void configure_mixed_mode<Mode::kFwd>();
template void launch_mixed_mode<Mode::kFwdFromX>(const PassParams&, cudaStream_t);
template void configure_mixed_mode<Mode::kFwdFromX>();
template void launch_mixed_mode<Mode::kInv>(const PassParams&, cudaStream_t);
template void configure_mixed_mode<Mode::kInv>();

}  // namespace qpb
