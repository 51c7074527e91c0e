// The mixed-radix passes' update modes.

#include "mixed_pass_kernel.cuh"

namespace qpb {

template void launch_mixed_mode<Mode::kUpd>(const PassParams&, cudaStream_t);
template void launch_mixed_mode<Mode::kCut>(const PassParams&, cudaStream_t);
template void configure_mixed_mode<Mode::kUpd>();
template void configure_mixed_mode<Mode::kCut>();

}  // namespace qpb
