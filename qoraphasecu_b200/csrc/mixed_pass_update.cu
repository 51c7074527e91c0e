// The mixed-radix passes' update mode.

#include "mixed_pass_kernel.cuh"

namespace qpb {

template void launch_mixed_mode<Mode::kUpd>(const PassParams&, cudaStream_t);
template void configure_mixed_mode<Mode::kUpd>();

}  // namespace qpb
