// Two-stage passes, mode kMod along columns: slice 1 of the lengths.

#include "two_stage_kernel.cuh"

namespace qpb {

template TwoStageList two_stage_slice<Mode::kMod, false, 1>();

}  // namespace qpb
