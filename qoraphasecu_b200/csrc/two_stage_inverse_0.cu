// Two-stage passes, mode kInv along columns: slice 0 of the lengths.

#include "two_stage_kernel.cuh"

namespace qpb {

template TwoStageList two_stage_slice<Mode::kInv, false, 0>();

}  // namespace qpb
