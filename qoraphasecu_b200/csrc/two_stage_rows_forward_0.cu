// Two-stage passes, mode kFwdFromX along rows: slice 0 of the lengths.

#include "two_stage_kernel.cuh"

namespace qpb {

template TwoStageList two_stage_slice<Mode::kFwdFromX, true, 0>();

}  // namespace qpb
