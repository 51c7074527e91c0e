// Two-stage passes, mode kFwd along columns: slice 1 of the lengths.

#include "two_stage_kernel.cuh"

namespace qpb {

template TwoStageList two_stage_slice<Mode::kFwd, false, 1>();

}  // namespace qpb
