// Two-stage passes, mode kCut along rows: slice 1 of the lengths.

#include "two_stage_kernel.cuh"

namespace qpb {

template TwoStageList two_stage_slice<Mode::kCut, true, 1>();

}  // namespace qpb
