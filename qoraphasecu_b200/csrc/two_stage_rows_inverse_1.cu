// Two-stage passes, mode kInv along rows: slice 1 of the lengths.

#include "two_stage_kernel.cuh"

namespace qpb {

template TwoStageList two_stage_slice<Mode::kInv, true, 1>();

}  // namespace qpb
