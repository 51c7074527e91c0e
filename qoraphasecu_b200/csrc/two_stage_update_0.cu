// Two-stage passes, mode kUpd along rows: slice 0 of the lengths.

#include "two_stage_kernel.cuh"

namespace qpb {

template TwoStageList two_stage_slice<Mode::kUpd, true, 0>();

}  // namespace qpb
