// Two-stage line passes compiled per length (two_stage_kernel.cuh): the passes
// of an iteration and of the loss gradient for lines of L = A B points, A and
// B at most 25 (two_stage.hpp).
#pragma once

#include "line_pass.cuh"
#include "two_stage.hpp"

namespace qpb {

// One length's pass of one mode.
struct TwoStagePass {
  int length;
  void (*launch)(const PassParams&, cudaStream_t);
  void (*configure)();
};

// The passes of mode M (columns, or rows), the lengths in kTwoStageSlices parts;
// instantiated by two_stage_*.cu.
struct TwoStageList {
  const TwoStagePass* passes;
  int count;
};
inline constexpr int kTwoStageSlices = 2;
template <Mode M, bool ROWS, int SLICE>
TwoStageList two_stage_slice();

// True when `mode` over the lines of `p` has a two-stage pass.
bool two_stage_supports(Mode mode, const PassParams& p);

void launch_two_stage_pass(Mode mode, const PassParams& p, cudaStream_t stream);

// Sets the shared-memory attributes of the passes of length L on the current
// device (configure_line_passes).
void configure_two_stage(int L);

}  // namespace qpb
