// Dispatch of the two-stage line passes (two_stage_kernel.cuh).

#include <array>

#include "two_stage_pass.cuh"

namespace qpb {

namespace {

using Table = std::array<const TwoStagePass*, kMaxTwoStage + 1>;

template <Mode M, bool ROWS>
const Table& table() {
  static const Table passes = [] {
    Table t{};
    for (const TwoStageList& list : {two_stage_slice<M, ROWS, 0>(), two_stage_slice<M, ROWS, 1>()}) {
      for (int i = 0; i < list.count; ++i) t[list.passes[i].length] = &list.passes[i];
    }
    return t;
  }();
  return passes;
}

// The pass of `mode` for lines of L points, or null: the passes of an
// iteration and of the loss gradient, in the direction they run in. The rest
// (starts, blurs, a lone axis) runs the run-time mixed-radix kernel.
const TwoStagePass* find(Mode mode, int L, bool rows) {
  if (L < 0 || L > kMaxTwoStage) return nullptr;
  if (rows) {
    switch (mode) {
      case Mode::kUpd: return table<Mode::kUpd, true>()[L];
      case Mode::kCut: return table<Mode::kCut, true>()[L];
      case Mode::kFwdFromX: return table<Mode::kFwdFromX, true>()[L];
      case Mode::kInv: return table<Mode::kInv, true>()[L];
      default: return nullptr;
    }
  }
  switch (mode) {
    case Mode::kMod: return table<Mode::kMod, false>()[L];
    case Mode::kGrad: return table<Mode::kGrad, false>()[L];
    case Mode::kFwd: return table<Mode::kFwd, false>()[L];
    case Mode::kInv: return table<Mode::kInv, false>()[L];
    default: return nullptr;
  }
}

}  // namespace

bool two_stage_supports(Mode mode, const PassParams& p) {
  // (offsets within a start are 32-bit)
  return p.two_stage_twiddle && p.n <= 0x7fffffffLL && !p.amp_tiled && !p.wave_half &&
         !p.iter_half && find(mode, p.L, p.S == 1);
}

void launch_two_stage_pass(Mode mode, const PassParams& p, cudaStream_t stream) {
  find(mode, p.L, p.S == 1)->launch(p, stream);
}

void configure_two_stage(int L) {
  for (const Mode mode : {Mode::kUpd, Mode::kCut, Mode::kFwdFromX, Mode::kInv, Mode::kMod, Mode::kGrad,
                          Mode::kFwd}) {
    for (const bool rows : {false, true}) {
      if (const TwoStagePass* pass = find(mode, L, rows)) pass->configure();
    }
  }
}

}  // namespace qpb
