// Dispatch of the mixed-radix line passes (mixed_pass_kernel.cuh).

#include "mixed_pass.cuh"

namespace qpb {

bool mixed_pass_supports(const PassParams& p) {
  // (offsets within a start are 32-bit)
  return p.plan && p.plan->mixed_stages > 0 && p.n <= 0x7fffffffLL && !p.amp_tiled && !p.wave_half && !p.iter_half;
}

void launch_mixed_pass(Mode mode, const PassParams& p, cudaStream_t stream) {
  switch (mode) {
    case Mode::kFwd:
      return launch_mixed_mode<Mode::kFwd>(p, stream);
    case Mode::kFwdFromX:
      return launch_mixed_mode<Mode::kFwdFromX>(p, stream);
    case Mode::kInv:
      return launch_mixed_mode<Mode::kInv>(p, stream);
    case Mode::kMod:
      return launch_mixed_mode<Mode::kMod>(p, stream);
    case Mode::kUpd:
      return launch_mixed_mode<Mode::kUpd>(p, stream);
    case Mode::kCut:
      return launch_mixed_mode<Mode::kCut>(p, stream);
    case Mode::kBlur:
      return launch_mixed_mode<Mode::kBlur>(p, stream);
    case Mode::kBlurMag:
      return launch_mixed_mode<Mode::kBlurMag>(p, stream);
    case Mode::kGrad:
      return launch_mixed_mode<Mode::kGrad>(p, stream);
  }
}

void configure_mixed_passes() {
  configure_mixed_mode<Mode::kFwd>();
  configure_mixed_mode<Mode::kFwdFromX>();
  configure_mixed_mode<Mode::kInv>();
  configure_mixed_mode<Mode::kMod>();
  configure_mixed_mode<Mode::kUpd>();
  configure_mixed_mode<Mode::kCut>();
  configure_mixed_mode<Mode::kBlur>();
  configure_mixed_mode<Mode::kBlurMag>();
  configure_mixed_mode<Mode::kGrad>();
}

}  // namespace qpb
