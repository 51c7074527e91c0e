// The lengths of the two-stage line passes (two_stage_kernel.cuh) and how they
// factor, for the kernels and for the host code that plans them.
#pragma once

namespace qpb {

// Longest line with a two-stage pass: both DFTs of at most 25 points.
inline constexpr int kMaxTwoStage = 625;

constexpr bool two_stage_radix(int r) {
  return (r >= 2 && r <= 10) || r == 12 || (r >= 14 && r <= 16) || r == 18 || r == 20 || r == 21 ||
         r == 24 || r == 25;
}

// The larger factor A of L = A B, both two_stage_radix and A as small as it
// can be; 0 when L has no such factors (or takes one stage).
constexpr int two_stage_large(int L) {
  if (L <= 16 || L > kMaxTwoStage) return 0;
  for (int a = 2; a <= 25; ++a) {
    if (L % a == 0 && L / a <= a && two_stage_radix(a) && two_stage_radix(L / a)) return a;
  }
  return 0;
}

}  // namespace qpb
