// Host-side plans for the line FFTs: the radix sequence of each length and its
// twiddle table W_L^k = exp(-2 pi i k / L), computed in FP64 and rounded once
// to FP32 on upload.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <memory>
#include <mutex>
#include <vector>

namespace qpb {

inline constexpr int kMaxStages = 16;
// Stages of a mixed-radix pass (mixed_pass.cu), radices 2..16.
inline constexpr int kMaxMixedStages = 6;
// Largest prime factor a line length may have; such radices run as a direct
// DFT inside a Stockham stage.
inline constexpr int kMaxPrimeRadix = 127;
// Longest line a shared-memory line pass holds.
inline constexpr int kMaxLine = 8192;

struct LinePlan {
  int length = 1;
  int stages = 0;
  int radix[kMaxStages] = {};
  const float2* twiddle = nullptr;  // device, `length` entries
  // device, the stage-major table of the register-resident transform
  // (stage_table.hpp) for lengths that have one, else `twiddle`
  const float2* stage_twiddle = nullptr;
  // the mixed-radix pass's radices (mixed_stages 0: a prime factor above 13)
  // and, on the device, its stage-major twiddles: for each stage after the
  // first, with N the product of the radices before it, W_{N R}^{q k} at
  // (q - 1) N + k; then the same for the radices in reverse order
  int mixed_stages = 0;
  int mixed_radix[kMaxMixedStages] = {};
  // slots from one block of N R outputs to the next in the exchange after each
  // stage, for the radices in order and reversed (exchange_pitch)
  int mixed_pitch[2][kMaxMixedStages] = {};
  const float2* mixed_twiddle = nullptr;
  // on the device, the two-stage pass's W_L^{q t} for L = A B (two_stage.hpp;
  // null without one): at (q - 1) A + t for q < B, t < A, then at
  // (q - 1) B + t for q < A, t < B
  const float2* two_stage_twiddle = nullptr;
};

// Radix sequence for a line of length `n` (throws InvalidArgument when a prime
// factor exceeds kMaxPrimeRadix or n exceeds kMaxLine).
std::vector<int> factorize(int n);

// Radices 2..16 whose product is n, as few as there can be and among those
// with the smallest largest and then the largest smallest one; empty for n < 2 and when a prime factor of n
// is above 13.
std::vector<int> mixed_radices(int n);

// The smallest P >= N R at which 16 neighbouring items j of a stage, which
// write 8-byte values to slots (j / N) P + j mod N (+ q N), meet the fewest
// shared-memory bank conflicts.
int exchange_pitch(int n, int radix);

// Per-device cache of line plans; twiddle tables live until the cache dies.
class PlanCache {
 public:
  PlanCache() = default;
  PlanCache(const PlanCache&) = delete;
  PlanCache& operator=(const PlanCache&) = delete;
  ~PlanCache();

  const LinePlan& get(int length);

  // Device counter of the line-pass CTAs whose bounded wait for their staged
  // inputs gave up (those CTAs wrote nothing), shared by every pass planned
  // from this cache: a solver's own cache makes it per solver. Allocated and
  // zeroed on first use, which must not fall inside a stream capture.
  int* wait_failures();

  // Reads the counter on `stream` after the work enqueued there, clears it
  // when it is set, and returns what it held. Synchronises `stream`.
  int take_wait_failures(cudaStream_t stream);

 private:
  std::mutex mutex_;
  std::map<int, LinePlan> plans_;
  std::vector<void*> allocations_;
  int* failures_ = nullptr;
};

}  // namespace qpb
