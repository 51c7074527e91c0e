// Two-stage line passes: lines of L = A B points (A >= B, both at most 25),
// one kernel per length, mode and direction, for lengths that are no power of
// two (and powers of two whose lines do not fill the tiles of the other
// passes).
//
// A line belongs to A threads. Thread t < B transforms the A points t + q B
// straight from global memory, an exchange in shared memory gives every
// thread t its B points t + q A, which it twiddles and transforms; a pass of
// two transforms applies the point-wise step there, in registers, and runs
// the same way back. The A-point DFTs, the ends of the pass, keep B of the A
// threads busy; the B-point DFTs with the point-wise step, its larger part,
// keep all of them.
//
// Bound: issue and latency. Against the run-time mixed-radix kernel
// (mixed_pass_kernel.cuh) everything but the strides of the arrays is a
// compile-time constant, and the code runs straight through: with one kernel
// for all radices the instruction fetches of the scattered stages cost about
// 3 us at every change of pass (96 x 96, 4 starts: 4.2 + 3.9 us for the two
// passes repeated alone, 13.7 us an iteration; here 2.9 + 2.8 and 6.0). Other
// iterations, line_pass.cu -> here: 16 starts of 240 x 240 71 -> 18 us, 4 of
// 300 x 200 36 -> 10, 2 of 96^3 125 -> 37.
//
// Shared memory holds a line's exchange as consecutive slots. After the
// A-point stage output q of thread j sits at j (A | 1) + q and after the
// B-point one at j (B | 1) + q: odd distances, so the threads of a half-warp
// write to different banks. The lines of a column block, on adjacent threads,
// are 2 mod 16 slots apart: 8 lines and 2 threads a half-warp.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <array>
#include <stdexcept>

#include "dependent_launch.cuh"
#include "projection.cuh"
#include "reduce.cuh"
#include "small_dft.cuh"
#include "two_stage_pass.cuh"

namespace qpb {

namespace {

template <int L, Mode M, bool ROWS>
struct TwoStage {
  static constexpr int A = two_stage_large(L);
  static constexpr int B = L / A;
  static constexpr int T = A;  // threads of a line
  static constexpr bool kTwo =
      M == Mode::kMod || M == Mode::kGrad || M == Mode::kUpd || M == Mode::kCut;
  static constexpr bool kFirstInverse = M == Mode::kInv || M == Mode::kUpd || M == Mode::kCut;
  static constexpr int kPitchA = A | 1;  // slots from thread to thread after the A-point stage
  static constexpr int kPitchB = B | 1;
  static constexpr int kUsed = std::max(B * kPitchA, kTwo ? A * kPitchB : 0);
  // slots of a line: 2 mod 16 for columns, T mod 16 for rows (the next line's
  // threads continue the half-warp's banks)
  static constexpr int kWant = ROWS ? T % 16 : 2;
  static constexpr int kLine = kUsed + ((kWant - kUsed) % 16 + 16) % 16;
  // Lines per block at most: columns 8 (64-byte segments of a row), rows about
  // 128 threads.
  static constexpr int kLines = ROWS ? std::max(1, 128 / T) : 8;
  static constexpr int kThreads = (kLines * T + 31) / 32 * 32;
  // An update holds one exchange and the old iterate (written and read by the
  // same thread); the other passes of two transforms hold two exchanges, which
  // spares them a barrier; one transform needs one.
  static constexpr int kSideSlots = M == Mode::kUpd ? L : (kTwo ? kLine : 0);
  // Amplitudes read before the wait for the pass before hold B registers over
  // the A-point DFT. Measured at 21 lengths of 45 to 625, launches of 300 k and
  // of 2 M elements, early against late: with A at most 16 the small launches
  // gain 4 to 7% (5 starts of 240: 4.77 -> 4.44 us; nothing at 144 and 150, -3%
  // at 100) and the large ones 0 to 3%, with A = 18, 20 and 24 both lose 7 to
  // 22% (2 of 360: 5.2 -> 6.3 us); at A = 21 and 25 it is within 6% either way.
  static constexpr bool kEarlyAmplitude = A <= 16;
  // Registers: about 2 A + 48 a thread for the larger DFT and its addresses.
  // At the same lengths a step less (64, 80, 104) costs the modulus pass of the
  // small launches 5 to 18% with A at most 16 and up to 32% above (of the large
  // ones -4 to 24%), a step more (104, 128, 168) that of the large launches 0 to
  // 23%; small ones gain 4 to 7% from it at 100, 144, 600 and 625 alone. The
  // updates are indifferent (5% at most).
  static constexpr int kRegisters = A <= 10 ? 80 : (A <= 16 ? 104 : 128);
  static constexpr int kBlocks = std::max(1, std::min(16, 65536 / (kThreads * kRegisters)));
};

// Copies one complex value from global to shared memory asynchronously.
__device__ __forceinline__ void copy_async8(float2* dst, const float2* src) {
  const auto d = static_cast<std::uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
// Waits for all of this thread's copies.
__device__ __forceinline__ void wait_async() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int L, Mode M, bool ROWS>
__global__ void __launch_bounds__(TwoStage<L, M, ROWS>::kThreads, TwoStage<L, M, ROWS>::kBlocks)
    two_stage_kernel(const __grid_constant__ PassParams p, const int lpc, const int shift,
                     const int tiles) {
  using K = TwoStage<L, M, ROWS>;
  constexpr int A = K::A, B = K::B, T = K::T;
  extern __shared__ float2 smem[];
  const int tid = threadIdx.x;
  const int l = ROWS ? tid / T : tid & (lpc - 1);
  const int t = ROWS ? tid - l * T : tid >> shift;
  const int start = static_cast<int>(blockIdx.x) / tiles;
  const int line = (static_cast<int>(blockIdx.x) - start * tiles) * lpc + l;
  const bool active = t < T && l < lpc && line < p.lines_per_start;
  // element 0 of the line within its start, and the distance of its elements
  const int S = ROWS ? 1 : p.S;
  int first = line;
  if constexpr (ROWS) {
    first = line * L;
  } else if (p.S != p.lines_per_start) {
    first = line + line / p.S * (L - 1) * p.S;
  }
  const long long start_off = static_cast<long long>(start) * p.n;
  const int e = first + t * S;  // element t of the line
  float2* __restrict__ w = p.w + start_off + e;
  float2* __restrict__ x = p.x + start_off + e;
  float2* ex = smem + l * K::kLine;
  float2* side = smem + lpc * K::kLine;  // second exchange, or the old iterate

  // What the point-wise step reads besides the arrays of the iteration: its
  // writers (problem set-up, threshold, detwin) are never the kernel right
  // before a pass (dependent_launch.cuh), so the loads are issued before the
  // wait for that one (an iteration of 4 starts of 96 x 96 5.8 -> 5.3 us, of 16 of
  // 240 x 240 15.5 -> 14.5).
  [[maybe_unused]] float amp[M == Mode::kMod || M == Mode::kGrad ? B : 1];
  constexpr bool kUpdate = M == Mode::kUpd || M == Mode::kCut;
  [[maybe_unused]] unsigned char inside[kUpdate ? B : 1];
  [[maybe_unused]] float ca = p.coef_a, cb = p.coef_b;
  auto read_amplitude = [&] {
    if constexpr (M == Mode::kMod || M == Mode::kGrad) {
      if (active) {
        const long long at = amp_offset(p, p.start0 + start) + e;
        if (p.amp_storage == AmpStorage::kF32) {
          const float* a = static_cast<const float*>(p.amp) + at;
#pragma unroll
          for (int q = 0; q < B; ++q) amp[q] = __ldg(a + q * A * S);
        } else if (p.amp_storage == AmpStorage::kF16) {
          const __half* a = static_cast<const __half*>(p.amp) + at;
#pragma unroll
          for (int q = 0; q < B; ++q) amp[q] = to_float(a[q * A * S]);
        } else {
          const __nv_bfloat16* a = static_cast<const __nv_bfloat16*>(p.amp) + at;
#pragma unroll
          for (int q = 0; q < B; ++q) amp[q] = to_float(a[q * A * S]);
        }
      }
    }
  };
  if constexpr (K::kEarlyAmplitude) read_amplitude();
  if constexpr (kUpdate) {
    if (active) {
      const std::uint8_t* s = p.support + start_off + e;
#pragma unroll
      for (int q = 0; q < B; ++q) inside[q] = s[q * A * S];
    }
  }
  wait_for_prior_kernel();  // the wave, the iterate and the control block
  allow_next_kernel();

  if constexpr (M == Mode::kUpd) {
    if (p.coef_from_ctrl) {
      ca = p.ctrl->a;
      cb = p.ctrl->b;
    }
    if (active) {
#pragma unroll
      for (int q = 0; q < B; ++q) copy_async8(side + q * lpc * T + tid, x + q * A * S);
    }
  }
  if (active && t < B) {
    float2 v[A];
#pragma unroll
    for (int q = 0; q < A; ++q) v[q] = M == Mode::kFwdFromX ? x[q * B * S] : w[q * B * S];
    small_dft<A, K::kFirstInverse>(v);
#pragma unroll
    for (int q = 0; q < A; ++q) ex[t * K::kPitchA + q] = v[q];
  }
  if constexpr (!K::kEarlyAmplitude) read_amplitude();  // in flight over the barrier
  __syncthreads();

  float2 u[B];
  if (active) {
    const float2* tw = p.two_stage_twiddle + t;
    u[0] = ex[t];
#pragma unroll
    for (int q = 1; q < B; ++q) {
      const float2 f = __ldg(tw + (q - 1) * A);
      u[q] = ex[q * K::kPitchA + t];
      u[q] = K::kFirstInverse ? cmulc(u[q], f) : cmul(u[q], f);
    }
    small_dft<B, K::kFirstInverse>(u);
  }

  if constexpr (!K::kTwo) {
    if (active) {
#pragma unroll
      for (int q = 0; q < B; ++q) w[q * A * S] = u[q];
    }
    return;
  }

  [[maybe_unused]] float error = 0.0f;
  float2* ex2 = M == Mode::kUpd ? ex : side + l * K::kLine;
  if constexpr (M == Mode::kUpd) __syncthreads();  // every thread has read the exchange
  if (active) {
    if constexpr (M == Mode::kUpd) {
      wait_async();
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const float2 xo = side[q * lpc * T + tid];
        if (!inside[q]) u[q] = relaxed(ca, xo, cb, u[q]);
        x[q * A * S] = u[q];
      }
    } else if constexpr (M == Mode::kCut) {
#pragma unroll
      for (int q = 0; q < B; ++q) {
        if (!inside[q]) u[q] = cscale(u[q], 0.0f);
      }
    } else {
#pragma unroll
      for (int q = 0; q < B; ++q) u[q] = pointwise_projection<M>(u[q], amp[q], p.scale, error);
    }
    small_dft<B, !K::kFirstInverse>(u);
#pragma unroll
    for (int q = 0; q < B; ++q) ex2[t * K::kPitchB + q] = u[q];
  }
  if constexpr (kUpdate) {
    if (p.bump_counter && blockIdx.x == 0 && tid == 0) ++p.ctrl->counters[p.group];
    __syncthreads();
  } else {
    // its barrier also ends the exchange's writes
    const double sum = block_sum_double<false>(static_cast<double>(error));
    if (tid == 0) {
      const Ctrl* c = p.ctrl;
      const int row = c->counters[p.group];
      if (row < c->capacity) {
        atomicAdd(&c->errs[static_cast<long long>(row) * p.starts_total + p.start0 + start], sum);
      }
    }
  }
  if (active && t < B) {
    const float2* tw = p.two_stage_twiddle + (B - 1) * A + t;
    float2 v[A];
    v[0] = ex2[t];
#pragma unroll
    for (int q = 1; q < A; ++q) {
      const float2 f = __ldg(tw + (q - 1) * B);
      v[q] = ex2[q * K::kPitchB + t];
      v[q] = K::kFirstInverse ? cmul(v[q], f) : cmulc(v[q], f);
    }
    small_dft<A, !K::kFirstInverse>(v);
#pragma unroll
    for (int q = 0; q < A; ++q) w[q * B * S] = v[q];
  }
}

// Lines per block: the most the kernel takes, halved while the launch has
// fewer than two blocks per SM (columns stop at 4 lines, a sector per row).
template <int L, Mode M, bool ROWS>
void launch_two_stage(const PassParams& p, cudaStream_t stream) {
  using K = TwoStage<L, M, ROWS>;
  constexpr int kTargetBlocks = 296;
  const int starts = p.lines / p.lines_per_start;
  int lpc = K::kLines;
  auto tiles = [&] { return (p.lines_per_start + lpc - 1) / lpc; };
  while (lpc > (ROWS ? 1 : 4) && static_cast<long long>(starts) * tiles() < kTargetBlocks) lpc /= 2;
  int shift = 0;
  while ((1 << shift) < lpc) ++shift;
  const int threads = (lpc * K::T + 31) / 32 * 32;
  const std::size_t smem =
      sizeof(float2) * lpc * static_cast<std::size_t>(K::kLine + K::kSideSlots);
  launch_dependent(two_stage_kernel<L, M, ROWS>, dim3(static_cast<unsigned>(starts * tiles())),
                   dim3(static_cast<unsigned>(threads)), smem, stream, p, lpc, shift, tiles());
  count_launches(1);
}

template <int L, Mode M, bool ROWS>
void configure_one() {
  using K = TwoStage<L, M, ROWS>;
  constexpr int bytes = static_cast<int>(sizeof(float2)) * K::kLines * (K::kLine + K::kSideSlots);
  static_assert(bytes <= 226 * 1024);
  QPB_CHECK(cudaFuncSetAttribute(two_stage_kernel<L, M, ROWS>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  prefer_shared_memory(two_stage_kernel<L, M, ROWS>);
}

constexpr int two_stage_count(int slice) {
  int n = 0, k = 0;
  for (int L = 2; L <= kMaxTwoStage; ++L) {
    if (two_stage_large(L) && k++ % kTwoStageSlices == slice) ++n;
  }
  return n;
}

template <int SLICE>
constexpr auto two_stage_lengths() {
  std::array<int, two_stage_count(SLICE)> out{};
  int n = 0, k = 0;
  for (int L = 2; L <= kMaxTwoStage; ++L) {
    if (two_stage_large(L) && k++ % kTwoStageSlices == SLICE) out[n++] = L;
  }
  return out;
}

}  // namespace

template <Mode M, bool ROWS, int SLICE>
TwoStageList two_stage_slice() {
  static constexpr auto lengths = two_stage_lengths<SLICE>();
  constexpr int n = static_cast<int>(lengths.size());
  static constexpr auto passes = []<int... I>(std::integer_sequence<int, I...>) {
    return std::array<TwoStagePass, n>{TwoStagePass{lengths[I], &launch_two_stage<lengths[I], M, ROWS>,
                                                    &configure_one<lengths[I], M, ROWS>}...};
  }(std::make_integer_sequence<int, n>{});
  return {passes.data(), n};
}

}  // namespace qpb
