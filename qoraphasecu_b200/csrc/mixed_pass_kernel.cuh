// The mixed-radix line-pass kernel and its launch, instantiated per group of
// modes by mixed_pass_*.cu: lines of any length whose prime factors are at
// most 13, radices chosen at run time. Lengths with a kernel of their own
// (column_pass.cu, fast_pass.cu, two_stage_kernel.cuh) come here only for the
// modes and line counts those do not take.
//
// A line of L = R_0 R_1 .. R_{K-1} points (every radix 2..16, as few stages as
// the length allows; fft_plan.cpp) is transformed by K Stockham stages. A
// stage's work item is one R-point DFT held in registers; between stages the
// values cross shared memory once. The first stage reads its inputs j + q M
// (M = L / R) straight from global memory and the last stage writes its
// outputs j + q M straight back, both coalesced, so a two-stage line (up to
// 256 points) crosses shared memory once per transform. A pass of two
// transforms runs the second with the radices reversed: the first one's last
// stage and the second one's first then are the same work item, with the
// point-wise step between them in registers. Each place in that sequence is
// its own code (Place), so a stage carries no tests of where it stands.
//
// Exchange layout: after a stage with inputs N apart and radix R, output o of
// a line sits at (o / N R) P + o mod N R, P >= N R (exchange_pitch). Both the
// writing item (o = (j / N) N R + j mod N + q N) and the reading one (j' + q M',
// M' a multiple of N R) then step through it by a constant per q, and P keeps
// the items of a half-warp on different banks.
//
// Bound: issue and instruction fetch (the stages of a launch are a few of the
// many compiled here). Against line_pass.cu, which ran these lengths before:
// 16 starts of 240 x 240 71 -> 23 us an iteration, 2 starts of 96^3 125 -> 51.
//
// Columns (stride S > 1): adjacent lines on adjacent threads and next to each
// other in shared memory ([slot][line]), so a half-warp reads neighbouring
// elements of a row. Rows: a line's DFTs on adjacent threads. A block never
// spans two starts; the last block of a start may hold fewer lines.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <iterator>
#include <stdexcept>

#include "dependent_launch.cuh"
#include "mixed_pass.cuh"
#include "projection.cuh"
#include "reduce.cuh"
#include "small_dft.cuh"

namespace qpb {

namespace {

constexpr int kMaxThreads = 128;
constexpr int kMinBlocks = 5;  // resident blocks per SM the registers are budgeted for
constexpr int kMaxSmem = 224 * 1024;

// One stage of one transform as its work items see it; strides in slots of
// the exchange buffer (times the lines per block for columns).
struct MixedStage {
  int m_len;         // items per line, L / R
  int ns;            // distance of a butterfly's outputs, the radices before multiplied
  int step;          // global elements between a butterfly's inputs (m_len S)
  int twiddle;       // offset of the stage's table
  unsigned m_recip;  // fast_div reciprocals of m_len and ns
  unsigned ns_recip;
  int read_pitch;  // block of the exchange read: (j / ns) read_pitch + j mod ns + q read_step
  int read_step;
  int write_pitch;  // block of the exchange written: (j / ns) write_pitch + j mod ns + q write_step
  int write_step;
};

// What a launch adds to PassParams.
struct MixedShape {
  int lpc;        // lines per block (a power of two for columns)
  int lpc_shift;  // log2(lpc) for columns
  int tiles;      // blocks per start
  int pitch;      // slots per line
  int stages;
  int radix[kMaxMixedStages];
  MixedStage stage[2][kMaxMixedStages];  // the first transform's and the reversed second's
};

// n / d for n < 2^16 and d < 2^16 from recip = ceil(2^32 / d) (0 for d = 1):
// the excess n (d recip - 2^32) / 2^32 stays below n / 2^16 < 1 of a unit of
// 1 / d, so the quotient is exact.
inline unsigned reciprocal(int d) {
  return d == 1 ? 0u : static_cast<unsigned>(((1ull << 32) + d - 1) / d);
}
__device__ __forceinline__ int fast_div(int n, unsigned recip) {
  return recip == 0 ? n : static_cast<int>(__umulhi(static_cast<unsigned>(n), recip));
}

constexpr bool two_transforms(Mode m) {
  return m == Mode::kMod || m == Mode::kGrad || m == Mode::kUpd || m == Mode::kCut ||
         m == Mode::kBlur ||
         m == Mode::kBlurMag;
}

// Where a stage stands in its pass.
enum class Place {
  kOnly,   // a line of one stage: load, DFT (point-wise step, second DFT), store
  kFirst,  // from global memory
  kInner,  // between two exchanges
  kMiddle, // the first transform's last stage, the point-wise step, the second's first stage
  kLast,   // to global memory
};

// The values a thread carries from its items to the end of the pass.
struct MixedSums {
  float error = 0.0f;  // modulus and gradient: sum (|y| - A)^2
  float peak = 0.0f;   // blur: level
  float square = 0.0f;
  unsigned count = 0;
};

template <Mode M, bool ROWS>
struct MixedPass {
  static constexpr bool kFirstInverse =
      M == Mode::kInv || M == Mode::kUpd || M == Mode::kCut;

  const PassParams& p;
  const MixedShape& g;
  const int start;  // start of the launch this block works on
  float2* const w;  // this start's arrays
  float2* const x;
  const std::uint8_t* const support;
  const long long amp_base;
  const int line0;  // first line of the block, within its start
  const int lines_here;
  float ca = 0.0f, cb = 0.0f;  // update coefficients
  MixedSums sums;

  // Element 0 of line `l` of the block within its start.
  __device__ __forceinline__ int line_base(int l) const {
    const int line = line0 + l;
    if constexpr (ROWS) {
      return line * p.L;
    } else {
      if (p.S == p.lines_per_start) return line;
      const int outer = line / p.S;
      return line + outer * (p.L - 1) * p.S;
    }
  }

  __device__ __forceinline__ float2 load(int e) const {
    if constexpr (M == Mode::kFwdFromX) {
      return x[e];
    } else if constexpr (M == Mode::kBlurMag) {
      const float2 xv = x[e];
      return {sqrtf(xv.x * xv.x + xv.y * xv.y), 0.0f};
    } else {
      return w[e];
    }
  }

  __device__ __forceinline__ void store(int e, float2 v) {
    w[e] = v;
    if constexpr (M == Mode::kBlur || M == Mode::kBlurMag) {
      if (p.level_method == 1) {
        sums.peak = fmaxf(sums.peak, v.x);
      } else if (p.level_method == 2 && support[e]) {
        sums.square += v.x * v.x;
        ++sums.count;
      }
    }
  }

  // What the point-wise step reads besides the transform, issued before the
  // first DFT: the amplitudes, or the support as one bit per element.
  template <int R>
  struct Side {
    float amp[M == Mode::kMod || M == Mode::kGrad ? R : 1];
    unsigned outside = 0;
  };

  template <int R>
  __device__ __forceinline__ void read_side(Side<R>& side, int e, int step) const {
    if constexpr (M == Mode::kMod || M == Mode::kGrad) {
      if (p.amp_storage == AmpStorage::kF32) {
        const float* a = static_cast<const float*>(p.amp) + amp_base + e;
#pragma unroll
        for (int q = 0; q < R; ++q) side.amp[q] = __ldg(a + q * step);
      } else if (p.amp_storage == AmpStorage::kF16) {
        const __half* a = static_cast<const __half*>(p.amp) + amp_base + e;
#pragma unroll
        for (int q = 0; q < R; ++q) side.amp[q] = to_float(a[q * step]);
      } else {
        const __nv_bfloat16* a = static_cast<const __nv_bfloat16*>(p.amp) + amp_base + e;
#pragma unroll
        for (int q = 0; q < R; ++q) side.amp[q] = to_float(a[q * step]);
      }
    } else if constexpr (M == Mode::kUpd || M == Mode::kCut) {
#pragma unroll
      for (int q = 0; q < R; ++q) side.outside |= (support[e + q * step] == 0 ? 1u : 0u) << q;
    }
  }

  // The point-wise step between the two transforms on the R elements e + q step.
  template <int R>
  __device__ __forceinline__ void pointwise(float2 (&v)[R], const Side<R>& side, int e, int step,
                                            int j, int m_len) {
    if constexpr (M == Mode::kMod || M == Mode::kGrad) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        v[q] = pointwise_projection<M>(v[q], side.amp[q], p.scale, sums.error);
      }
    } else if constexpr (M == Mode::kUpd) {
      // the old iterate in two batches, whose loads are in flight together
      constexpr int B = (R + 1) / 2;
#pragma unroll
      for (int q0 = 0; q0 < R; q0 += B) {
        float2 xo[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
          if (q0 + b < R && (side.outside >> (q0 + b) & 1u)) xo[b] = x[e + (q0 + b) * step];
        }
#pragma unroll
        for (int b = 0; b < B; ++b) {
          const int q = q0 + b;
          if (q < R) {
            if (side.outside >> q & 1u) {
              v[q] = relaxed(ca, xo[b], cb, v[q]);
            }
            x[e + q * step] = v[q];
          }
        }
      }
    } else if constexpr (M == Mode::kCut) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        if (side.outside >> q & 1u) v[q] = cscale(v[q], 0.0f);
      }
    } else if constexpr (M == Mode::kBlur || M == Mode::kBlurMag) {
      const float inv_l = 1.0f / static_cast<float>(p.L);
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const float f = fftfreq(static_cast<std::uint32_t>(j + q * m_len),
                                static_cast<std::uint32_t>(p.L));
        v[q] = cscale(v[q], expf(p.blur_k * f * f) * inv_l);
      }
    }
  }

  template <int R, Place PLACE, bool SECOND>
  __device__ __forceinline__ void stage(const MixedStage& st, const float2* src, float2* dst) {
    constexpr bool kInverse = SECOND ? !kFirstInverse : kFirstInverse;
    constexpr bool kGlobalIn = PLACE == Place::kOnly || PLACE == Place::kFirst;
    constexpr bool kGlobalOut = PLACE == Place::kOnly || PLACE == Place::kLast;
    constexpr bool kPoint =
        two_transforms(M) && (PLACE == Place::kOnly || PLACE == Place::kMiddle);
    const int unit = ROWS ? 1 : g.lpc;
    const int items = g.lpc * st.m_len;
#pragma unroll 1
    for (int item = threadIdx.x; item < items; item += blockDim.x) {
      int l, j;
      if constexpr (ROWS) {
        l = fast_div(item, st.m_recip);
        j = item - l * st.m_len;
      } else {
        l = item & (g.lpc - 1);
        j = item >> g.lpc_shift;
      }
      if (l >= lines_here) continue;
      const int slot0 = ROWS ? l * g.pitch : l;
      int e = 0;
      if constexpr (kGlobalIn || kGlobalOut || kPoint) e = line_base(l) + j * p.S;
      Side<R> side;
      if constexpr (kPoint) read_side<R>(side, e, st.step);
      float2 v[R];
      int block = j, k = 0;  // j / ns, j mod ns
      if constexpr (kGlobalIn) {
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = load(e + q * st.step);
      } else {
        if constexpr (PLACE == Place::kInner) {
          block = fast_div(j, st.ns_recip);
          k = j - block * st.ns;
        } else {  // the last stage of a transform: ns = m_len
          block = 0;
          k = j;
        }
        const float2* from = src + slot0 + block * st.read_pitch + k * unit;
        const float2* tw = p.mixed_twiddle + st.twiddle + k;
        v[0] = from[0];
#pragma unroll
        for (int q = 1; q < R; ++q) {
          const float2 f = __ldg(tw + (q - 1) * st.ns);
          const float2 u = from[q * st.read_step];
          v[q] = kInverse ? cmulc(u, f) : cmul(u, f);
        }
      }
      small_dft<R, kInverse>(v);
      if constexpr (kPoint) {
        pointwise<R>(v, side, e, st.step, j, st.m_len);
        small_dft<R, !kInverse>(v);
      }
      if constexpr (kGlobalOut) {
#pragma unroll
        for (int q = 0; q < R; ++q) store(e + q * st.step, v[q]);
      } else if constexpr (PLACE == Place::kMiddle) {
        // the second transform's first stage: its item j too
        float2* to = dst + slot0 + j * g.stage[1][0].write_pitch;
#pragma unroll
        for (int q = 0; q < R; ++q) to[q * unit] = v[q];
      } else if constexpr (PLACE == Place::kFirst) {
        float2* to = dst + slot0 + j * st.write_pitch;
#pragma unroll
        for (int q = 0; q < R; ++q) to[q * unit] = v[q];
      } else {
        float2* to = dst + slot0 + block * st.write_pitch + k * unit;
#pragma unroll
        for (int q = 0; q < R; ++q) to[q * st.write_step] = v[q];
      }
    }
  }

  // The stage of the radix in [LO, HI], by halving: a switch becomes an
  // indirect branch through a table in constant memory, cold at every launch.
  template <Place PLACE, bool SECOND, int LO = 2, int HI = 16>
  __device__ __forceinline__ void run(int radix, int s, const float2* src, float2* dst) {
    if constexpr (LO == HI) {
      stage<LO, PLACE, SECOND>(g.stage[SECOND ? 1 : 0][s], src, dst);
    } else {
      constexpr int MID = (LO + HI) / 2;
      if (radix <= MID) {
        run<PLACE, SECOND, LO, MID>(radix, s, src, dst);
      } else {
        run<PLACE, SECOND, MID + 1, HI>(radix, s, src, dst);
      }
    }
  }
};

template <Mode M, bool ROWS>
__global__ void __launch_bounds__(kMaxThreads, kMinBlocks)
    mixed_pass_kernel(const __grid_constant__ PassParams p, const __grid_constant__ MixedShape g) {
  extern __shared__ float2 smem[];
  const int start = static_cast<int>(blockIdx.x) / g.tiles;
  const int line0 = (static_cast<int>(blockIdx.x) - start * g.tiles) * g.lpc;
  const long long start_off = static_cast<long long>(start) * p.n;
  MixedPass<M, ROWS> pass{p,
                          g,
                          start,
                          p.w + start_off,
                          p.x + start_off,
                          p.support + start_off,
                          amp_offset(p, p.start0 + start),
                          line0,
                          min(g.lpc, p.lines_per_start - line0)};
  wait_for_prior_kernel();  // its wave, iterate, support and control block
  allow_next_kernel();
  if constexpr (M == Mode::kUpd) {
    pass.ca = p.coef_a;
    pass.cb = p.coef_b;
    if (p.coef_from_ctrl) {
      pass.ca = p.ctrl->a;
      pass.cb = p.ctrl->b;
    }
  }

  const int stages = g.stages;
  if (stages == 1) {
    pass.template run<Place::kOnly, false>(g.radix[0], 0, nullptr, nullptr);
  } else {
    float2* src = smem + g.lpc * g.pitch;
    float2* dst = smem;
    auto next = [&] {
      __syncthreads();
      float2* t = src;
      src = dst;
      dst = t;
    };
    pass.template run<Place::kFirst, false>(g.radix[0], 0, src, dst);
    for (int s = 1; s < stages - 1; ++s) {
      next();
      pass.template run<Place::kInner, false>(g.radix[s], s, src, dst);
    }
    next();
    if constexpr (two_transforms(M)) {
      pass.template run<Place::kMiddle, false>(g.radix[stages - 1], stages - 1, src, dst);
      for (int s = 1; s < stages - 1; ++s) {
        next();
        pass.template run<Place::kInner, true>(g.radix[stages - 1 - s], s, src, dst);
      }
      next();
      pass.template run<Place::kLast, true>(g.radix[0], stages - 1, src, dst);
    } else {
      pass.template run<Place::kLast, false>(g.radix[stages - 1], stages - 1, src, dst);
    }
  }

  if constexpr (M == Mode::kMod || M == Mode::kGrad) {
    const double sum = block_sum_double<false>(static_cast<double>(pass.sums.error));
    if (threadIdx.x == 0) {
      const Ctrl* c = p.ctrl;
      const int row = c->counters[p.group];
      if (row < c->capacity) {
        atomicAdd(&c->errs[static_cast<long long>(row) * p.starts_total + p.start0 + start], sum);
      }
    }
  } else if constexpr (M == Mode::kUpd || M == Mode::kCut) {
    if (p.bump_counter && blockIdx.x == 0 && threadIdx.x == 0) ++p.ctrl->counters[p.group];
  } else if constexpr (M == Mode::kBlur || M == Mode::kBlurMag) {
    if (p.level_method == 1) {
      const float peak = warp_max(pass.sums.peak);
      if ((threadIdx.x & 31) == 0) atomicMax(&p.level[start].max_bits, __float_as_int(peak));
    } else if (p.level_method == 2) {
      const double s2 = block_sum_double(static_cast<double>(pass.sums.square));
      __syncthreads();
      const double c2 = block_sum_double(static_cast<double>(pass.sums.count));
      if (threadIdx.x == 0) {
        atomicAdd(&p.level[start].sum, s2);
        atomicAdd(&p.level[start].count, static_cast<unsigned long long>(c2));
      }
    }
  }
}

// ------------------------------------------------------------------- host side
// The launch's shape for `lpc` lines per block.
inline MixedShape mixed_shape(const PassParams& p, int lpc) {
  const LinePlan& plan = *p.plan;
  MixedShape g{};
  g.stages = plan.mixed_stages;
  std::copy(std::begin(plan.mixed_radix), std::end(plan.mixed_radix), g.radix);
  g.lpc = lpc;
  while ((1 << g.lpc_shift) < lpc) ++g.lpc_shift;
  g.tiles = (p.lines_per_start + lpc - 1) / lpc;
  const int unit = p.S == 1 ? 1 : lpc;  // slots are [slot][line] for columns
  g.pitch = 1;
  int twiddle = 0;
  for (int order = 0; order < 2; ++order) {
    int ns = 1, pitch = 0;
    for (int s = 0; s < g.stages; ++s) {
      const int radix = g.radix[order ? g.stages - 1 - s : s];
      MixedStage& st = g.stage[order][s];
      st.m_len = p.L / radix;
      st.ns = ns;
      st.step = st.m_len * p.S;
      st.m_recip = reciprocal(st.m_len);
      st.ns_recip = reciprocal(ns);
      st.read_pitch = pitch * unit;
      st.read_step = st.m_len / ns * pitch * unit;
      st.twiddle = twiddle;
      if (s > 0) twiddle += (radix - 1) * ns;
      const int width = ns * radix;  // outputs of one block of the exchange
      pitch = plan.mixed_pitch[order][s];
      st.write_pitch = pitch * unit;
      st.write_step = ns * unit;
      if (s + 1 < g.stages) g.pitch = std::max(g.pitch, (p.L / width - 1) * pitch + width);
      ns = width;
    }
  }
  return g;
}

inline long long mixed_smem(const MixedShape& g) {
  return g.stages > 1 ? 2LL * g.pitch * g.lpc * static_cast<long long>(sizeof(float2)) : 0;
}

// Lines per block: columns take 8 lines (a 64-byte segment per row) where that
// leaves two blocks per SM, else 4; rows as many lines as fill a block's
// threads in the widest stage. Long lines take fewer, within a quarter of the
// shared memory.
inline int choose_lines(const PassParams& p) {
  constexpr int kTargetBlocks = 296;
  int most = 1;  // work items a line has in its widest stage
  for (int s = 0; s < p.plan->mixed_stages; ++s) most = std::max(most, p.L / p.plan->mixed_radix[s]);
  const long long starts = p.lines / p.lines_per_start;
  auto blocks = [&](int lpc) { return starts * ((p.lines_per_start + lpc - 1) / lpc); };
  auto too_large = [&](int lpc) { return mixed_smem(mixed_shape(p, lpc)) > kMaxSmem / 4; };
  int lpc;
  if (p.S == 1) {
    lpc = std::max(1, std::min(p.lines_per_start, kMaxThreads / most));
    while (lpc > 1 && (too_large(lpc) || blocks(lpc) < kTargetBlocks)) lpc = (lpc + 1) / 2;
  } else {
    lpc = 8;
    while (lpc > 1 && (too_large(lpc) || (lpc > 4 && blocks(lpc) < kTargetBlocks))) lpc /= 2;
  }
  return lpc;
}

template <Mode M, bool ROWS>
void launch_mixed(const PassParams& p, cudaStream_t stream) {
  const int lpc = choose_lines(p);
  const MixedShape g = mixed_shape(p, lpc);
  int most = 1;
  for (int s = 0; s < g.stages; ++s) most = std::max(most, g.stage[0][s].m_len);
  // a stage's items spread evenly over the threads
  const int items = lpc * most;
  const int rounds = (items + kMaxThreads - 1) / kMaxThreads;
  const int threads = ((items + rounds - 1) / rounds + 31) / 32 * 32;
  const long long smem = mixed_smem(g);
  if (smem > kMaxSmem) {
    throw std::logic_error("mixed line pass: shared memory request above the configured maximum");
  }
  const long long starts = p.lines / p.lines_per_start;
  const dim3 grid(static_cast<unsigned>(starts * g.tiles));
  launch_dependent(mixed_pass_kernel<M, ROWS>, grid, dim3(threads), static_cast<std::size_t>(smem),
                   stream, p, g);
  count_launches(1);
}

}  // namespace

template <Mode M>
void launch_mixed_mode(const PassParams& p, cudaStream_t stream) {
  if (p.S == 1) {
    launch_mixed<M, true>(p, stream);
  } else {
    launch_mixed<M, false>(p, stream);
  }
}

template <Mode M>
void configure_mixed_mode() {
  auto allow = [](auto kernel) {
    QPB_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
    prefer_shared_memory(kernel);
  };
  allow(mixed_pass_kernel<M, true>);
  allow(mixed_pass_kernel<M, false>);
}

}  // namespace qpb
